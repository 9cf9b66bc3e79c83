"""The angle multiples the translator gives to ndw::MulAngle (`let a = acos(x) * f;` or
atan2, used as sin(a) and cos(a) only): which declarations it takes, and the FP64 DE that
comes of them on the device, against extended precision."""

import numpy as np
import pytest

from numericdream_b200.translator import translate

HEAD = "// @param A min=0 max=9 default=8\nfn de_iterations(p: Params) -> i32 { return 4; }\n"
FIN = "fn de_finalize(carry: IterCarry) -> f32 { return bulb_log_escape(carry); }\n"


def _step(body):
    return (HEAD + "fn de_step(carry: IterCarry, pos: vec3f, p: Params) -> IterCarry {\n" + body +
            "    return IterCarry(vec3f(x, y, 0.0), carry.dr);\n}\n" + FIN)


@pytest.mark.parametrize("body,count", [
    ("let a = acos(carry.z.x) * p[0]; let x = sin(a); let y = cos(a);", 1),
    ("let a = atan2(carry.z.x, carry.z.y) * p[0]; let x = sin(a) * 2.0; let y = x;", 1),
    ("let a = acos(carry.z.x) * p[0]; let x = sin(a) + a; let y = cos(a);", 0),      # used as a number too
    ("let a = acos(carry.z.x) + p[0]; let x = sin(a); let y = cos(a);", 0),
    ("var a = acos(carry.z.x) * p[0]; let x = sin(a); let y = cos(a);", 0),
    ("let a = acos(carry.z.x) * p[0]; let x = sin(a * 2.0); let y = cos(a);", 0),
    ("let a = acos(carry.z.xy) * p[0]; let x = sin(a).x; let y = cos(a).y;", 0),
    ("let a = acos(carry.z.x) * p[0]; var x = 0.0; { let a = 1.0; x = sin(a); } let y = cos(a);", 0),
])
def test_recognised_angles(body, count):
    assert translate(_step(body), "f").cpp.count("const ndw::MulAngle<T>") == count


@pytest.mark.gpu
@pytest.mark.parametrize("power", [2.0, 3.0, 8.0, 16.0, 7.5])
def test_fp64_de_on_the_device(ctx, power):
    from numericdream_b200 import abi, runtime

    v = abi.make_view(runtime.find_formula("mandelbulb_bailout"), 8, 8, (0, 0, -3.0), params=[power, 6.0, 2.0])
    rng = np.random.default_rng(5)
    pts = rng.normal(size=(4096, 3))
    pts *= (rng.uniform(0.2, 1.9, 4096) / np.linalg.norm(pts, axis=1))[:, None]
    pts[:64, :2] = 0.0   # on the polar axis: atan2 of zeros
    pts[64:128, :2] *= 1e-150
    pts[128:160, 2] = 0.0
    de, _, _ = ctx.de_points(v, pts, de_precision=64)
    L = np.longdouble
    p, z, dr = pts.astype(L), pts.astype(L), np.ones(4096, L)
    for _ in range(6):
        r = np.sqrt((z * z).sum(1))
        go = ~(r > 2)
        th, ph = np.arccos(np.clip(z[:, 2] / r, -1, 1)) * L(power), np.arctan2(z[:, 1], z[:, 0]) * L(power)
        rp = r ** L(power - 1.0)
        n = np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], 1) * (rp * r)[:, None] + p
        z = np.where(go[:, None], n, z)
        dr = np.where(go, rp * L(power) * dr + 1, dr)
    r = np.sqrt((z * z).sum(1))
    ref = np.minimum(0.5 * np.log(np.maximum(r, 1e-6)) * r / np.maximum(dr, 1e-6), r)
    # a step's rounding is a few 1e-15 of |z| (times 16 for the angle), which the estimate
    # divides by the growth dr of the steps before it: six steps stay below 1e-12
    assert np.isfinite(de).all() and np.abs(de - ref).max() <= 1e-12
