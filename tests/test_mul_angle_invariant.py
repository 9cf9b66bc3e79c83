"""An angle multiple built from the position and the parameters alone is the same in every
iteration, whether the translator keeps it as a number or as ndw::MulAngle: its sine and
cosine stay invariant addends."""

import pytest

from numericdream_b200.translator import translate

FORMULA = """// @param A min=0 max=9 default=8
fn de_iterations(p: Params) -> i32 { return 4; }
fn de_step(carry: IterCarry, pos: vec3f, p: Params) -> IterCarry {
    let a = %s;
    let x = carry.z.x * 2.0 + pos.x + p[0] * sin(a);
    return IterCarry(vec3f(x, cos(a), 0.0), carry.dr);
}
fn de_finalize(carry: IterCarry) -> f32 { return bulb_log_escape(carry); }
"""


@pytest.mark.parametrize("angle,folded,grouped", [
    ("atan2(pos.y, pos.x) * p[0]", True, True),
    ("acos(pos.z) * p[0]", True, True),
    ("acos(pos.z) + p[0]", False, True),
    ("atan2(carry.z.y, carry.z.x) * p[0]", True, False),
    ("acos(pos.z) * carry.dr", True, False),
])
def test_an_invariant_angle_is_an_invariant_addend(angle, folded, grouped):
    cpp = translate(FORMULA % angle, "f").cpp
    assert ("const ndw::MulAngle<T> a" in cpp) == folded
    assert ("ndw::add_inv((carry.z.x * T(2.0)), pos.x, " in cpp) == grouped
