"""What bench.py divides by what: the evaluations of both kernels by the time of both, and
the FLOPs of an evaluation without the iterations that an escaped orbit no longer runs."""

import types

import pytest

import bench
from numericdream_b200 import abi, opcount, runtime


def test_moving_evaluations_between_the_kernels_moves_no_rate():
    st = types.SimpleNamespace(de_evals=10**9, march_evals=9 * 10**8)
    assert bench.forward_tflops(st, 50.0, 2.0, 0.5) == pytest.approx(20.0)
    st.march_evals = 7 * 10**8
    assert bench.forward_tflops(st, 50.0, 1.2, 1.3) == pytest.approx(20.0)


def test_flops_leave_out_the_iterations_after_the_escape(ndlib):
    # a camera at distance 30: every probe before the last lies outside the escape radius,
    # where the first step returns the carry, however many iterations are asked for
    per = []
    for iterations in (2.0, 16.0):
        v = abi.make_view(runtime.find_formula("mandelbulb_bailout"), 16, 16, (0.0, 0.0, -30.0), fov_y_deg=0.1,
                          params=[8.0, iterations, 2.0], max_dist=27.0)
        per.append(opcount.flops_per_eval_for([v])[0])
    assert per[1] == pytest.approx(per[0], rel=1e-12)
