"""The 1D step loops on one thread-block cluster against the oracle: the smallest grids, one
and several CTAs, sizes around the chunk of points a CTA owns (the last CTA then holds few),
the largest size the cluster takes and the first that is launched stage by stage, more steps
than one launch runs, constant and varying velocities.

Tolerances, as the other parity tests: 1e-12 (max norm, relative) in FP64, 1e-5 in FP32.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

# one CTA up to 128 points, then ceil(n / 128) up to eight
SIZES = [12, 63, 128, 129, 257, 511, 513, 1025, 3001]


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


def _run(sbp, port, kind, order, n, steps, fp32, field):
    kw = {}
    if kind == "advection":
        sp, op = sbp.ADVECTION_1D, O.ADVECTION_1D
        kw["a"] = -0.8 if n % 2 else 1.0
        if field:
            kw["a_field"] = 0.5 + np.random.default_rng(n).random(n)
    else:
        sp, op = sbp.REFLECTION_1D, O.REFLECTION_1D
    v = np.random.default_rng(n + order).standard_normal(n * (1 if kind == "advection" else 2))
    dt = 0.05 / n
    with sbp.Context(sp, order, n, precision=sbp.FP32 if fp32 else sbp.FP64, **kw) as ctx:
        got = ctx.rk4(v, 0.0, dt, steps)
    assert _rel(got, port.rk4(O.Problem(op, order, n, **kw), v, 0.0, dt, steps)) < (1e-5 if fp32 else 1e-12)


@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32"])
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("kind", ["advection", "reflection"])
def test_step_loops(sbp, port, kind, order, fp32):
    for k, n in enumerate(SIZES):
        _run(sbp, port, kind, order, n, 7 + k % 2, fp32, field=k % 3 == 2)


@pytest.mark.parametrize("kind,n,fp32", [("advection", 6500, False), ("advection", 6501, False),
                                          ("reflection", 5000, False), ("reflection", 5001, False),
                                          ("advection", 8192, True), ("reflection", 8193, True)])
def test_the_line_between_the_forms(sbp, port, kind, n, fp32):
    _run(sbp, port, kind, 4, n, 3, fp32, False)


def test_more_steps_than_a_launch(sbp, port):
    _run(sbp, port, "advection", 4, 201, 2003, False, False)
