"""The cell form of the FP64 2D advection stages against the oracle: sizes one below, at and
above the cell (32 x 8 points, 32 x 16 above 450 thousand points), the sizes on both sides of
the lines between the forms, constant and varying velocities of either sign, values outside
the fixed-point range, and the adaptive integrator, whose stopped attempts skip.

Tolerance 1e-12 (max norm, relative), as the other FP64 parity tests.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(200, 200), (201, 200), (33, 1217), (1281, 32), (225, 209), (671, 671), (705, 639), (1500, 321)]


def _close(a, b):
    return np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


def _pair(sbp, order, nx, ny, field):
    kw = {"a": 1.5, "b": -1.0} if nx % 2 else {"a": -0.7, "b": 0.0}
    if field:
        rng = np.random.default_rng(nx)
        kw.update(a_field=rng.standard_normal(nx * ny), b_field=rng.standard_normal(nx * ny))
    return (sbp.Context(sbp.ADVECTION_2D, order, nx, ny, **kw), O.Problem(O.ADVECTION_2D, order, nx, ny, **kw))


@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("field", [False, True], ids=["constant", "field"])
def test_stages(sbp, port, order, field):
    for nx, ny in SIZES:
        ctx, pb = _pair(sbp, order, nx, ny, field)
        v = np.random.default_rng(order).standard_normal(nx * ny)
        dt = 0.02 / max(nx, ny)
        with ctx:
            assert _close(ctx.rhs(v), port.rhs(pb, v))
            assert _close(ctx.rk4(v, 0.0, dt, 3), port.rk4(pb, v, 0.0, dt, 3))


def test_values_outside_the_fixed_point_range(sbp, port):
    ctx, pb = _pair(sbp, 4, 225, 209, False)
    v = np.random.default_rng(2).standard_normal(225 * 209)
    with ctx:
        for scale in (2.0 ** -990, 2.0 ** 1010, 0.0):
            got, ref = ctx.rhs(v * scale), port.rhs(pb, v * scale)
            assert _close(got, ref)
        v[100 * 225 + 100] = np.nan
        got = ctx.rhs(v)
        assert np.isnan(got).sum() == 8  # the stencil's points, not the cell's


def test_adaptive_integrator(sbp, port):
    ctx, pb = _pair(sbp, 4, 225, 209, False)
    x = np.linspace(-1, 1, 225)
    y = np.linspace(-1, 1, 209)
    v = np.exp(-((x / 0.3) ** 2)[None, :] - ((y / 0.3) ** 2)[:, None]).ravel()
    with ctx:
        ctx.set_state(v)
        st = ctx.rk45_resident(0.0, 0.01, 0.002, atol=1e3, rtol=0.0)
        got = ctx.get_state()
    ref, rst = port.rk45(pb, v, 0.0, 0.01, 0.002, atol=1e3, rtol=0.0)
    assert (st["accepted"], st["rejected"]) == (rst["accepted"], rst["rejected"])
    assert _close(got, ref)
