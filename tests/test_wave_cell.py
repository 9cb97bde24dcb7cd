"""The two forms of the 2D wave stages against the oracle where each can go wrong: the cell
form (one CTA per 32 x 8 points, grids up to about 1.1 to 1.6 million points) at cell edges
and the smallest grids, on planes and on AoS device arrays, and the persistent form on a
ragged grid above the rule's line.

Tolerances, as the other parity tests: 1e-12 (max norm, relative) in FP64; FP32 states after
RK4 1e-5, FP32 right-hand sides 1e-5 plus the inputs' 2^-24 rounding amplified by the
derivative (1/h times the stencil's weight sum, at most 4).
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(12, 12), (31, 24), (32, 26), (33, 14), (65, 30), (97, 42)]


def _pair(sbp, kind, order, nx, ny, bc, precision):
    rng = np.random.default_rng(nx + ny)
    names = {"hom": "WAVE_HOM_2D", "var": "WAVE_VAR_2D", "two_block": "WAVE_2BLOCK_2D", "mms": "WAVE_MMS_2D"}
    kw = {"bc": bc}
    if kind in ("var", "two_block"):
        kw.update(rho=0.5 + rng.random(nx * ny), K=0.5 + rng.random(nx * ny))
    return (sbp.Context(getattr(sbp, names[kind]), order, nx, ny, precision=precision, **kw),
            O.Problem(getattr(O, names[kind]), order, nx, ny, **kw))


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


def _rhs_device(sbp, ctx, v, t, overlap=False):
    import torch

    n = v.size
    buf = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    buf[:n] = torch.from_numpy(v)
    out = buf[:n] if overlap else buf[n:]
    torch.cuda.synchronize()
    ctx.rhs_ptr(t, buf.data_ptr(), out.data_ptr(), sbp.DEVICE)
    return out.cpu().numpy()


@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32"])
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("kind", ["hom", "var", "two_block", "mms"])
def test_cells_match_the_oracle(sbp, port, kind, order, fp32):
    if fp32 and kind == "mms":
        pytest.skip("the manufactured-solution problem is FP64 only")
    for n, (nx, ny) in enumerate(SIZES):
        if kind == "two_block" and ny < 24:
            continue
        bc = 0 if kind == "mms" else n % 2
        ctx, pb = _pair(sbp, kind, order, nx, ny, bc, sbp.FP32 if fp32 else sbp.FP64)
        v = port.init_wave_pulse(nx, ny, 0.1, -0.1, 0.4, 1.0)
        v = v + 0.05 * np.random.default_rng(n).standard_normal(v.size)
        dt = 0.1 / max(nx, ny)
        with ctx:
            ref = port.rhs(pb, v, 0.2)
            tol = 1e-12
            if fp32:
                tol = 1e-5 + 2.0 ** -24 * 8 * max(nx, ny) * np.max(np.abs(v)) / np.max(np.abs(ref))
            assert _rel(ctx.rhs(v, 0.2), ref) < tol  # planes
            assert _rel(_rhs_device(sbp, ctx, v, 0.2), ref) < tol  # AoS device arrays
            assert _rel(_rhs_device(sbp, ctx, v, 0.2, overlap=True), ref) < tol  # in place: planes
            assert _rel(ctx.rk4(v, 0.0, dt, 5), port.rk4(pb, v, 0.0, dt, 5)) < (1e-5 if fp32 else 1e-12)


@pytest.mark.parametrize("kind,fp32,order", [("hom", False, 6), ("var", False, 4), ("mms", False, 4), ("hom", True, 4),
                                              ("var", True, 6)])
def test_persistent_form_above_the_line(sbp, port, kind, fp32, order):
    nx, ny = 1283, 1279
    ctx, pb = _pair(sbp, kind, order, nx, ny, 0 if kind == "mms" else 1, sbp.FP32 if fp32 else sbp.FP64)
    v = port.init_wave_pulse(nx, ny, 0.1, -0.1, 0.4, 1.0)
    v = v + 1e-3 * np.random.default_rng(5).standard_normal(v.size)
    dt = 0.1 / nx
    with ctx:
        assert _rel(ctx.rk4(v, 0.0, dt, 2), port.rk4(pb, v, 0.0, dt, 2)) < (1e-5 if fp32 else 1e-12)


@pytest.mark.parametrize("kind,nx,ny", [("hom", 1283, 1279), ("two_block", 65, 42), ("mms", 33, 14)])
def test_fehlberg_attempts_in_both_forms(sbp, port, kind, nx, ny):
    """A fixed interval at a tolerance that accepts every attempt: the oracle's steps."""
    ctx, pb = _pair(sbp, kind, 4, nx, ny, 0 if kind == "mms" else 1, sbp.FP64)
    v = port.init_wave_pulse(nx, ny, 0.1, -0.1, 0.4, 1.0)
    dt = 0.2 / max(nx, ny)
    with ctx:
        ctx.set_state(v)
        st = ctx.rk45_resident(0.0, 3 * dt, dt, atol=1e3, rtol=0.0)
        got = ctx.get_state()
    ref, rst = port.rk45(pb, v, 0.0, 3 * dt, dt, atol=1e3, rtol=0.0)
    assert (st["accepted"], st["rejected"]) == (rst["accepted"], rst["rejected"])
    assert _rel(got, ref) < 1e-12
