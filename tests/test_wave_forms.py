"""Every form of the 2D wave stages at the sizes where it can go wrong. Which kernels a grid runs
depends on its number of points, so small grids only meet the persistent tiles, and the cells
stage by stage, when a context is held to them (sbp_test_wave_form).

Sizes: one below, at and above the tiles (64 columns; 12 rows FP64 variable, 11 manufactured, 14
constant coefficients; 24 and 32 FP32) and the cells (32 x 8), a last cell that holds only the
x face, the smallest grids, two-block halves that end inside a tile, and several tiles per CTA
and per ring stage.

Tolerances, as the other parity tests: 1e-12 (max norm, relative) in FP64; FP32 states after RK4
1e-5, FP32 right-hand sides 1e-5 plus the inputs' 2^-24 rounding amplified by the derivative (1/h
times the stencil's weight sum, at most 4).
"""
import numpy as np
import pytest

import oracle as O

SIZES = [("hom", 12, 12), ("hom", 64, 14), ("hom", 65, 15), ("hom", 129, 70), ("var", 12, 12), ("var", 63, 12),
         ("var", 64, 13), ("var", 65, 24), ("var", 131, 25), ("mms", 12, 12), ("mms", 64, 12), ("mms", 65, 22),
         ("mms", 129, 23), ("two_block", 64, 24), ("two_block", 65, 26), ("two_block", 130, 50)]
RAGGED = [(289, 301), (415, 330), (449, 323)]  # cells above the whole steps' size, narrow last cells


def _pair(sbp, kind, order, nx, ny, bc, fp32=False):
    rng = np.random.default_rng(nx * 1000 + ny)
    name = {"hom": "WAVE_HOM_2D", "var": "WAVE_VAR_2D", "two_block": "WAVE_2BLOCK_2D", "mms": "WAVE_MMS_2D"}[kind]
    kw = {"bc": 0 if kind == "mms" else bc}
    if kind in ("var", "two_block"):
        kw.update(rho=0.5 + rng.random(nx * ny), K=0.5 + rng.random(nx * ny))
    return (sbp.Context(getattr(sbp, name), order, nx, ny, precision=sbp.FP32 if fp32 else sbp.FP64, **kw),
            O.Problem(getattr(O, name), order, nx, ny, **kw))


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


def test_test_aid_rejects_bad_arguments(sbp):
    assert sbp.load().sbp_test_wave_form(None, 0) == sbp.ERR_INVALID


@pytest.mark.gpu
def test_unknown_forms_and_problems_are_refused(sbp):
    with sbp.Context(sbp.WAVE_HOM_2D, 4, 64, 64) as c:
        for form in (-1, 3):
            with pytest.raises(sbp.SbpError) as e:
                c.test_wave_form(form)
            assert e.value.code == sbp.ERR_INVALID
    with sbp.Context(sbp.ADVECTION_2D, 4, 64, 64) as c:
        with pytest.raises(sbp.SbpError):
            c.test_wave_form(sbp.FORM_CELLS)


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("form", [1, 2], ids=["persistent", "cells"])
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("kind,nx,ny", SIZES)
def test_fp64(sbp, port, kind, nx, ny, order, form, bc):
    ctx, pb = _pair(sbp, kind, order, nx, ny, bc)
    v = np.random.default_rng(order).standard_normal(3 * nx * ny)
    dt = 0.05 / max(nx, ny)
    with ctx:
        ctx.test_wave_form(form)
        assert _rel(ctx.rhs(v, 0.3), port.rhs(pb, v, 0.3)) < 1e-12
        assert _rel(ctx.rk4(v, 0.1, dt, 53), port.rk4(pb, v, 0.1, dt, 53)) < 1e-12  # two step graphs
        ctx.set_state(v)
        st = ctx.rk45_resident(0.0, 3 * dt, dt, atol=1e3, rtol=0.0)
        ref, rst = port.rk45(pb, v, 0.0, 3 * dt, dt, atol=1e3, rtol=0.0)
        assert (st["accepted"], st["rejected"]) == (rst["accepted"], rst["rejected"])
        assert _rel(ctx.get_state(), ref) < 1e-12
        ctx.test_wave_form(3 - form)  # the other form's graphs and partial sums
        ctx.set_state(v)
        ctx.rk45_resident(0.0, 3 * dt, dt, atol=1e3, rtol=0.0)
        assert _rel(ctx.get_state(), ref) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("form", [1, 2], ids=["persistent", "cells"])
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("kind,nx,ny", [s for s in SIZES if s[0] != "mms"])
def test_fp32(sbp, port, kind, nx, ny, order, form):
    for bc in (0, 1):
        ctx, pb = _pair(sbp, kind, order, nx, ny, bc, fp32=True)
        v = port.init_wave_pulse(nx, ny, 0.1, -0.1, 0.4, 1.0)
        v = v + 0.05 * np.random.default_rng(nx).standard_normal(v.size)
        dt = 0.1 / max(nx, ny)
        ref = port.rhs(pb, v, 0.0)
        with ctx:
            ctx.test_wave_form(form)
            tol = 1e-5 + 2.0 ** -24 * 8 * max(nx, ny) * np.max(np.abs(v)) / np.max(np.abs(ref))
            assert _rel(ctx.rhs(v), ref) < tol
            assert _rel(ctx.rk4(v, 0.0, dt, 5), port.rk4(pb, v, 0.0, dt, 5)) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("kind", ["hom", "var", "two_block", "mms"])
def test_ragged_grids_by_size(sbp, port, kind, order):
    for n, (nx, ny) in enumerate(RAGGED):
        if kind == "two_block":
            ny += ny % 2
        ctx, pb = _pair(sbp, kind, order, nx, ny, n % 2)
        v = np.random.default_rng(n).standard_normal(3 * nx * ny)
        dt = 0.05 / max(nx, ny)
        with ctx:
            assert _rel(ctx.rk4(v, 0.1, dt, 2), port.rk4(pb, v, 0.1, dt, 2)) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("kind,nx,ny", [("hom", 700, 517), ("two_block", 700, 518), ("var", 700, 517),
                                         ("mms", 700, 517)])
def test_several_tiles_per_cta(sbp, port, kind, nx, ny):
    """407 tiles or more for 152 CTAs: ring stages and their barriers' phases come round again."""
    ctx, pb = _pair(sbp, kind, 4, nx, ny, 1)
    v = np.random.default_rng(3).standard_normal(3 * nx * ny)
    with ctx:
        ctx.test_wave_form(1)
        assert _rel(ctx.rk4(v, 0.1, 5e-5, 3), port.rk4(pb, v, 0.1, 5e-5, 3)) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("form", [1, 2], ids=["persistent", "cells"])
@pytest.mark.parametrize("kind", ["var", "two_block", "mms"])
def test_values_outside_the_fixed_point_range(sbp, port, kind, form):
    """Values below 2^-959, from 2^1008, and one NaN point: FP64 taps."""
    nx, ny = 70, 40
    ctx, pb = _pair(sbp, kind, 4, nx, ny, 1)
    v = np.random.default_rng(1).standard_normal(3 * nx * ny)
    with ctx:
        ctx.test_wave_form(form)
        if kind != "mms":
            for scale in (2.0 ** -990, 2.0 ** 1010):
                assert _rel(ctx.rhs(v * scale), port.rhs(pb, v * scale)) < 1e-12
        v[3 * (9 * nx + 35) + 2] = np.nan
        got, ref = ctx.rhs(v), port.rhs(pb, v)
        # the point's neighbours, and nothing the oracle (whose zero centre tap reads it too) has finite
        assert np.isnan(got).sum() == 8 and not (np.isnan(got) & ~np.isnan(ref)).any()
        assert _rel(got[~np.isnan(ref)], ref[~np.isnan(ref)]) < 1e-12
