"""The fixed-point FP64 stages of the variable-coefficient, two-block and manufactured-
solution problems and of the Fehlberg integrator: their conversions restated on the CPU
(finer unit, sums rounded to nearest), and the kernels against the oracle at tile edges and
outside the fixed-point range.

Tolerances. Conversions: a value errs by under one unit of 2^(emax-1077), a sum by half an
ulp. Kernels: 1e-12 relative (max norm), the bar of the other FP64 parity tests.
"""
from fractions import Fraction

import numpy as np
import pytest

import oracle as O
from test_fixed_point_arithmetic import COEF, DEN, WEIGHTS, bits, dexp, from_bits


def fx_from(v, emax):
    b = bits(v)
    e = (b >> 52) & 0x7FF
    m = ((b & ((1 << 52) - 1)) | (1 << 52)) << 2
    sh = 64 if e == 0 else emax - e
    mag = 0 if sh >= 64 else m >> sh
    return -mag if b >> 63 else mag


def fx_to(s, emax):
    a = abs(s)
    if a == 0:
        return 0.0
    assert a < 2 ** 63
    lz = 64 - a.bit_length()
    n = ((a << (lz - 1)) + 0x200) & (2 ** 64 - 1)
    mh, ml = n >> 42, (n >> 10) & 0xFFFFFFFF
    hw = (((emax + 9 - lz - 1) << 20) + mh) & 0xFFFFFFFF
    return from_bits(((hw | (0x80000000 if s < 0 else 0)) << 32) | ml)


def test_sum_rounds_to_nearest_and_carries_into_the_exponent():
    rng = np.random.default_rng(3)
    cases = [int(rng.integers(-(2 ** 62), 2 ** 62)) >> int(rng.integers(0, 62)) for _ in range(3000)]
    cases += [2 ** 62 - 1, -(2 ** 62 - 1), 2 ** 62 + (2 ** 62 - 1), 2 ** 53 - 1, 1, -1]
    for s in cases:
        emax = int(rng.integers(64, 2030))
        exact = Fraction(s) * Fraction(2) ** (emax - 1077)
        got = fx_to(s, emax)
        if s:
            ulp = Fraction(float(np.nextafter(abs(got), np.inf))) - abs(Fraction(got))
            assert abs(Fraction(got) - exact) <= ulp / 2


@pytest.mark.parametrize("order", [2, 4, 6])
def test_stencil_on_converted_values(order):
    R = order // 2
    rng = np.random.default_rng(order)
    for trial in range(600):
        line = rng.standard_normal(2 * R + 1) * 10.0 ** rng.integers(-20, 3, size=2 * R + 1)
        emax = max(dexp(float(v)) for v in line)
        V = [fx_from(float(v), emax) for v in line]
        S = sum(w * (V[R + k + 1] - V[R - k - 1]) for k, w in enumerate(WEIGHTS[order]))
        assert abs(2 * S) < 2 ** 63  # the sum of the u and v terms fits as well
        exact = sum(COEF[order][s] * Fraction(float(line[s])) for s in range(2 * R + 1)) * DEN[order]
        unit = Fraction(2) ** (emax - 1077)
        bound = 2 * sum(abs(w) for w in WEIGHTS[order]) * unit + abs(exact) * Fraction(1, 2 ** 52)
        assert abs(Fraction(fx_to(S, emax)) - exact) <= bound


def _pair(sbp, kind, order, nx, ny):
    rng = np.random.default_rng(nx * 1000 + ny)
    if kind == "mms":
        return sbp.Context(sbp.WAVE_MMS_2D, order, nx, ny), O.Problem(O.WAVE_MMS_2D, order, nx, ny)
    rho, K = 0.5 + rng.random(nx * ny), 0.5 + rng.random(nx * ny)
    sp, op = ((sbp.WAVE_VAR_2D, O.WAVE_VAR_2D) if kind == "var" else (sbp.WAVE_2BLOCK_2D, O.WAVE_2BLOCK_2D))
    return sbp.Context(sp, order, nx, ny, bc=1, rho=rho, K=K), O.Problem(op, order, nx, ny, bc=1, rho=rho, K=K)


def _close(a, b):
    return np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


# one below, at and above the tile sizes (64 columns; 12 rows variable, 11 manufactured), the
# smallest grids, and two-block halves that end inside a tile
SIZES = [("var", 12, 12), ("var", 63, 12), ("var", 64, 13), ("var", 65, 24), ("var", 131, 25), ("mms", 12, 12),
         ("mms", 64, 11 + 1), ("mms", 65, 22), ("mms", 129, 23), ("two_block", 64, 24), ("two_block", 65, 26),
         ("two_block", 130, 50)]


@pytest.mark.gpu
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("kind,nx,ny", SIZES)
def test_stages_match_the_oracle_at_tile_edges(sbp, port, kind, nx, ny, order):
    ctx, pb = _pair(sbp, kind, order, nx, ny)
    v = np.random.default_rng(order).standard_normal(3 * nx * ny)
    dt = 0.05 / max(nx, ny)
    with ctx:
        assert _close(ctx.rhs(v, 0.3), port.rhs(pb, v, 0.3))
        assert _close(ctx.rk4(v, 0.1, dt, 53), port.rk4(pb, v, 0.1, dt, 53))  # two step graphs


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["var", "mms"])
def test_values_outside_the_fixed_point_range(sbp, port, kind):
    """Values below 2^-959 and from 2^1008, and a NaN point: FP64 taps, as the oracle."""
    ctx, pb = _pair(sbp, kind, 4, 70, 40)
    v = np.random.default_rng(1).standard_normal(3 * 70 * 40)
    with ctx:
        if kind == "var":
            for scale in (2.0 ** -990, 2.0 ** 1010):
                assert _close(ctx.rhs(v * scale), port.rhs(pb, v * scale))
        v[3 * (20 * 70 + 35) + 2] = np.nan
        got, ref = ctx.rhs(v), port.rhs(pb, v)
        # the point's neighbours, and nothing the oracle (whose zero centre tap reads it too) has finite
        assert np.isnan(got).sum() == 8 and not (np.isnan(got) & ~np.isnan(ref)).any()
        assert _close(got[~np.isnan(ref)], ref[~np.isnan(ref)])
