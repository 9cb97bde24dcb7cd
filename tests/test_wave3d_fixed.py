"""The FP64 3D wave stages with integer stencils against the oracle: sizes one below, at and
above the tile (32 x 8 columns) and the planes of a CTA (4 to 12), states whose magnitude
changes from plane to plane (the z stencil then shifts values to a common exponent), planes of
zeros, and values outside the fixed-point range (FP64 taps).

Tolerance 1e-12 (max norm, relative), as the other FP64 parity tests; a state whose planes
differ in magnitude is compared plane by plane, each with the largest value within a stencil's
reach.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(12, 12, 12), (31, 15, 13), (32, 16, 24), (33, 17, 25), (65, 12, 37), (40, 70, 49)]


def _close(a, b):
    return np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("order", [2, 4, 6])
def test_tile_edges(sbp, port, order, bc):
    for nx, ny, nz in SIZES:
        pb = O.Problem(O.WAVE_3D, order, nx, ny, nz=nz, bc=bc)
        v = np.random.default_rng(nx).standard_normal(4 * nx * ny * nz)
        dt = 0.02 / max(nx, ny, nz)
        with sbp.Context(sbp.WAVE_3D, order, nx, ny, nz, bc=bc) as ctx:
            assert _close(ctx.rhs(v), port.rhs(pb, v))
            assert _close(ctx.rk4(v, 0.0, dt, 3), port.rk4(pb, v, 0.0, dt, 3))


@pytest.mark.parametrize("order", [2, 4, 6])
def test_planes_of_different_magnitude(sbp, port, order):
    nx, ny, nz = 34, 18, 40
    rng = np.random.default_rng(order)
    scale = 10.0 ** rng.integers(-9, 3, size=nz)
    scale[20:24] = 0.0
    v = rng.standard_normal((nz, ny, nx, 4)) * scale[:, None, None, None]
    pb = O.Problem(O.WAVE_3D, order, nx, ny, nz=nz)
    with sbp.Context(sbp.WAVE_3D, order, nx, ny, nz) as ctx:
        got = ctx.rhs(v.ravel()).reshape(v.shape)
    ref = port.rhs(pb, v.ravel()).reshape(v.shape)
    reach = 9  # closure rows read up to 9 planes
    for k in range(nz):
        near = np.max(np.abs(v[max(0, k - reach):k + reach + 1])) * max(nx, ny, nz)
        assert np.max(np.abs(got[k] - ref[k])) <= 1e-12 * near


def test_values_outside_the_fixed_point_range(sbp, port):
    nx, ny, nz = 34, 18, 20
    pb = O.Problem(O.WAVE_3D, 4, nx, ny, nz=nz)
    v = np.random.default_rng(1).standard_normal(4 * nx * ny * nz)
    with sbp.Context(sbp.WAVE_3D, 4, nx, ny, nz) as ctx:
        for scale in (2.0 ** -990, 2.0 ** 1010, 0.0):
            assert _close(ctx.rhs(v * scale), port.rhs(pb, v * scale))
        w = v.reshape(nz, ny, nx, 4).copy()
        w[10, 9, 15, 3] = np.inf
        got = ctx.rhs(w.ravel())
        assert (~np.isfinite(got)).sum() == 12  # four neighbours along each direction
