"""Grids with few columns and more rows than a grid of 32 x 8 cells can have (65535 rows of
cells): the 2D wave stages take the persistent form whatever the number of points. The largest
grid of cells, one row more, and the most rows whose points would still call for cells.

Tolerance 1e-12 (max norm, relative), as the other FP64 parity tests.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,ny", [("var", 524280), ("var", 524281), ("var", 533333), ("mms", 533333),
                                     ("two_block", 533332)])
def test_narrow_grids(sbp, port, kind, ny):
    nx, kw = 3, {}
    if kind != "mms":
        rng = np.random.default_rng(ny)
        kw = {"bc": 1, "rho": 0.5 + rng.random(nx * ny), "K": 0.5 + rng.random(nx * ny)}
    name = {"var": "WAVE_VAR_2D", "mms": "WAVE_MMS_2D", "two_block": "WAVE_2BLOCK_2D"}[kind]
    pb = O.Problem(getattr(O, name), 2, nx, ny, **kw)
    v = np.random.default_rng(1).standard_normal(3 * nx * ny)
    dt = 0.1 / ny
    with sbp.Context(getattr(sbp, name), 2, nx, ny, **kw) as ctx:
        for got, ref in ((ctx.rhs(v, 0.1), port.rhs(pb, v, 0.1)),
                         (ctx.rk4(v, 0.0, dt, 2), port.rk4(pb, v, 0.0, dt, 2))):
            assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
        ctx.set_state(v)
        st = ctx.rk45_resident(0.0, 2 * dt, dt, atol=1e3, rtol=0.0)
        got = ctx.get_state()
    ref, rst = port.rk45(pb, v, 0.0, 2 * dt, dt, atol=1e3, rtol=0.0)
    assert (st["accepted"], st["rejected"]) == (rst["accepted"], rst["rejected"])
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
