"""The bounded waits of the FP64 3D wave kernel: a CTA whose first planes are never loaded
(sbp_test_drop_tile) lets its wait run out after the context's limit, the call returns
SBP_ERR_DEVICE, and the same context then gives the oracle's results. Nothing faults, traps or
hangs the GPU: the missing load is never issued, and every wait has a limit.
"""
import time

import numpy as np
import pytest

import oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("cta", [0, 17])
@pytest.mark.parametrize("order", [2, 4, 6])
def test_a_wait_that_runs_out(sbp, port, order, cta):
    nx, ny, nz = 66, 40, 30
    pb = O.Problem(O.WAVE_3D, order, nx, ny, nz=nz)
    v = np.random.default_rng(order).standard_normal(4 * nx * ny * nz)
    ref = port.rhs(pb, v)
    with sbp.Context(sbp.WAVE_3D, order, nx, ny, nz) as c:
        c.set_wait_limit(5_000_000)  # 5 ms: a plane's load takes microseconds
        for _ in range(2):
            c.test_drop_tile(cta)
            t = time.perf_counter()
            with pytest.raises(sbp.SbpError) as e:
                c.rhs(v)
            assert e.value.code == sbp.ERR_DEVICE and "timed out" in str(e.value)
            assert time.perf_counter() - t < 0.15  # the context's limit, not the default 200 ms
            assert np.max(np.abs(c.rhs(v) - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.gpu
def test_the_aid_has_bounds(sbp):
    with sbp.Context(sbp.WAVE_3D, 4, 40, 40, 40) as c:
        for tile in (-1, 10 ** 6):
            with pytest.raises(sbp.SbpError) as e:
                c.test_drop_tile(tile)
            assert e.value.code == sbp.ERR_INVALID
    with sbp.Context(sbp.WAVE_3D, 4, 40, 40, 40, precision=sbp.FP32) as c:
        with pytest.raises(sbp.SbpError):
            c.test_drop_tile(0)
