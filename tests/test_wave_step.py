"""Whole RK4 steps of small FP64 2D wave grids in one launch (csrc/wave_step.cuh).

CPU: the intervals a cell's stages read, restated, fit the box the kernel keeps, hold every
stencil, closure block and interface partner, and lie on the grid, for every cell of many line
lengths. GPU: the step against the oracle (1e-12 relative max norm, the bar of the other FP64
parity tests) around the cells' sides and the line to the stage-by-stage form, odd and even
step counts over several step graphs, and outside the fixed-point range.
"""
import numpy as np
import pytest

import oracle as O

SHAPE = {2: (1, 1, 2), 4: (2, 4, 6), 6: (3, 6, 9)}  # reach, closure rows, closure width
MIN = {2: 3, 4: 8, 6: 12}


def reads(order, lo, hi, n, split):
    R, CS, CW = SHAPE[order]
    a, b = lo - R, hi + R
    for s, e in ([(0, split), (split, n)] if split else [(0, n)]):
        if lo < s + CS and hi > s:
            b, a = max(b, s + CW), min(a, s)
        if hi > e - CS and lo < e:
            a, b = min(a, e - CW), max(b, e)
    return max(a, 0), min(b, n)


def needed(order, i, n, split):
    """Points the derivative (and interface SAT) of point i reads."""
    R, CS, CW = SHAPE[order]
    s, e = (0, n) if not split else ((0, split) if i < split else (split, n))
    if i < s + CS:
        r = set(range(s, s + CW))
    elif i >= e - CS:
        r = set(range(e - CW, e))
    else:
        r = set(range(i - R, i + R + 1))
    if split and i in (split - 1, split):
        r |= {split - 1, split}
    return r | {i}


@pytest.mark.parametrize("order,T", [(2, 16), (2, 24), (4, 16), (4, 24), (6, 16), (6, 20)])
def test_boxes_hold_what_the_stages_read(order, T):
    R, CS, CW = SHAPE[order]
    M = 3 * R + max(R, CS - 1)
    P = T + max(2 * M, 7 * R + CW)
    lengths = list(range(MIN[order], 90))
    for n, split in [(n, 0) for n in lengths] + [(2 * h, h) for h in range(MIN[order], 70)]:
        for c in range(0, n, T):
            lo, hi = c, min(c + T, n)
            for _ in range(4):
                a, b = reads(order, lo, hi, n, split)
                assert 0 <= a <= lo and hi <= b <= n
                for i in (lo, hi - 1, *range(lo, hi, 3)):
                    assert needed(order, i, n, split) <= set(range(a, b)), (n, split, c, i)
                lo, hi = a, b
            assert hi - lo <= P, (n, split, c, hi - lo, P)


def _pair(sbp, kind, order, nx, ny, bc):
    rng = np.random.default_rng(nx + ny)
    names = {"hom": "WAVE_HOM_2D", "var": "WAVE_VAR_2D", "two_block": "WAVE_2BLOCK_2D", "mms": "WAVE_MMS_2D"}
    kw = {"bc": bc}
    if kind in ("var", "two_block"):
        kw.update(rho=0.5 + rng.random(nx * ny), K=0.5 + rng.random(nx * ny))
    return (sbp.Context(getattr(sbp, names[kind]), order, nx, ny, **kw),
            O.Problem(getattr(O, names[kind]), order, nx, ny, **kw))


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


# around cells of 16, 20 and 24 points, and the last and first sizes on either side of 152 of the
# larger cells (two of them per row fewer or more at order 6)
SIZES = [(12, 24), (15, 26), (16, 32), (17, 34), (33, 48), (65, 50), (161, 130), (240, 200), (264, 264), (288, 290)]


@pytest.mark.gpu
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("kind", ["hom", "var", "two_block", "mms"])
def test_steps_match_the_oracle(sbp, port, kind, order):
    for n, (nx, ny) in enumerate(SIZES):
        bc = 0 if kind == "mms" else n % 2
        ctx, pb = _pair(sbp, kind, order, nx, ny, bc)
        v = port.init_wave_pulse(nx, ny, 0.1, -0.1, 0.4, 1.0)
        v = v + 0.05 * np.random.default_rng(n).standard_normal(v.size)
        dt = 0.1 / max(nx, ny)
        with ctx:
            for steps in (1, 4) + ((53,) if nx < 40 else ()):  # 53: two step graphs, an odd one last
                assert _rel(ctx.rk4(v, 0.2, dt, steps), port.rk4(pb, v, 0.2, dt, steps)) < 1e-12


@pytest.mark.gpu
def test_unequal_spacings(sbp, port):
    with sbp.Context(sbp.WAVE_HOM_2D, 4, 70, 41, bc=1, xl=(-1.0, 0.0), xr=(1.0, 3.0)) as ctx:
        pb = O.Problem(O.WAVE_HOM_2D, 4, 70, 41, bc=1, xl=(-1.0, 0.0, -1.0), xr=(1.0, 3.0, 1.0))
        v = np.random.default_rng(3).standard_normal(3 * 70 * 41)
        assert _rel(ctx.rk4(v, 0.0, 1e-3, 6), port.rk4(pb, v, 0.0, 1e-3, 6)) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["hom", "var", "two_block"])
def test_values_outside_the_fixed_point_range(sbp, port, kind):
    nx, ny = 40, 38
    ctx, pb = _pair(sbp, kind, 4, nx, ny, 1)
    v = np.random.default_rng(1).standard_normal(3 * nx * ny)
    with ctx:
        for scale in (2.0 ** -990, 2.0 ** 1012):
            assert _rel(ctx.rk4(v * scale, 0.0, 1e-3, 2), port.rk4(pb, v * scale, 0.0, 1e-3, 2)) < 1e-12
        assert not ctx.rk4(0.0 * v, 0.0, 1e-3, 3).any()
        v[3 * (19 * nx + 20)] = np.inf
        got = ctx.rk4(v, 0.0, 1e-3, 1)
        assert np.isfinite(got.reshape(ny, nx, 3)[:8]).all()  # four reaches per stage, not the grid
