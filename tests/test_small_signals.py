"""Small values beside large ones: every FP64 stage has to be as accurate at a point as FP64
arithmetic on the values that its stencil reads, whatever larger values lie in the same tile,
cell or plane.

The states fall by a factor of 8 per column, 4 per row and 2 per plane, so that a tile holds
values over a hundred binades apart. Result and oracle are compared point by point. The bound:
with |L| the right-hand side's operator of absolute coefficients, one evaluation in FP64 errs by
at most 32 * 2^-53 |L||v| at each point (under 32 roundings on any path from an input to the
result, the integer stencils' units of 2^-54 of the largest value read included); result and
oracle together by twice that. A Runge-Kutta step's bound follows the stages with absolute
coefficients, each stage adding such a term to what the ones before it carry on.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
HINV = {2: 2.0, 4: 48 / 17, 6: 43200 / 13649}
RK4 = ([[], [0.5], [0, 0.5], [0, 0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6])
RKF = ([[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197],
        [439 / 216, -8, 3680 / 513, -845 / 4104], [-8 / 27, 2, -3544 / 2565, 1859 / 4104, -11 / 40]],
       [16 / 135, 0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55])


def abs_d1(port, order, n):
    """|D1| for a unit spacing, from the oracle's 1D operator."""
    pb = O.Problem(O.ADVECTION_1D, order, n, a=-1.0)
    return np.abs(np.stack([port.apply(pb, np.eye(n)[k]) for k in range(n)], axis=1)) / pb.hix


class Bar:
    """v -> |L| v for v >= 0 of shape (nz, ny, nx, dofs) or (ny, nx, dofs); coefficients within 4
    on the boundary terms (rho, K in [0.5, 1.5])."""

    def __init__(self, port, pb):
        self.pb, self.hi = pb, [pb.hix, pb.hiy, pb.hiz]
        two = pb.problem == O.WAVE_2BLOCK_2D
        self.ys = pb.ny // 2 if two else 0
        self.d = [abs_d1(port, pb.order, pb.nx) * pb.hix]
        if two:
            half = abs_d1(port, pb.order, self.ys) * pb.hiy
            self.d.append(np.kron(np.eye(2), half))
        elif pb.ny > 1:
            self.d.append(abs_d1(port, pb.order, pb.ny) * pb.hiy)
        if pb.nz > 1:
            self.d.append(abs_d1(port, pb.order, pb.nz) * pb.hiz)

    def along(self, v, k):
        ax = len(self.d) - 1 - k
        return np.moveaxis(np.tensordot(self.d[k], v, axes=(1, ax)), 0, ax)

    def __call__(self, v):
        pb, nd = self.pb, len(self.d)
        out = np.zeros_like(v)
        if pb.problem == O.ADVECTION_2D:
            a = abs(pb.a) if pb.a_field is None else np.abs(pb.a_field.reshape(pb.ny, pb.nx))
            b = abs(pb.b) if pb.b_field is None else np.abs(pb.b_field.reshape(pb.ny, pb.nx))
            u = v[..., 0]
            out[..., 0] = a * self.along(u, 0) + b * self.along(u, 1)
            c = 4.0
        else:
            ri = kk = 1.0
            if pb.problem == O.WAVE_MMS_2D:
                x, y = np.linspace(-1, 1, pb.nx)[None, :], np.linspace(-1, 1, pb.ny)[:, None]
                ri = 1 / (2 + x * y)
            elif pb.rho is not None:
                ri, kk = 1 / pb.rho.reshape(pb.ny, pb.nx), pb.K.reshape(pb.ny, pb.nx)
            for k in range(nd):
                out[..., k] = ri * self.along(v[..., nd], k)
                out[..., nd] += kk * self.along(v[..., k], k)
            c = 4.0
        for k in range(nd):  # boundary terms on the two faces across direction k
            ax = nd - 1 - k
            for at in (0, v.shape[ax] - 1):
                sel = tuple([slice(None)] * ax + [at])
                if v.shape[-1] == 1:
                    out[sel][..., 0] += c * self.hi[k] * HINV[pb.order] * v[sel][..., 0]
                else:
                    g = c * self.hi[k] * HINV[pb.order] * (v[sel][..., nd] + v[sel][..., k])
                    out[sel][..., nd] += g
                    out[sel][..., k] += g
        if self.ys:
            both = v[self.ys - 1] + v[self.ys]
            g = c * self.hi[1] * HINV[pb.order] * (both[..., 2] + both[..., 1])
            for j in (self.ys - 1, self.ys):
                out[j, :, 2] += g
                out[j, :, 1] += g
        return out


def steep(shape, seed, fall=(3, 2, 1), top=0):
    """Random signs and mantissas; exponents fall along x, y, z; components 2^-20 apart."""
    rng = np.random.default_rng(seed)
    e = np.full(shape, float(top))
    for k in range(len(shape) - 1):
        ax = len(shape) - 2 - k
        sh = [1] * len(shape)
        sh[ax] = -1
        e = e - fall[k] * np.arange(shape[ax]).reshape(sh)
    e = e - 20.0 * np.arange(shape[-1])
    return rng.choice([-1.0, 1.0], shape) * rng.uniform(0.5, 1.0, shape) * 2.0 ** e


def step_bound(bar, tableau, v, f, dt):
    """Bound of result minus oracle after one step from v (f: |forcing|)."""
    rows, b = tableau
    stages = len(rows)
    w, e, k, ek = None, None, [], []
    for row in rows:
        w = np.abs(v) + dt * sum((abs(c) * q for c, q in zip(row, k)), np.zeros_like(v))
        e = 16 * EPS * w + dt * sum((abs(c) * q for c, q in zip(row, ek)), np.zeros_like(v))
        k.append(bar(w) + f)
        ek.append(64 * EPS * (bar(w) + f) + bar(e))
    out = np.abs(v) + dt * sum(abs(c) * q for c, q in zip(b, k))
    assert stages == len(k)
    return 32 * EPS * out + dt * sum(abs(c) * q for c, q in zip(b, ek))


def within(got, ref, bound, shape):
    got, ref = got.reshape(shape), ref.reshape(shape)
    assert np.isfinite(got).all()
    worst = np.max(np.abs(got - ref) / bound)
    assert worst <= 1.0, worst


def pair(sbp, kind, order, nx, ny, bc):
    rng = np.random.default_rng(nx + ny)
    name = {"hom": "WAVE_HOM_2D", "var": "WAVE_VAR_2D", "two_block": "WAVE_2BLOCK_2D", "mms": "WAVE_MMS_2D"}[kind]
    kw = {"bc": bc}
    if kind in ("var", "two_block"):
        kw.update(rho=0.5 + rng.random(nx * ny), K=0.5 + rng.random(nx * ny))
    return sbp.Context(getattr(sbp, name), order, nx, ny, **kw), O.Problem(getattr(O, name), order, nx, ny, **kw)


@pytest.mark.parametrize("form", [0, 1, 2], ids=["whole_steps", "persistent", "cells"])
@pytest.mark.parametrize("order", [2, 4, 6])
@pytest.mark.parametrize("kind,nx,ny", [("var", 67, 38), ("two_block", 66, 50), ("mms", 67, 38), ("hom", 67, 38)])
def test_wave_2d(sbp, port, kind, nx, ny, order, form):
    bc = 0 if kind == "mms" or order == 4 else 1
    ctx, pb = pair(sbp, kind, order, nx, ny, bc)
    shape = (ny, nx, 3)
    v = steep(shape, order, top=60 if kind == "mms" else 0)  # the forcing of order 10 far below
    bar = Bar(port, pb)
    t, dt = 0.3, 0.1 / max(nx, ny)
    f = np.abs(port.rhs(pb, np.zeros(v.size), t)).reshape(shape)
    fmax = np.abs(port.rhs(pb, np.zeros(v.size), 0.0)).reshape(shape) if kind == "mms" else f
    with ctx:
        ctx.test_wave_form(form)
        if kind != "hom":
            within(ctx.rhs(v.ravel(), t), port.rhs(pb, v.ravel(), t), 64 * EPS * (bar(np.abs(v)) + f), shape)
        if kind != "hom" or form == 0:  # constant coefficients stage by stage: box units (wave2d_fixed.cuh)
            within(ctx.rk4(v.ravel(), t, dt, 1), port.rk4(pb, v.ravel(), t, dt, 1),
                   step_bound(bar, RK4, v, fmax, dt), shape)
        if form:
            ctx.set_state(v.ravel())
            st = ctx.rk45_resident(t, t + dt, dt, atol=1e30, rtol=0.0)
            assert st["accepted"] == 1
            ref = port.rk45(pb, v.ravel(), t, t + dt, dt, atol=1e30, rtol=0.0)[0]
            within(ctx.get_state(), ref, step_bound(bar, RKF, v, fmax, dt), shape)


@pytest.mark.parametrize("field", [False, True], ids=["constant", "field"])
@pytest.mark.parametrize("order", [2, 4, 6])
def test_advection_2d(sbp, port, order, field):
    # the line form at order 2, cells of one row per thread, of two (constant velocities), of two
    for nx, ny in ((205, 203), (411, 401), (703, 651), (1101, 1001), (1056, 1072)):
        kw = {"a": 1.5, "b": -1.0}
        if field:
            rng = np.random.default_rng(nx)
            kw.update(a_field=rng.uniform(-1, 1, nx * ny), b_field=rng.uniform(-1, 1, nx * ny))
        pb = O.Problem(O.ADVECTION_2D, order, nx, ny, **kw)
        shape = (ny, nx, 1)
        v = steep(shape, order, fall=(300 / nx, 200 / ny), top=0)
        v *= 2.0 ** -(8.0 * (np.arange(nx) % 32))[None, :, None]  # and within every cell
        bar, dt = Bar(port, pb), 0.05 / nx
        with sbp.Context(sbp.ADVECTION_2D, order, nx, ny, **kw) as ctx:
            within(ctx.rhs(v.ravel()), port.rhs(pb, v.ravel()), 64 * EPS * bar(np.abs(v)), shape)
            within(ctx.rk4(v.ravel(), 0.0, dt, 1), port.rk4(pb, v.ravel(), 0.0, dt, 1),
                   step_bound(bar, RK4, v, 0.0, dt), shape)


@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("order", [2, 4, 6])
def test_wave_3d(sbp, port, order, bc):
    nx, ny, nz = 66, 21, 19
    pb = O.Problem(O.WAVE_3D, order, nx, ny, nz=nz, bc=bc)
    shape = (nz, ny, nx, 4)
    bar, dt = Bar(port, pb), 0.1 / nx
    for fall in ((3, 2, 1), (1, 2, 9)):
        v = steep(shape, order, fall=fall)
        with sbp.Context(sbp.WAVE_3D, order, nx, ny, nz, bc=bc) as ctx:
            within(ctx.rhs(v.ravel()), port.rhs(pb, v.ravel()), 64 * EPS * bar(np.abs(v)), shape)
            within(ctx.rk4(v.ravel(), 0.0, dt, 1), port.rk4(pb, v.ravel(), 0.0, dt, 1),
                   step_bound(bar, RK4, v, 0.0, dt), shape)


@pytest.mark.parametrize("order", [2, 4, 6])
def test_line_steps(sbp, port, order):
    """1D step loops: a steep line, and a stretch of subnormal values, whose products round at
    2^-1074 (up to 16 of them per stage and point, each times dt)."""
    n = 150
    pb = O.Problem(O.ADVECTION_1D, order, n)
    bar, dt = Bar(port, pb), 0.1 / n
    shape = (n, 1)
    rng = np.random.default_rng(order)
    for v in (steep(shape, order, fall=(5,)), rng.uniform(0.5, 1.0, shape) * 2.0 ** -1030,
              rng.uniform(0.5, 1.0, shape) * 2.0 ** np.where(np.arange(n) < 70, -1030.0, -900.0)[:, None]):
        with sbp.Context(sbp.ADVECTION_1D, order, n) as ctx:
            bound = step_bound(lambda w: bar_1d(bar, pb, w), RK4, v, 0.0, dt) + 64 * 2.0 ** -1074
            within(ctx.rk4(v.ravel(), 0.0, dt, 1), port.rk4(pb, v.ravel(), 0.0, dt, 1), bound, shape)


def bar_1d(bar, pb, v):
    out = bar.d[0] @ v
    for at in (0, -1):
        out[at] += pb.hix * HINV[pb.order] * v[at]
    return out
