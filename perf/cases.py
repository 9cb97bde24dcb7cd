"""The calls this library is used for, as timed cases.

Each case is one call (or one set / step / read-back sequence) through the public Python binding
(hpc-reading-course_gb300/python/sbpgpu.py) at sizes that the reference's demos, this repository's
studies and its tests use, plus `draw` for others of the same ranges. `exact` restates the
operators in plain torch FP64 for the comparison.
"""
import math
import os
import sys

import numpy as np
import torch

_PY = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hpc-reading-course_gb300", "python")
if _PY not in sys.path:
    sys.path.insert(0, _PY)

import sbpgpu  # noqa: E402

DEV = "cuda:0"
PROBLEM = {"hom": sbpgpu.WAVE_HOM_2D, "mms": sbpgpu.WAVE_MMS_2D, "var": sbpgpu.WAVE_VAR_2D,
           "two_block": sbpgpu.WAVE_2BLOCK_2D, "advection_1d": sbpgpu.ADVECTION_1D,
           "advection_2d": sbpgpu.ADVECTION_2D, "reflection_1d": sbpgpu.REFLECTION_1D, "wave_3d": sbpgpu.WAVE_3D}
DOFS = {"advection_1d": 1, "advection_2d": 1, "reflection_1d": 2, "wave_3d": 4}


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the reference's 1D advection demo: 201 points to T = 1.8 at CFL 0.1 from host arrays
        # (1800 steps of a tiny grid: the smallest call, all latency)
        _case("advection_1d", "advection_1d_demo", order=4, nx=201, steps=1800, cfl=0.1, host=True),
        # the reference's 2D advection demo (a = 1.5, b = -1), an ordinary grid
        _case("advection_2d", "advection_2d_801", order=4, nx=801, ny=801, steps=100),
        # the reference's forced wave demo on the grid its convergence rows end at, host arrays
        _case("mms", "wave_forced_161", order=4, nx=161, ny=161, steps=150, host=True),
        # the right-hand side as a host framework's time stepper calls it, once per stage, on a
        # device vector; an odd size, the widest stencil
        _case("hom", "wave_rhs_callback", call="rhs", order=6, nx=1025, ny=1023, bc="free"),
        # the coarse two-layer solve of the learned correction: 257 x 2*129, four windows of 4 steps
        _case("two_block", "two_layer_coarse", order=4, nx=257, ny=258, steps=16, bc="char"),
        # the plain wave at 1024^2 with the lowest order
        _case("hom", "wave_1024_o2", order=2, nx=1024, ny=1024, steps=50, bc="free"),
        # the headline grid: 4096^2, order 4, characteristic boundaries, FP64
        _case("hom", "wave_4096_fp64", order=4, nx=4096, ny=4096, steps=20, bc="char"),
        # variable density and bulk modulus in compensated FP32, the long-run form of the headline grid
        _case("var", "wave_var_4096_fp32", order=4, nx=4096, ny=4096, steps=20, bc="char", precision="fp32"),
        # the 3D wave in FP64, an odd box
        _case("wave_3d", "wave_3d_fp64", order=4, nx=201, ny=193, nz=161, steps=10, bc="char"),
        # the adaptive integrator with default tolerances over a short interval
        _case("hom", "wave_rk45", call="rk45", order=4, nx=1024, ny=1024, steps=40, bc="char"),
        # many uneven independent instances (waves and advection, all orders) advanced together
        {"name": "batch_48_fp32", "kind": "batch", "count": 48, "pick": 2, "steps": 300, "precision": "fp32"},
        # one training step of the correction network at the learned study's shape
        {"name": "network_train", "kind": "network_train", "batch": 8, "height": 258, "width": 257},
    ]


def _case(kind, name=None, *, call="rk4", order, nx, ny=1, nz=1, steps=1, bc="free", precision="fp64", cfl=0.2,
          host=False, fields=False):
    c = {"kind": kind, "call": call, "order": order, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "bc": bc,
         "precision": precision, "cfl": cfl, "host": host, "fields": fields}
    if name:
        c["name"] = name
    return c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(rng, points, budget, most):
    """A step count that keeps points x steps under `budget`."""
    return max(3, min(_log_int(rng, max(3, most // 10), most), int(budget // points)))


def draw(rng):
    kind = rng.choice(["line", "advection_2d", "mms", "rhs", "two_block", "hom", "hom", "var", "wave_3d", "rk45",
                       "batch", "network_train", "network_forward"])
    order = rng.choice([2, 4, 6])
    precision = rng.choice(["fp64", "fp64", "fp32"])
    bc = rng.choice(["free", "char"])
    if kind == "line":
        return _case(rng.choice(["advection_1d", "reflection_1d"]), order=order, nx=_log_int(rng, 51, 6401),
                     steps=_log_int(rng, 100, 2000), cfl=0.1, host=rng.random() < 0.5, precision=precision,
                     fields=rng.random() < 0.25)
    if kind == "advection_2d":
        nx, ny = _log_int(rng, 101, 2001), _log_int(rng, 101, 2001)
        return _case(kind, order=order, nx=nx, ny=ny, steps=_steps(rng, nx * ny, 1e8, 200), precision=precision,
                     fields=rng.random() < 0.25)
    if kind == "mms":
        nx, ny = _log_int(rng, 41, 1001), _log_int(rng, 41, 1001)
        return _case(kind, order=order, nx=nx, ny=ny, steps=_steps(rng, nx * ny, 2e7, 200), host=rng.random() < 0.5)
    if kind == "rhs":
        return _case(rng.choice(["hom", "var"]), call="rhs", order=order, nx=_log_int(rng, 65, 2500),
                     ny=_log_int(rng, 65, 2500), bc=bc, precision=precision)
    if kind == "two_block":
        nx, ny = _log_int(rng, 129, 1025), 2 * _log_int(rng, 65, 513)
        return _case(kind, order=order, nx=nx, ny=ny, steps=_steps(rng, nx * ny, 3e7, 100), bc=bc,
                     precision=precision)
    if kind in ("hom", "var"):
        nx, ny = _log_int(rng, 101, 4096), _log_int(rng, 101, 4096)
        return _case(kind, order=order, nx=nx, ny=ny, steps=_steps(rng, nx * ny, 1.5e8, 200), bc=bc,
                     precision=precision, host=nx * ny < 300000 and rng.random() < 0.3)
    if kind == "wave_3d":
        nx, ny, nz = (_log_int(rng, 40, 220) for _ in range(3))
        return _case(kind, order=order, nx=nx, ny=ny, nz=nz, steps=_steps(rng, nx * ny * nz, 6e7, 50), bc=bc,
                     precision=precision)
    if kind == "rk45":
        nx, ny = _log_int(rng, 101, 1200), _log_int(rng, 101, 1200)
        return _case(rng.choice(["hom", "var"]), call="rk45", order=order, nx=nx, ny=ny,
                     steps=_steps(rng, nx * ny, 3e7, 60), bc=bc)
    if kind == "batch":
        return {"kind": "batch", "count": _log_int(rng, 8, 64), "pick": rng.randrange(1000),
                "steps": _log_int(rng, 100, 300), "precision": precision}
    return {"kind": kind, "batch": rng.randint(1, 8), "height": _log_int(rng, 33, 260), "width": _log_int(rng, 33, 260)}


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return np.random.default_rng(seed)


def _dims(case):
    k = case["kind"]
    n = [case["nx"]]
    if k not in ("advection_1d", "reflection_1d"):
        n.append(case["ny"])
    if k == "wave_3d":
        n.append(case["nz"])
    return n


def _spacing(case):
    """Grid spacing per direction on [-1, 1] (two-block: each block half the height)."""
    h = [2.0 / (n - 1) for n in _dims(case)]
    if case["kind"] == "two_block":
        h[1] = 1.0 / (case["ny"] // 2 - 1)
    return h


def _axes(case):
    """Point coordinates per direction as device tensors."""
    ax = [torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device=DEV) for n in _dims(case)]
    if case["kind"] == "two_block":
        m = case["ny"] // 2
        lo = torch.linspace(-1.0, 0.0, m, dtype=torch.float64, device=DEV)
        ax[1] = torch.cat([lo, lo + 1.0])
    return ax


def _initial(case, seed):
    """A pulse (width 0.05 to 0.2) off centre plus a smooth background, AoS FP64 on the device."""
    r = _gen(seed)
    k = case["kind"]
    ax = _axes(case)
    c = r.uniform(-0.5, 0.5, len(ax))
    w = r.uniform(0.05, 0.2)
    ph = r.uniform(0, 2 * math.pi, 8)
    pulse, back = None, None
    for d, x in enumerate(ax):  # x innermost
        shape = [1] * len(ax)
        shape[len(ax) - 1 - d] = -1
        g = torch.exp(-((x - c[d]) / w) ** 2).reshape(shape)
        s = torch.cos((2 + d) * math.pi * x + ph[d]).reshape(shape)
        pulse = g if pulse is None else pulse * g
        back = s if back is None else back * s
    full = pulse + 0.05 * back
    dofs = DOFS.get(k, 3)
    if k == "mms":  # the manufactured solution's own initial state
        x, y = ax[0][None, :], ax[1][:, None]
        return torch.stack([torch.zeros_like(full), torch.zeros_like(full),
                            torch.sin(3 * math.pi * x) * torch.sin(4 * math.pi * y)
                            * (1 + 0.1 * math.cos(ph[0]))], -1).contiguous()
    out = torch.empty(full.shape + (dofs,), dtype=torch.float64, device=DEV)
    for q in range(dofs):
        out[..., q] = (full if q == dofs - 1 else 0.2 * back * math.cos(ph[q + 4]))
    return out


def _coefficients(case, seed):
    """rho, K in (0.5, 1.5) (a jump of 4 across the interface for two blocks), host arrays."""
    ax = [a.cpu().numpy() for a in _axes(case)]
    ph = _gen(seed + 77).uniform(0, 2 * math.pi, 4)
    if case["kind"] == "two_block":
        up = (np.arange(case["ny"]) >= case["ny"] // 2)[:, None] * np.ones((1, case["nx"]))
        f = np.where(up > 0, 4.0, 1.0)
        return f, f.copy()
    rho = 1 + 0.45 * np.cos(3 * ax[1] + ph[0])[:, None] * np.sin(4 * ax[0] + ph[1])[None, :]
    K = 1 + 0.45 * np.sin(5 * ax[1] + ph[2])[:, None] * np.cos(2 * ax[0] + ph[3])[None, :]
    return rho, K


def _velocities(case):
    """Velocity at every point (1D: positive inflow on the left; 2D: a rotation-like field)."""
    ax = [a.cpu().numpy() for a in _axes(case)]
    if len(ax) == 1:
        return 1.0 + 0.3 * np.sin(3 * ax[0]), None
    x, y = ax[0][None, :], ax[1][:, None]
    return 1.0 + 0.5 * np.sin(2 * y) + 0 * x, -0.8 + 0.3 * np.cos(2 * x) + 0 * y


def _dt(case):
    h = min(_spacing(case))
    cmax = {"advection_1d": 1.5, "advection_2d": 2.0, "var": 1.7}.get(case["kind"], 1.0)
    return case["cfl"] * h / cmax


def _cells(case):
    return math.prod(_dims(case))


def _batch_list(case):
    r = _gen(case["pick"])
    out = []
    for k in range(case["count"]):
        nx, ny = (int(round(math.exp(r.uniform(math.log(64), math.log(512))))) for _ in range(2))
        c = float(r.uniform(0.5, 2.0))
        h = min(2.0 / (nx - 1), 2.0 / (ny - 1))
        d = dict(order=int(r.choice([2, 4, 6])), nx=nx, ny=ny, dt=0.2 * h / c)
        if k % 2 == 0:
            d.update(problem=sbpgpu.WAVE_HOM_2D, c=c, bc=sbpgpu.BC_CHARACTERISTIC)
        else:
            ang = float(r.uniform(0, 2 * math.pi))
            d.update(problem=sbpgpu.ADVECTION_2D, a=c * math.cos(ang), b=c * math.sin(ang))
        out.append(d)
    return out


def _batch_states(insts, seed):
    r = _gen(seed)
    states = []
    for d in insts:
        x = np.linspace(-1, 1, d["nx"]) - r.uniform(-0.5, 0.5)
        y = np.linspace(-1, 1, d["ny"]) - r.uniform(-0.5, 0.5)
        g = np.exp(-(x / 0.1) ** 2)[None, :] * np.exp(-(y / 0.1) ** 2)[:, None]
        if d["problem"] == sbpgpu.WAVE_HOM_2D:
            v = np.zeros(g.shape + (3,))
            v[..., 2] = g
            states.append(v.ravel())
        else:
            states.append(g.ravel())
    return states


def _network_io(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    b, h, w = case["batch"], case["height"], case["width"]
    x = torch.randn((b, h, w, 24), generator=g, device=DEV)
    t = 0.1 * torch.randn((b, h, w, 3), generator=g, device=DEV)
    return x, t


def _network_weights(seed, count):
    """Weights and biases as after some training: He-normal layers, a small output layer."""
    r = _gen(seed + 5)
    v = np.zeros(count, dtype=np.float32)
    o = 0
    for cin, cout, last in ((32, 32, False), (32, 32, False), (32, 32, False), (32, 16, True)):
        w = r.standard_normal((cout, 9, cin)) * math.sqrt(2.0 / (9 * cin)) * (0.3 if last else 1.0)
        if o == 0:
            w[:, :, 24:] = 0
        if last:
            w[3:] = 0
        v[o:o + w.size] = w.ravel()
        o += w.size + cout
    return v


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.kind = case, case["kind"]
    if s.kind == "batch":
        s.insts = _batch_list(case)
        s.states = _batch_states(s.insts, seed)
        s.handle = sbpgpu.Batch(s.insts, precision=sbpgpu.FP32 if case["precision"] == "fp32" else sbpgpu.FP64)
        return s
    if s.kind.startswith("network"):
        s.x, s.target = _network_io(case, seed)
        s.handle = sbpgpu.Cnn(case["height"], case["width"], case["batch"])
        s.handle.set_params(_network_weights(seed, s.handle.param_count()))
        s.out = torch.empty_like(s.target)
        return s
    kw = {}
    if s.kind in ("var", "two_block"):
        kw["rho"], kw["K"] = _coefficients(case, seed)
    if s.kind.startswith("advection"):
        kw["a"], kw["b"] = 1.5 if s.kind == "advection_2d" else 1.0, -1.0
        if case["fields"]:
            kw["a_field"], kw["b_field"] = _velocities(case)
    bc = sbpgpu.BC_CHARACTERISTIC if case["bc"] == "char" else sbpgpu.BC_REFERENCE
    s.handle = sbpgpu.Context(PROBLEM[s.kind], case["order"], case["nx"], case["ny"], case["nz"], bc=bc,
                              precision=sbpgpu.FP32 if case["precision"] == "fp32" else sbpgpu.FP64, **kw)
    s.v0 = _initial(case, seed)
    s.dt = _dt(case)
    s.t_end = s.dt * case["steps"]
    s.out = torch.empty_like(s.v0)
    if case["host"]:
        s.host = s.v0.cpu().numpy().ravel()
    return s


def run(s):
    c, h = s.case, s.handle
    if s.kind == "batch":
        for k, v in enumerate(s.states):
            h.set_state(k, v)
        h.step_resident(c["steps"])
        return np.concatenate([h.get_state(k) for k in range(len(s.states))])
    if s.kind == "network_train":
        loss = h.train_step(s.x.data_ptr(), s.target.data_ptr(), c["batch"], 1e-4)
        return {"loss": loss, "params": h.get_params()}
    if s.kind == "network_forward":
        h.forward(s.x.data_ptr(), c["batch"], s.out.data_ptr())
        return s.out
    if c["call"] == "rhs":
        h.rhs_ptr(0.0, s.v0.data_ptr(), s.out.data_ptr(), sbpgpu.DEVICE)
        return s.out
    if c["call"] == "rk45":
        h.set_state_ptr(s.v0.data_ptr(), sbpgpu.DEVICE)
        st = h.rk45_resident(0.0, s.t_end, s.dt)
        h.get_state_ptr(s.out.data_ptr(), sbpgpu.DEVICE)
        return {"state": s.out, "t": st["t"], "accepted": st["accepted"], "rejected": st["rejected"]}
    if c["host"]:
        return h.ts_rk4(s.host, s.t_end, s.dt)
    h.set_state_ptr(s.v0.data_ptr(), sbpgpu.DEVICE)
    h.step_resident(0.0, s.dt, c["steps"])
    h.get_state_ptr(s.out.data_ptr(), sbpgpu.DEVICE)
    return s.out


# ---------------------------------------------------------------- work
def _flops_per_stage(kind, order):
    """Operations of one point's RHS (antisymmetric stencils: order/2 differences, as many products,
    their sums) and of its Runge-Kutta update."""
    d1 = order + order // 2 - 1
    derivs, dofs = {"advection_1d": (1, 1), "reflection_1d": (2, 2), "advection_2d": (2, 1),
                    "wave_3d": (6, 4)}.get(kind, (4, 3))
    return derivs * d1 + dofs * 4


def work(case):
    k = case["kind"]
    if k == "batch":
        by = fl = 0.0
        for d in _batch_list(case):
            wave = d["problem"] == sbpgpu.WAVE_HOM_2D
            n = d["nx"] * d["ny"]
            by += 2 * 8.0 * n * (3 if wave else 1)
            fl += 4.0 * case["steps"] * n * _flops_per_stage("hom" if wave else "advection_2d", d["order"])
        return {"bytes": by, "flops": fl}
    if k.startswith("network"):
        px = case["batch"] * case["height"] * case["width"]
        macs = 9 * (24 * 32 + 32 * 32 + 32 * 32 + 32 * 3)
        back = 9 * (24 * 32 + 2 * (32 * 32 + 32 * 32 + 32 * 3)) if k == "network_train" else 0
        return {"bytes": 4.0 * px * 27, "flops": 2.0 * px * (macs + back)}
    n, dofs = _cells(case), DOFS.get(k, 3)
    by = 2 * 8.0 * n * dofs
    if k == "var":
        by += n * 2 * (4.0 if case["precision"] == "fp32" else 8.0)
    stages = {"rhs": 1, "rk45": 6 * max(1, case["steps"] // 5)}.get(case["call"], 4 * case["steps"])
    return {"bytes": by, "flops": float(stages) * n * _flops_per_stage(k, case["order"])}


# ---------------------------------------------------------------- the same in plain FP64
_INT = {2: [-1 / 2, 0, 1 / 2], 4: [1 / 12, -2 / 3, 0, 2 / 3, -1 / 12],
        6: [-1 / 60, 3 / 20, -3 / 4, 0, 3 / 4, -3 / 20, 1 / 60]}
_CLS = {2: [[-1.0, 1.0]],
        4: [[-24 / 17, 59 / 34, -4 / 17, -3 / 34, 0, 0], [-1 / 2, 0, 1 / 2, 0, 0, 0],
            [4 / 43, -59 / 86, 0, 59 / 86, -4 / 43, 0], [3 / 98, 0, -59 / 98, 0, 32 / 49, -4 / 49]],
        6: [[-21600 / 13649, 104009 / 54596, 30443 / 81894, -33311 / 27298, 16863 / 27298, -15025 / 163788, 0, 0, 0],
            [-104009 / 240260, 0, -311 / 72078, 20229 / 24026, -24337 / 48052, 36661 / 360390, 0, 0, 0],
            [-30443 / 162660, 311 / 32532, 0, -11155 / 16266, 41287 / 32532, -21999 / 54220, 0, 0, 0],
            [33311 / 107180, -20229 / 21436, 485 / 1398, 0, 4147 / 21436, 25427 / 321540, 72 / 5359, 0, 0],
            [-16863 / 78770, 24337 / 31508, -41287 / 47262, -4147 / 15754, 0, 342523 / 472620, -1296 / 7877,
             144 / 7877, 0],
            [15025 / 525612, -36661 / 262806, 21999 / 87602, -25427 / 262806, -342523 / 525612, 0, 32400 / 43801,
             -6480 / 43801, 720 / 43801]]}
_HINV = {2: 2.0, 4: 48 / 17, 6: 43200 / 13649}


def _d1(v, dim, order, h):
    """First derivative along `dim`: central stencil inside, closure rows at both ends."""
    n, r = v.shape[dim], order // 2
    cls = torch.tensor(_CLS[order], dtype=torch.float64, device=v.device)
    cs, cw = cls.shape
    out = torch.zeros_like(v)
    mid = out.narrow(dim, r, n - 2 * r)
    for s, w in enumerate(_INT[order]):
        if w:
            mid += w * v.narrow(dim, s, n - 2 * r)
    first = torch.tensordot(cls, v.narrow(dim, 0, cw).movedim(dim, 0), 1).movedim(0, dim)
    last = torch.tensordot(-cls.flip(0, 1), v.narrow(dim, n - cw, cw).movedim(dim, 0), 1).movedim(0, dim)
    out.narrow(dim, 0, cs).copy_(first)
    out.narrow(dim, n - cs, cs).copy_(last)
    return out / h


def _faces(f, v, bw, dim, c, rho, k, bc, comp_p):
    """Boundary terms of a wave problem on the two faces across `dim` (velocity component c)."""
    for lo in (True, False):
        at = 0 if lo else v.shape[dim] - 1
        sel = lambda a: a.select(dim, at) if torch.is_tensor(a) else a  # noqa: E731
        p, u = sel(v[..., comp_p]), sel(v[..., c])
        sg = 1.0 if lo else -1.0
        fu, fp = sel(f[..., c]), sel(f[..., comp_p])
        r, kk = sel(rho), sel(k)
        if bc == "free":
            fu -= sg * bw * p / r
        else:
            z = (r * kk) ** 0.5
            cc = (kk / r) ** 0.5
            g = bw * (p + sg * z * u)
            fu -= sg * 0.5 / r * g
            fp -= 0.5 * cc * g


def _wave_block(v, case, hx, hy, rho, k):
    o = case["order"]
    f = torch.empty_like(v)
    f[..., 0] = -_d1(v[..., 2], 1, o, hx) / rho
    f[..., 1] = -_d1(v[..., 2], 0, o, hy) / rho
    f[..., 2] = -k * (_d1(v[..., 0], 1, o, hx) + _d1(v[..., 1], 0, o, hy))
    return f


def _rhs_fn(case, seed):
    kind, o = case["kind"], case["order"]
    h = _spacing(case)
    bw = [_HINV[o] / x for x in h]
    if kind == "advection_1d":
        a = torch.full((case["nx"],), 1.0, dtype=torch.float64, device=DEV)
        if case["fields"]:
            a = torch.from_numpy(_velocities(case)[0]).to(DEV)

        def rhs(v, t):
            f = -a[:, None] * _d1(v, 0, o, h[0])
            f[0] += 0.5 * (-0.5 * (a[0] + a[0].abs())) * bw[0] * v[0]
            f[-1] += 0.5 * (0.5 * (a[-1] - a[-1].abs())) * bw[0] * v[-1]
            return f
        return rhs
    if kind == "reflection_1d":
        def rhs(v, t):
            f = torch.stack([_d1(v[:, 1], 0, o, h[0]), _d1(v[:, 0], 0, o, h[0])], -1)
            f[0, 0] = 0
            f[-1, 0] = 0
            return f
        return rhs
    if kind == "advection_2d":
        a = torch.full((case["ny"], case["nx"]), 1.5, dtype=torch.float64, device=DEV)
        b = torch.full_like(a, -1.0)
        if case["fields"]:
            a, b = (torch.from_numpy(np.ascontiguousarray(q)).to(DEV) for q in _velocities(case))

        def rhs(v, t):
            u = v[..., 0]
            f = -(a * _d1(u, 1, o, h[0]) + b * _d1(u, 0, o, h[1]))
            f[:, 0] += 0.5 * (-0.5 * (a[:, 0] + a[:, 0].abs())) * bw[0] * u[:, 0]
            f[0] += 0.5 * (-0.5 * (b[0] + b[0].abs())) * bw[1] * u[0]
            f[:, -1] += 0.5 * (0.5 * (a[:, -1] - a[:, -1].abs())) * bw[0] * u[:, -1]
            f[-1] += 0.5 * (0.5 * (b[-1] - b[-1].abs())) * bw[1] * u[-1]
            return f[..., None]
        return rhs
    if kind == "wave_3d":
        def rhs(v, t):
            f = torch.empty_like(v)
            for d in range(3):
                f[..., d] = -_d1(v[..., 3], 2 - d, o, h[d])
            f[..., 3] = -(_d1(v[..., 0], 2, o, h[0]) + _d1(v[..., 1], 1, o, h[1]) + _d1(v[..., 2], 0, o, h[2]))
            for d in range(3):
                _faces(f, v, bw[d], 2 - d, d, 1.0, 1.0, case["bc"], 3)
            return f
        return rhs
    if kind == "mms":
        x, y = _axes(case)
        x, y = x[None, :], y[:, None]
        ri = 1.0 / (2 + x * y)
        pi = math.pi
        gu = -3 * pi * torch.cos(3 * pi * x) * torch.sin(4 * pi * y) * (x * y + 1) / (x * y + 2)
        gv = -4 * pi * torch.cos(4 * pi * y) * torch.sin(3 * pi * x) * (x * y + 1) / (x * y + 2)

        def rhs(v, t):
            f = _wave_block(v, case, h[0], h[1], 1.0 / ri, 1.0)
            f[..., 0] += gu * math.cos(5 * pi * t)
            f[..., 1] += gv * math.cos(5 * pi * t)
            _faces(f, v, bw[0], 1, 0, 1.0, 1.0, "free", 2)
            _faces(f, v, bw[1], 0, 1, 1.0, 1.0, "free", 2)
            return f
        return rhs
    if kind == "hom":
        rho = k = 1.0
    else:
        rho, k = (torch.from_numpy(q).to(DEV) for q in _coefficients(case, seed))

    def rhs(v, t):
        if kind != "two_block":
            f = _wave_block(v, case, h[0], h[1], rho, k)
        else:
            m = case["ny"] // 2
            f = torch.cat([_wave_block(v[:m], case, h[0], h[1], rho[:m], k[:m]),
                           _wave_block(v[m:], case, h[0], h[1], rho[m:], k[m:])])
        _faces(f, v, bw[0], 1, 0, rho, k, case["bc"], 2)
        _faces(f, v, bw[1], 0, 1, rho, k, case["bc"], 2)
        if kind == "two_block":
            jump = v[m - 1] - v[m]
            for row in (m - 1, m):
                f[row, :, 1] += 0.5 / rho[row] * bw[1] * jump[:, 2]
                f[row, :, 2] += 0.5 * k[row] * bw[1] * jump[:, 1]
        return f
    return rhs


def _rk4(rhs, v, dt, steps):
    t = 0.0
    for _ in range(steps):
        k1 = rhs(v, t)
        k2 = rhs(v + 0.5 * dt * k1, t + 0.5 * dt)
        k3 = rhs(v + 0.5 * dt * k2, t + 0.5 * dt)
        k4 = rhs(v + dt * k3, t + dt)
        v = v + dt / 6 * (k1 + 2 * (k2 + k3) + k4)
        t += dt
    return v


_RKF_A = [[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197],
          [439 / 216, -8, 3680 / 513, -845 / 4104], [-8 / 27, 2, -3544 / 2565, 1859 / 4104, -11 / 40]]
_RKF_B5 = [16 / 135, 0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55]
_RKF_B4 = [25 / 216, 0, 1408 / 2565, 2197 / 4104, -1 / 5, 0]


def _land(t, t_end, h):
    left = t_end - t
    if h >= left or 1.01 * h > left:
        return left, True
    return (0.5 * left if 2 * h > left else h), False


def _rk45(rhs, v, t_end, dt):
    t, acc, rej, ok = 0.0, 0, 0, True
    h, fin = _land(t, t_end, dt)
    while True:
        k = []
        for row in _RKF_A:
            w = v
            if row:
                w = v + h * sum(c * q for c, q in zip(row, k))
            k.append(rhs(w, 0.0))
        u5 = v + h * sum(c * q for c, q in zip(_RKF_B5, k) if c)
        u4 = v + h * sum(c * q for c, q in zip(_RKF_B4, k) if c)
        e = float((((u5 - u4) / (1e-4 + 1e-4 * torch.maximum(u5.abs(), u4.abs()))) ** 2).mean().sqrt())
        accept, safety = e <= 1, 0.9 * (0.5 if e > 1 and not ok else 1.0)
        hn = h * min(max(safety * e ** -0.2 if e > 0 else 10.0, 0.1), 10.0)
        ok = accept
        if accept:
            v, acc, t = u5, acc + 1, (t_end if fin else t + h)
            if fin:
                return v, t, acc, rej
        else:
            rej += 1
        h, fin = _land(t, t_end, hn)


def _network(case, seed):
    """The network in FP64 (no rounding of weights or activations): prediction, and one Adam step."""
    x, target = _network_io(case, seed)
    vec = torch.from_numpy(_network_weights(seed, 32368)).to(DEV).double()
    y = torch.nn.functional.pad(x.double(), (0, 8)).permute(0, 3, 1, 2)
    o, parts = 0, []
    for cin, cout, relu in ((32, 32, True), (32, 32, True), (32, 32, True), (32, 16, False)):
        w = vec[o:o + cout * 9 * cin].reshape(cout, 3, 3, cin).clone().requires_grad_()
        o += cout * 9 * cin + cout
        parts.append(w)
        y = torch.nn.functional.pad(y, (1, 1, 1, 1))
        ht, wd = y.shape[2] - 2, y.shape[3] - 2
        acc = 0
        for dy in range(3):
            for dx in range(3):
                acc = acc + torch.einsum("bchw,oc->bohw", y[:, :, dy:dy + ht, dx:dx + wd], w[:, dy, dx, :])
        y = torch.relu(acc) if relu else acc
    out = y[:, :3].permute(0, 2, 3, 1)
    loss = ((out - target.double()) ** 2).mean()
    return out, loss, target


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        insts = _batch_list(case)
        outs = []
        for d, v in zip(insts, _batch_states(insts, seed)):
            wave = d["problem"] == sbpgpu.WAVE_HOM_2D
            c = _case("hom" if wave else "advection_2d", order=d["order"], nx=d["nx"], ny=d["ny"], bc="char")
            v = torch.from_numpy(v).to(DEV).reshape(d["ny"], d["nx"], 3 if wave else 1)
            h, o = _spacing(c), d["order"]
            bw = [_HINV[o] / q for q in h]
            if wave:
                k = d["c"] ** 2

                def rhs(q, t, c=c, h=h, bw=bw, k=k):
                    f = _wave_block(q, c, h[0], h[1], 1.0, k)
                    _faces(f, q, bw[0], 1, 0, 1.0, k, "char", 2)
                    _faces(f, q, bw[1], 0, 1, 1.0, k, "char", 2)
                    return f
            else:
                a, b = d["a"], d["b"]

                def rhs(q, t, h=h, bw=bw, o=o, a=a, b=b):
                    u = q[..., 0]
                    f = -(a * _d1(u, 1, o, h[0]) + b * _d1(u, 0, o, h[1]))
                    f[:, 0] -= 0.25 * (a + abs(a)) * bw[0] * u[:, 0]
                    f[0] -= 0.25 * (b + abs(b)) * bw[1] * u[0]
                    f[:, -1] += 0.25 * (a - abs(a)) * bw[0] * u[:, -1]
                    f[-1] += 0.25 * (b - abs(b)) * bw[1] * u[-1]
                    return f[..., None]
            outs.append(_rk4(rhs, v, d["dt"], case["steps"]).reshape(-1).cpu().numpy())
        return np.concatenate(outs)
    if kind == "network_forward":
        with torch.no_grad():
            return _network(case, seed)[0].contiguous()
    if kind == "network_train":
        with torch.no_grad():
            loss = _network(case, seed)[1]
        return {"loss": float(loss), "params": None}  # Adam's first step keeps the gradients' signs only
    v = _initial(case, seed)
    rhs = _rhs_fn(case, seed)
    dt = _dt(case)
    if case["call"] == "rhs":
        return rhs(v, 0.0)
    if case["call"] == "rk45":
        state, t, acc, rej = _rk45(rhs, v, dt * case["steps"], dt)
        return {"state": state, "t": t, "accepted": acc, "rejected": rej}
    out = _rk4(rhs, v, dt, case["steps"])
    return out.cpu().numpy().ravel() if case["host"] else out
