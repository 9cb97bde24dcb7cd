"""Contexts on a caller's own stream: launches that overlap the kernel before them in the stream
wait for that kernel, also when it is the caller's, and the caller's next kernel waits for them;
the manufactured problem's steps captured into the caller's graph (its stage times are then
values of the launches) give the results of the steps run directly.

The stream's other work is a long matrix product whose result decides what is read, so that a
kernel that did not wait would read the old values. Same calls, same kernels: equal bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _slow(torch, v):
    """v, as the end of some milliseconds of work on the current stream."""
    a = torch.ones((4096, 4096), device="cuda")
    for _ in range(4):
        a = a @ a
        a /= a.max()
    return v * a.min().double()  # times one


@pytest.mark.parametrize("kind,nx,ny", [("hom", 300, 290), ("hom", 65, 66), ("var", 300, 290), ("adv", 401, 300),
                                         ("line", 201, 1), ("wave3d", 40, 40)])
def test_work_around_the_launches(sbp, kind, nx, ny):
    import torch

    rng = np.random.default_rng(nx)
    s = torch.cuda.Stream()
    kw, nz = {"stream": s.cuda_stream}, 1
    if kind == "var":
        kw.update(rho=0.5 + rng.random(nx * ny), K=0.5 + rng.random(nx * ny))
    if kind == "wave3d":
        nz = 30
    problem = {"hom": sbp.WAVE_HOM_2D, "var": sbp.WAVE_VAR_2D, "adv": sbp.ADVECTION_2D, "line": sbp.ADVECTION_1D,
               "wave3d": sbp.WAVE_3D}[kind]
    with sbp.Context(problem, 4, nx, ny, nz, **kw) as c:
        v = torch.from_numpy(rng.standard_normal(c.size)).cuda()
        src, dst, after = torch.zeros_like(v), torch.zeros_like(v), torch.zeros_like(v)
        torch.cuda.synchronize()
        want = np.empty((2, c.size))
        c.rhs_ptr(0.0, v.data_ptr(), dst.data_ptr(), sbp.DEVICE)
        want[0] = dst.cpu().numpy()
        c.set_state_ptr(v.data_ptr(), sbp.DEVICE)
        c.step_resident(0.0, 1e-4, 3)
        c.get_state_ptr(dst.data_ptr(), sbp.DEVICE)
        c.synchronize()
        want[1] = dst.cpu().numpy()
        for _ in range(3):
            src.zero_()
            dst.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(s):
                src.copy_(_slow(torch, v))
                c.rhs_ptr(0.0, src.data_ptr(), dst.data_ptr(), sbp.DEVICE)
                after.copy_(dst)
            torch.cuda.synchronize()
            assert np.array_equal(after.cpu().numpy(), want[0])
            src.zero_()
            torch.cuda.synchronize()
            with torch.cuda.stream(s):
                src.copy_(_slow(torch, v))
                c.set_state_ptr(src.data_ptr(), sbp.DEVICE)
                c.step_resident(0.0, 1e-4, 3)
                c.get_state_ptr(dst.data_ptr(), sbp.DEVICE)
                after.copy_(dst)
            torch.cuda.synchronize()
            assert np.array_equal(after.cpu().numpy(), want[1])


@pytest.mark.parametrize("n", [60, 700])
def test_forced_steps_in_the_callers_graph(sbp, port, n):
    import torch

    import oracle as O

    s = torch.cuda.Stream()
    v = np.random.default_rng(n).standard_normal(3 * n * n)
    dt = 0.05 / n
    with sbp.Context(sbp.WAVE_MMS_2D, 4, n, n, stream=s.cuda_stream) as c:
        c.set_state(v)
        c.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            c.step_resident(0.1, dt, 3)
        for _ in range(2):  # the replay starts from the state the context holds
            c.set_state(v)
            with torch.cuda.stream(s):
                g.replay()
            got = c.get_state()
            ref = port.rk4(O.Problem(O.WAVE_MMS_2D, 4, n, n), v, 0.1, dt, 3)
            assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
        c.set_state(v)
        c.step_resident(0.1, dt, 3)  # and outside the capture: the context's own graph and table
        assert np.max(np.abs(c.get_state() - ref)) <= 1e-12 * np.max(np.abs(ref))
