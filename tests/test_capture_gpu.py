"""Step graphs: the handle's own and the caller's."""
import threading

import numpy as np
import pytest

import smectic3d_b200 as S

pytestmark = pytest.mark.gpu


def _psi(n):
    return S.ic.undulated_lamellae(n, 2 * np.pi / 8, amp=0.9, wavelength_cells=min(64, n), seed=1) + S.ic.noise(n, 2, 0.05)


@pytest.mark.parametrize("kw", [dict(n=64), dict(n=256), dict(n=256, advection=True, dt=0.02),
                                dict(n=256, boundary="neumann", batch=2)], ids=str)
def test_a_few_steps_can_be_captured_by_the_caller(kw):
    """Fewer steps than a replayed chunk are plain launches on the handle's stream
    while the caller captures it, also where they go slab by slab."""
    import torch

    p = S.Params(precision="fp32", **kw)
    psi = np.broadcast_to(_psi(p.n), (p.batch, p.n, p.n, p.n)).copy()
    with S.Solver(p) as a, S.Solver(p) as b:
        for s in (a, b):
            s.set_psi(psi.reshape(s.shape))
        b.step(4)
        st = torch.cuda.ExternalStream(a.stream)
        a.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(st):
            g.capture_begin()
            a.step_async(2)
            g.capture_end()
            g.replay()
            g.replay()
        assert np.array_equal(a.get_psi(), b.get_psi())


@pytest.mark.parametrize("n", [32, 256])
def test_prepare_leaves_a_restored_state_to_be_computed(n):
    """sh_prepare records the step graph and changes no state: the velocity and the
    surface pass of a restored checkpoint are those without it (the real-space fields
    they read belong to the handle's state before, or to none)."""
    kw = dict(n=n, precision="fp32", advection=True, dt=0.02)
    with S.Solver(S.Params(**kw)) as s:
        s.set_psi(_psi(n))
        s.step(3)
        blob = s.checkpoint()
    out = {}
    for prepare in (False, True):
        for what in ("velocity", "surface_step"):
            with S.Solver(S.Params(**kw)) as s:
                s.set_psi(S.ic.noise(n, 5, 0.3))
                s.step(1)
                s.restore(blob)
                if prepare:
                    s.prepare()
                out[prepare, what] = getattr(s, what)()
    for what in ("velocity", "surface_step"):
        for a, b in zip(out[False, what], out[True, what]):
            assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("kw", [dict(n=32), dict(n=128, boundary="neumann", sub_sigma=0.5), dict(n=64, variant=2),
                                dict(n=256, precision="fp64"), dict(n=64, advection=True, dt=0.02),
                                dict(n=256, boundary="neumann", advection=True, dt=0.02),
                                dict(n=256, scheme="imex_euler", w_mid=0.01)], ids=str)
def test_a_new_handle_can_be_captured(kw):
    """The first calls of a handle, psi in, steps and psi out on the device, recorded by
    the caller before any kernel of it has run."""
    import torch

    p = S.Params(**{"precision": "fp32", **kw})
    with S.Solver(p) as a, S.Solver(p) as b:
        psi = torch.tensor(_psi(p.n), device="cuda")
        out, want = torch.zeros_like(psi), torch.zeros_like(psi)
        torch.cuda.synchronize()
        st = torch.cuda.ExternalStream(a.stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(st):
            g.capture_begin()
            a.set_psi_device(psi.data_ptr())
            a.step_async(2)
            a.get_psi_device(out.data_ptr())
            g.capture_end()
            g.replay()
        a.synchronize()
        b.set_psi_device(psi.data_ptr())
        b.step(2)
        b.get_psi_device(want.data_ptr())
        b.synchronize()
        assert torch.equal(out, want) and float(want.abs().max()) > 0.1
