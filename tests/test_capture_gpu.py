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
