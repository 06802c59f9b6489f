"""Checkpoints of advected handles and of handles that fill the GPU."""
import numpy as np
import pytest

import smectic3d_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 128])  # 128: fields above the 4 MB that are staged by threads
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
def test_advected_checkpoint_round_trip(boundary, prec, n):
    """Saved, stepped on, restored and stepped again, in the same handle and in a new
    one: the same bits, the velocity of the restored state included."""
    p = S.Params(n=n, boundary=boundary, precision=prec, advection=True, dt=0.02)
    psi = S.ic.undulated_lamellae(n, p.dx, amp=0.9, wavelength_cells=32, seed=1)
    with S.Solver(p) as s:
        s.set_psi(psi)
        s.step(3)
        blob = s.checkpoint()
        u = s.velocity()
        s.step(4)
        end = s.get_psi()
        s.restore(blob)
        s.step(4)
        assert np.array_equal(s.get_psi(), end)
    with S.Solver(p) as s:
        s.restore(blob)
        for a, b in zip(s.velocity(), u):
            assert np.array_equal(a, b)
        s.step(4)
        assert np.array_equal(s.get_psi(), end)
