"""The forms of the plane pass against one another: one CTA per plane
(flat_kernel.cuh), clusters (plane_kernel.cuh), one axis at a time
(split_kernel.cuh)."""
import numpy as np
import pytest

import smectic3d_b200 as S

pytestmark = pytest.mark.gpu


def _psi(n, amp=0.9):
    return S.ic.undulated_lamellae(n, 2 * np.pi / 8, amp=amp, wavelength_cells=min(64, n), seed=1) + S.ic.noise(n, 2, 0.05)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
@pytest.mark.parametrize("n,cl", [(64, 2), (128, 2), (128, 4)])
def test_one_cta_form_rounds_as_the_clusters(n, cl, boundary, prec):
    """Both forms pair the same rows and round in the same order: psi after some steps
    and the adjoint's gradients are equal bit for bit.  (FP64 cosine transforms form
    X[N-k] from the products of X[k]: a few roundings, 1e-14 of psi.)"""
    psi, out = _psi(n), {}
    for v in (1, cl):
        with S.Solver(S.Params(n=n, boundary=boundary, precision=prec, variant=v)) as s:
            s.set_psi(psi)
            s.step(5)
            out[v] = [s.get_psi()]
            if boundary == "periodic":
                s.adjoint_forward(psi, 7, 3)
                p = s.get_psi()
                out[v] += [p, *s.adjoint_backward(p - 0.5)]
    for a, b in zip(out[1], out[cl]):
        if boundary == "neumann" and prec == "fp64":
            assert np.linalg.norm(a - b) <= 1e-14 * np.linalg.norm(b)
        else:
            assert np.array_equal(a, b)
