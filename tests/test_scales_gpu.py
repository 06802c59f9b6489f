"""Calls at the limits of the number formats."""
import numpy as np
import pytest

import smectic3d_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
@pytest.mark.parametrize("n", [16, 32])
def test_stokes_flow_of_a_huge_box(n, boundary):
    """Grid spacings whose smallest |q|^2 is subnormal in FP32 (2^-126.5, 22 significant
    bits): L psi = psi there, the velocity is about 1/|q| and u . grad psi of order one.
    FP32 against FP64 after two steps; a few hundred roundings of 6e-8, 2^-22 in |q|^2."""
    q = 2.0 ** -63.25
    dx = (2.0 if boundary == "periodic" else 1.0) * np.pi / (n * q)
    if boundary == "neumann":
        dx *= np.sqrt(3.0)  # all three sine wavenumbers of the first mode are pi / L
    i = np.arange(n)
    psi = 0.5 * np.cos(2 * np.pi * i / n)[:, None, None] * np.cos(4 * np.pi * i / n)[None, :, None] \
        + 0.3 * np.sin(2 * np.pi * i / n)[None, None, :] + S.ic.noise(n, 1, 0.1)
    out = {}
    for prec in ("fp64", "fp32"):
        p = S.Params(n=n, boundary=boundary, precision=prec, advection=True, dx=dx, dt=0.01)
        with S.Solver(p) as s:
            s.set_psi(psi)
            s.step(2)
            out[prec] = s.get_psi()
        with S.Solver(S.Params(n=n, boundary=boundary, precision=prec, dx=dx, dt=0.01)) as s:
            s.set_psi(psi)
            s.step(2)
            out[prec + " at rest"] = s.get_psi()
    moved = np.linalg.norm(out["fp64"] - out["fp64 at rest"])
    assert moved > 0  # the flow does take part
    assert np.linalg.norm(out["fp32"] - out["fp64"]) <= 1e-5 * np.linalg.norm(out["fp64"])
