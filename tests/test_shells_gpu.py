"""The per-shell spectral power behind the dominant wavenumber."""
import numpy as np
import pytest

import smectic3d_b200 as S
from oracle import sh_oracle as O

pytestmark = pytest.mark.gpu


def _flat(n, boundary, k, seed):
    """Noise whose shells hold the same power each, but for shell k with 2 % more."""
    x = np.random.default_rng(seed).standard_normal((n, n, n))
    if boundary == "periodic":
        i = np.fft.fftfreq(n, 1.0 / n)
        spec, w = np.fft.rfftn(x), np.full(n // 2 + 1, 2.0)
        w[[0, -1]] = 1.0
        shell = np.rint(np.sqrt(i[:, None, None] ** 2 + i[None, :, None] ** 2 + i[None, None, : n // 2 + 1] ** 2))
        w = np.broadcast_to(w, spec.shape)
    else:
        i = np.arange(n)
        h = np.where(i == 0, 0.5, 1.0)
        spec, w = O.dct3d(x), h[:, None, None] * h[None, :, None] * h[None, None, :]
        shell = np.rint(np.sqrt(i[:, None, None] ** 2 + i[None, :, None] ** 2 + i[None, None, :] ** 2))
        i = i.astype(float)
    shell = np.abs(shell).astype(int)
    power = np.bincount(shell.ravel(), weights=(w * np.abs(spec) ** 2).ravel())
    scale = 1.0 / np.sqrt(np.maximum(power, 1e-300))
    scale[k] *= np.sqrt(1.02)
    scale[0] = 0.0
    spec = spec * scale[shell]
    y = np.fft.irfftn(spec, (n, n, n), axes=(0, 1, 2)) if boundary == "periodic" else O.idct3d(spec)
    return y / np.abs(y).max()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
@pytest.mark.parametrize("n,tile", [(16, 0), (32, 0), (64, 0), (64, 8), (64, 32), (128, 0)])
def test_every_shell_gets_its_power_once(n, tile, boundary, prec):
    """One shell of 2 % more power than the others is found, the lowest, the highest and
    some between (a mode lost or added twice in a shell of up to a few hundred shows)."""
    p = S.Params(n=n, boundary=boundary, precision=prec, pencil_tile=tile)
    top = int(np.rint(np.sqrt(3.0) * (n // 2 if boundary == "periodic" else n - 1)))
    dominant = O.dominant_wavenumber if boundary == "periodic" else O.dominant_wavenumber_neumann
    with S.Solver(p) as s:
        for k in sorted({1, 2, n // 4, n // 2 - 1, n // 2, top // 2, top - 1, top}):
            psi = _flat(n, boundary, k, k)
            s.set_psi(psi)
            want = dominant(psi, p.dx)
            assert want == pytest.approx(k * (2 if boundary == "periodic" else 1) * np.pi / (n * p.dx))
            assert s.dominant_wavenumber()[0] == pytest.approx(want), k
