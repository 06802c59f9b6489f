"""Checkpoints of advected handles and of handles that fill the GPU."""
import numpy as np
import pytest

import smectic3d_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 128])  # 128 FP64: fields large enough to be staged by threads
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


def _fill():
    """Arrays on the GPU, the last ones of 12 MB, until no more can be had."""
    import torch

    torch.cuda.empty_cache()
    full = [torch.empty(torch.cuda.mem_get_info()[0] - 2**28, dtype=torch.uint8, device="cuda")]
    try:
        while True:
            full.append(torch.empty(12 * 2**20, dtype=torch.uint8, device="cuda"))
    except torch.OutOfMemoryError:
        return full


@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
def test_checkpoint_needs_no_device_memory(boundary):
    """128^3 FP64 (fields of 34 MB and more) with less than 12 MB of the GPU left: saved
    (before and after the first step) and restored as with the GPU empty, and the state
    goes on as if nothing had been saved."""
    import torch

    n = 128
    p = S.Params(n=n, boundary=boundary, precision="fp64")
    psi = S.ic.noise(n, 3, 0.3)
    with S.Solver(p) as a, S.Solver(p) as b:
        for s in (a, b):
            s.set_psi(psi)
        zero = b.checkpoint()
        for s in (a, b):
            s.step(2)
        want = b.checkpoint()
        b.step(1)
        end = b.get_psi()
        b.step(3)
        full = _fill()
        blob = a.checkpoint()
        a.step(1)
        out = a.get_psi()
        b.restore(blob)
        b.step(1)
        again = b.get_psi()
        a.set_psi(psi)
        first = a.checkpoint()
        start = a.get_psi()
        a.step(3)
        third = a.get_psi()
        del full
        torch.cuda.empty_cache()
    assert blob == want and first == zero and np.array_equal(start, psi)
    assert np.array_equal(out, end) and np.array_equal(again, end) and np.array_equal(third, end)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
def test_checkpoint_of_replicas_is_theirs(boundary, prec):
    """Three replicas in one handle: per field the file holds what each replica's own
    file holds, before and after the first step."""
    n, b = 32, 3
    kw = dict(n=n, boundary=boundary, precision=prec)
    psi = S.ic.noise_batch(n, range(b), amp=0.3)
    field = n * n * (n // 2 + (boundary == "periodic")) * (16 if prec == "fp64" else 8)
    for steps in (0, 2):
        with S.Solver(S.Params(batch=b, **kw)) as s:
            s.set_psi(psi)
            s.step(steps)
            both = s.checkpoint()[-3 * b * field:]
        for i in range(b):
            with S.Solver(S.Params(**kw)) as s:
                s.set_psi(psi[i])
                s.step(steps)
                one = s.checkpoint()[-3 * field:]
            for f in range(3):
                assert both[(f * b + i) * field:][:field] == one[f * field:][:field]
