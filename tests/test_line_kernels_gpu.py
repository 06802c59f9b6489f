"""The lane-per-line passes (line_fft.cuh): the pencil pass, the one-CTA plane pass
and the split plane pass, at the edges of their tiles, against the FP64 oracle and
against one another.

Tolerances.  FP64: a step is about 6 log2(N) dependent roundings of 1.1e-16 on terms
of the size of psi; 1e-12 leaves three orders for the worst mode.  FP32: the same
count of 6.0e-8 roundings plus the rounded CNAB2 multipliers (6e-8 per step): 5e-6
after three steps.  W is compared relative to its norm.  What only regroups the same
arithmetic (replicas, slabs) is compared bit for bit."""
import ctypes as C

import numpy as np
import pytest

import smectic3d_b200 as S
from oracle import sh_oracle as O
from smectic3d_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _psi(n, seed, amp=1.2):
    return S.ic.undulated_lamellae(n, 2 * np.pi / 8, amp=amp, wavelength_cells=min(64, n), seed=seed) + S.ic.noise(
        n, seed, 0.05)


def _oracle(p, psi):
    op = O.Params(n=p.n, dx=p.dx, dt=p.dt, eps=p.eps, nonlinearity=p.nonlinearity, scheme=p.scheme, w_mid=p.w_mid,
                  sub_sigma=p.sub_sigma)
    return (O.PeriodicOracle if p.boundary == "periodic" else O.NeumannOracle)(psi, op, advect=p.advection)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 5e-6), ("fp32_u64", 5e-6)])
@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
@pytest.mark.parametrize("n", [16, 32, 64, 128])
def test_lean_and_general_steps_match_the_oracle(n, boundary, prec, tol):
    """The step without options, and the general kernels that the energy trace,
    IMEX Euler and the penalties take."""
    psi = _psi(n, 3)
    for kw in (dict(), dict(energy_trace=True), dict(nonlinearity="quad_cubic"), dict(scheme="imex_euler"),
               dict(w_mid=0.01)):
        p = S.Params(n=n, boundary=boundary, precision=prec, **kw)
        o = _oracle(p, psi)
        o.run(3)
        with S.Solver(p) as s:
            s.set_psi(psi)
            s.step(3)
            out = s.get_psi()
        assert np.linalg.norm(out - o.psi) <= tol * np.linalg.norm(o.psi), kw


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
def test_split_pass_replicas_cross_slabs_bit_for_bit(boundary, prec):
    """256^3: three replicas run through slabs that do not end with a replica; each
    equals its own single-replica run, with the monitor on and off."""
    n, b = 256, 3
    psi = np.stack([_psi(n, i, 0.8 + 0.2 * i) for i in range(b)])
    with S.Solver(S.Params(n=n, batch=b, boundary=boundary, precision=prec, l1_interval=2)) as s:
        s.set_psi(psi)
        s.step(3)
        both, l1 = s.get_psi(), s.l1()[0]
    for i in range(b):
        for monitor in (0, 2):
            with S.Solver(S.Params(n=n, boundary=boundary, precision=prec, l1_interval=monitor)) as s:
                s.set_psi(psi[i])
                s.step(3)
                assert np.array_equal(s.get_psi(), both[i])
                assert not monitor or s.l1()[0][0] == l1[i]


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-11), ("fp32", 1e-5)])
def test_advected_split_step_matches_a_small_box(prec, tol):
    """256^3 periodic with advection: a state that repeats every 32 points in each
    axis stays the repetition of the 32^3 run (another kernel)."""
    small = _psi(32, 5, 0.9)
    kw = dict(boundary="periodic", advection=True, dt=0.02)
    with S.Solver(S.Params(n=32, precision="fp64", **kw)) as s:
        s.set_psi(small)
        s.step(3)
        want = np.tile(s.get_psi(), (8, 8, 8))
        surf = s.surface_step()
    with S.Solver(S.Params(n=256, precision=prec, **kw)) as s:
        s.set_psi(np.tile(small, (8, 8, 8)))
        s.step(3)
        out = s.get_psi()
        if prec == "fp64":  # the surface pass needs L psi, which the split step keeps to itself
            for a, b in zip(s.surface_step(), surf):
                assert np.allclose(a, np.tile(b, (8, 8)), rtol=1e-7, atol=1e-9, equal_nan=True)
    assert np.linalg.norm(out - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
def test_checkpoint_file_keeps_w_by_line(boundary):
    """The checkpoint stores W = C1 psihat - dt/2 Nhat as [f][kx], f = (ky, kz), the
    layout of files written before W moved to [kx][f] on the device."""
    n = 32
    p = S.Params(n=n, boundary=boundary, precision="fp64")
    psi = _psi(n, 7)
    o = _oracle(p, psi)
    fwd = O.r2c if boundary == "periodic" else O.dct3d
    w = o.c1 * fwd(psi) - 0.5 * p.dt * fwd(O.nonlin(psi, o.p))
    with S.Solver(p) as s:
        s.set_psi(psi)
        blob = s.checkpoint()
        s.step(4)
        end = s.get_psi()
        s.restore(blob)
        s.step(4)
        assert np.array_equal(s.get_psi(), end)
    head = C.sizeof(L.ShParams) + 8
    if boundary == "periodic":
        fp = n * (n // 2 + 1)
        got = np.frombuffer(blob, np.complex128, fp * n, head).reshape(fp, n)
        want = np.concatenate([w[:, :, : n // 2].transpose(1, 2, 0).reshape(-1, n), w[:, :, n // 2].T])
    else:
        got = np.frombuffer(blob, np.float64, n * n * n, head).reshape(n, n // 2, n, 2)  # [ky][kz / 2][kx][kz % 2]
        want = w.reshape(n, n, n // 2, 2).transpose(1, 2, 0, 3)
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("n,b", [(64, 1), (64, 2), (32, 17), (128, 1)])
def test_host_arrays_cross_unchanged(n, b):
    """Pageable arrays below, at and above the size that is staged by threads (4 MB),
    with a ragged last chunk: psi^0 comes back as it went in, also when two handles
    copy at the same time from two threads (one of them then goes the plain way)."""
    import threading

    psi = np.random.default_rng(n + b).uniform(-1, 1, size=(b, n, n, n))
    p = S.Params(n=n, batch=b, precision="fp64")
    bad = []

    def loop(shift):
        with S.Solver(p) as s:
            for k in range(5):
                a = (psi + shift + k).reshape(s.shape)
                s.set_psi(a)
                if not np.array_equal(s.get_psi(), a):
                    bad.append((shift, k))

    loop(0)
    threads = [threading.Thread(target=loop, args=(10 * i,)) for i in range(1, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("n,boundary", [(64, "periodic"), (256, "periodic"), (256, "neumann")])
def test_advected_replays_equal_direct_steps(n, boundary):
    """Steps replayed from the graphs (one step at 256^3, 16 steps) leave the state,
    the velocity and the surface pass of steps launched one by one."""
    psi = _psi(n, 9, 0.9)
    kw = dict(n=n, boundary=boundary, precision="fp32", advection=True, dt=0.02)
    with S.Solver(S.Params(**kw)) as a, S.Solver(S.Params(energy_trace=True, **kw)) as b:  # a trace runs outside graphs
        for s in (a, b):
            s.set_psi(psi)
        for k in (3, 16, 1):
            for s in (a, b):
                s.step(k)
            assert np.array_equal(a.get_psi(), b.get_psi()), k
            for u, v in zip(a.velocity(), b.velocity()):
                assert np.array_equal(u, v), k
            if boundary == "periodic":
                for u, v in zip(a.surface_step(), b.surface_step()):
                    assert np.array_equal(u, v, equal_nan=True), k
