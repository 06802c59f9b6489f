"""The forms of the plane pass against one another: one CTA per plane
(flat_kernel.cuh), clusters (plane_kernel.cuh), one axis at a time
(split_kernel.cuh)."""
import time

import numpy as np
import pytest

import smectic3d_b200 as S
from oracle import sh_oracle as O
from smectic3d_b200 import _lib as L

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


@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_monitors_of_large_planes(boundary, prec):
    """256^3: the L1 monitor of every step and the energy trace against psi read back,
    and what they add to a step.  Sums of 1.7e7 terms in FP64, compensated: 1e-12; the
    trace of an FP32 run takes the gradient part from the new spectrum before it is
    rounded to real space and back: 1e-6.  The monitor moves two FP64 fields more than
    the 6 fields of a step (at most 1.7 times the bytes in FP32), the trace none: a
    step may take 4 and 2 times as long."""
    n, took = 256, {}
    kw = dict(n=n, boundary=boundary, precision=prec)
    for name, extra in (("plain", {}), ("l1", dict(l1_interval=1)), ("trace", dict(energy_trace=True))):
        with S.Solver(S.Params(**kw, **extra)) as s:
            s.set_psi(_psi(n))
            s.step(2)
            if name == "l1":
                old = s.get_psi()
                s.step(1)
                new = s.get_psi()
                want = np.abs(new - old).sum() / (s.params.dt * np.abs(new).sum())
                assert abs(s.l1()[0][0] - want) <= 1e-12 * want
            if name == "trace":
                e = s.energy()[0]
                assert abs(s.energy_trace()[-1] - e) <= (1e-12 if prec == "fp64" else 1e-6) * abs(e)
            t = []
            for _ in range(5):
                t0 = time.perf_counter()
                s.step(20)
                t.append(time.perf_counter() - t0)
            took[name] = min(t)
    assert took["l1"] <= 4 * took["plain"]
    assert took["trace"] <= 2 * took["plain"]


@pytest.mark.parametrize("advection", [False, True])
@pytest.mark.parametrize("prec", ["fp32", "fp32_u64", "fp64"])
@pytest.mark.parametrize("boundary", ["periodic", "neumann"])
@pytest.mark.parametrize("n", [16, 64, 128])
def test_a_traced_step_is_the_step(n, boundary, prec, advection):
    """The kernels with options round every mode as the one without: the energy trace
    changes no bit of psi, nor (plain steps) of the spectrum W and the partials."""
    psi, out = _psi(n, 0.8), []
    kw = dict(n=n, boundary=boundary, precision=prec, advection=advection, dt=0.02)
    for trace in (False, True):
        with S.Solver(S.Params(energy_trace=trace, **kw)) as s:
            s.set_psi(psi)
            s.step(6)
            out.append(s.get_psi())
            if not advection:
                fields = 3 * n * n * (n // 2 + (boundary == "periodic"))
                body = s.checkpoint()[-fields * (16 if prec == "fp64" else 8):]
                out[-1] = out[-1].tobytes() + body
    assert out[0].tobytes() == out[1].tobytes() if advection else out[0] == out[1]


def _clustered(monkeypatch, p):
    """A handle whose slab could not be allocated: its plane passes run clustered."""
    for k in range(5, 40):
        monkeypatch.setenv("SMECTIC_B200_TEST_FAIL_ALLOC", str(k))
        try:
            s = S.Solver(p)
        except S.ShError as e:
            assert e.code == L.SH_ENOMEM
            continue
        finally:
            monkeypatch.delenv("SMECTIC_B200_TEST_FAIL_ALLOC")
        return s
    raise AssertionError("no allocation that a handle can do without")


def _launches(s):
    before = s.kernel_launches
    s.step(1)
    return s.kernel_launches - before


LARGE = [dict(n=256, boundary="periodic"), dict(n=256, boundary="neumann"),
         dict(n=256, boundary="periodic", w_mid=0.01), dict(n=256, boundary="neumann", w_mid=0.01),
         dict(n=256, boundary="neumann", sub_sigma=0.5, sub_z0=0.7),
         dict(n=256, boundary="neumann", nonlinearity="quad_cubic"),
         dict(n=256, boundary="periodic", scheme="imex_euler"),
         dict(n=256, boundary="periodic", advection=True, dt=0.02, w_mid=0.01),
         dict(n=256, boundary="neumann", advection=True, dt=0.02, w_mid=0.01)]


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 2e-6)])
@pytest.mark.parametrize("kw", LARGE, ids=str)
def test_split_passes_match_the_clusters(monkeypatch, kw, prec, tol):
    """256^3 with each option, one axis at a time against clusters of the default size:
    psi^0 and its N, three steps with the monitor, the energy.  A step is some 50
    dependent roundings of 1.1e-16 or 6e-8 on terms of the size of psi, the sums of the
    monitor and the energy less: 1e-12 and 2e-6 after three steps, ten times that with
    the advected step's products of derivatives."""
    tol *= 10 if kw.get("advection") else 1
    psi, out = _psi(256, 0.8), []
    p = S.Params(precision=prec, l1_interval=2, **kw)
    for make in (lambda: S.Solver(p), lambda: _clustered(monkeypatch, p)):
        with make() as s:
            s.set_psi(psi)
            first = _launches(s)
            s.step(2)
            out.append([first, s.get_psi(), s.l1()[0], np.array(s.energy())])
    assert out[1][0] < out[0][0]  # fewer launches: the second handle did run clustered
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("n,boundary,cl", [(256, "neumann", 4), (256, "periodic", 16), (512, "neumann", 16),
                                           (512, "periodic", 16)])
def test_every_cluster_size_still_steps(monkeypatch, n, boundary, cl):
    """The other cluster sizes of 256^3 and the 512^3 planes (clusters of 16, direct
    exchange), FP32, as above."""
    psi, out = _psi(n, 0.8), []
    p = S.Params(n=n, boundary=boundary, precision="fp32", variant=cl)
    for make in (lambda: S.Solver(p), lambda: _clustered(monkeypatch, p)):
        with make() as s:
            s.set_psi(psi)
            first = _launches(s)
            s.step(2)
            out.append((first, s.get_psi()))
    assert out[1][0] < out[0][0]
    assert np.linalg.norm(out[0][1] - out[1][1]) <= 2e-6 * np.linalg.norm(out[1][1])


@pytest.mark.parametrize("kw", [dict(boundary="periodic", w_mid=0.01, nonlinearity="quad_cubic"),
                                dict(boundary="neumann", sub_sigma=0.5, sub_z0=0.7),
                                dict(boundary="neumann", w_mid=0.01, scheme="imex_euler")], ids=str)
def test_options_of_large_planes_match_the_oracle(kw):
    """256^3 FP64, two steps (the second takes N of a state the kernels made)."""
    n = 256
    p = S.Params(n=n, precision="fp64", **kw)
    psi = _psi(n, 0.8)
    op = O.Params(n=n, dx=p.dx, dt=p.dt, eps=p.eps, nonlinearity=p.nonlinearity, scheme=p.scheme, w_mid=p.w_mid,
                  sub_sigma=p.sub_sigma, sub_z0=p.sub_z0)
    o = (O.PeriodicOracle if p.boundary == "periodic" else O.NeumannOracle)(psi, op)
    o.run(2)
    with S.Solver(p) as s:
        s.set_psi(psi)
        s.step(2)
        out = s.get_psi()
    assert np.linalg.norm(out - o.psi) <= 1e-12 * np.linalg.norm(o.psi)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-11), ("fp32", 1e-5)])
def test_adjoint_of_large_planes_matches_a_small_box(prec, tol):
    """256^3: states that repeat every 64 points have the repeated gradient of the 64^3
    box and 64 times its parameter gradients.  The reverse sweep's planes run clustered,
    the recomputed steps one axis at a time; 7 steps out and back are some 700 roundings."""
    psi, out = _psi(64), {}
    for n, p in ((64, "fp64"), (256, prec)):
        with S.Solver(S.Params(n=n, precision=p)) as s:
            s.adjoint_forward(np.tile(psi, (n // 64,) * 3), 7, 3)
            end = s.get_psi()
            out[n] = [end, *s.adjoint_backward(end - 0.5)]
    for i, scale in ((0, 1), (3, 1), (1, 64), (2, 64)):
        want = scale * (np.tile(out[64][i], (4, 4, 4)) if i in (0, 3) else out[64][i])
        assert np.linalg.norm(out[256][i] - want) <= tol * np.linalg.norm(want), i


@pytest.mark.parametrize("curvature", ["difference", "spectral"])
def test_curvature_pass_of_large_planes(monkeypatch, curvature):
    """Neumann 256^3 FP64: the curvature pass on a state the split passes made against
    the one that the clusters made (1e-12 of psi; divided by gradients of order 0.1)."""
    psi, out = S.ic.hyperboloid(256, 2 * np.pi / 8, amp=1.3, r0_cells=20, seed=1), []
    p = S.Params(n=256, boundary="neumann", precision="fp64", curvature=curvature)
    for make in (lambda: S.Solver(p), lambda: _clustered(monkeypatch, p)):
        with make() as s:
            s.set_psi(psi)
            s.step(2)
            out.append(s.surface_step())
    assert (out[0][0] >= 0).any() and np.array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.linalg.norm(np.nan_to_num(a - b)) <= 1e-9 * np.linalg.norm(np.nan_to_num(b))
