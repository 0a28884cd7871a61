"""The one-launch kernels of small boxes against the one-launch-per-pass kernels (needs a B200).

Boxes up to 128^3 whose N x N plane fits a CTA's shared memory run all their
steps in one kernel; IFDM_NO_FUSE=1 keeps a kernel per pass.  Both do the same
transforms in another order of radices and axes, so they agree to rounding:
psi after a few steps to a few ulps per transform (12 transforms a step; FP64
1e-13, FP32 and mixed 2e-6), phi to that over the density contrast (0.02).
"""

import numpy as np
import pytest

import ifdm_code_b200 as ifdm
from ifdm_code_b200.synthetic_ic import zeldovich_psi
from tests.snapshot_util import rel_l2

pytestmark = pytest.mark.gpu

MFDM, XMAX, A0 = 2.5e-24, 5.0, 1.0 / 51.0
SIZES = [16, 32, 48, 64, 96, 128]
PSI = {"fp64": 1e-13, "fp32": 2e-6, "mixed": 2e-6}


def _both(monkeypatch, prec, n, g, fn):
    out = []
    for plain in (False, True):
        if plain:
            monkeypatch.setenv("IFDM_NO_FUSE", "1")
        else:
            monkeypatch.delenv("IFDM_NO_FUSE", raising=False)
        with ifdm.Simulation(MFDM, g, XMAX, n, precision=prec) as s:
            out.append(fn(s))
    return out


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("n", SIZES)
def test_box_steps_match_passes(n, prec, monkeypatch):
    psi0 = zeldovich_psi(n, seed=n)

    def run(s):
        s.set_psi(psi0, A0)
        phi0 = s.get_phi()
        s.step(1, 0.01)
        s.step(3, 0.01)
        return phi0, s.get_psi(), s.get_phi(), s.state()

    (f0, p, f, st), (f0r, pr, fr, sr) = _both(monkeypatch, prec, n, 1e-63, run)
    tol = PSI[prec]
    assert st["device_error"] == 0 and st["steps"] == sr["steps"] == 4 and st["a"] == sr["a"]
    assert rel_l2(p, pr) <= tol
    assert rel_l2(f0, f0r) <= tol / 0.02 and rel_l2(f, fr) <= tol / 0.02
    assert st["max_rho"] == pytest.approx(sr["max_rho"], rel=2 * tol)
    assert st["dt_QI"] == pytest.approx(sr["dt_QI"], rel=1e-12)


@pytest.mark.parametrize("a,g,crit", [(0.4, 0.0, 2), (0.02, 1e-60, 4)])
@pytest.mark.parametrize("n", [16, 48])
def test_box_timestep_criteria(n, a, g, crit, monkeypatch):
    """Steps that the potential or the self-interaction limits: their integrals
    are not the kinetic step's, which the kernel prepares ahead."""
    psi0 = zeldovich_psi(n, seed=3, rms_delta=0.5)

    def run(s):
        s.set_psi(psi0, a)
        s.step(5, 0.1)
        return s.get_psi(), s.state()

    (p, st), (pr, sr) = _both(monkeypatch, "fp64", n, g, run)
    assert st["criterion"] == sr["criterion"] == crit
    for k in ("a", "dt_KE", "dt_PE", "dt_QI"):
        assert st[k] == pytest.approx(sr[k], rel=1e-12)
    assert rel_l2(p, pr) <= 1e-11


def test_box_run_longer_than_one_launch(monkeypatch):
    psi0 = zeldovich_psi(16, seed=5)

    def run(s):
        s.set_psi(psi0, A0)
        s.step(1027, 1e-4)  # two full launches of 512 steps and three more
        return s.get_psi(), s.state()

    (p, st), (pr, sr) = _both(monkeypatch, "fp64", 16, 0.0, run)
    assert st["steps"] == 1027 and st["a"] == pytest.approx(sr["a"], rel=1e-12)
    assert rel_l2(p, pr) <= 1e-13 * 1027


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("n", [16, 48, 64, 128])
def test_box_adjoint_matches_passes(n, prec, monkeypatch):
    psi0 = zeldovich_psi(n, seed=n)
    rng = np.random.default_rng(n)
    cot = rng.standard_normal((n,) * 3) + 1j * rng.standard_normal((n,) * 3)

    def run(s):
        s.set_psi(psi0, A0)
        s.record_steps(5, 0.01, 2)  # three segments, the last one a single step
        g = np.empty_like(cot)
        psi = s.get_psi()
        s.adjoint(cot, g)
        return psi, g

    (p, g), (pr, gr) = _both(monkeypatch, prec, n, 1e-63, run)
    assert rel_l2(p, pr) <= PSI[prec]
    assert rel_l2(g, gr) <= 10 * PSI[prec]


@pytest.mark.parametrize("n", [16, 64])
def test_two_boxes_in_flight_on_two_streams(n):
    """Two contexts stepping at once (each a cluster or a cooperative grid) give
    what each gives alone."""
    psi0 = [zeldovich_psi(n, seed=i) for i in range(2)]
    alone = []
    for i in range(2):
        with ifdm.Simulation(MFDM, 0.0, XMAX, n) as s:
            s.set_psi(psi0[i], A0)
            s.step(40, 0.01)
            alone.append(s.get_psi())
    with ifdm.Simulation(MFDM, 0.0, XMAX, n) as a, ifdm.Simulation(MFDM, 0.0, XMAX, n) as b:
        a.set_psi(psi0[0], A0)
        b.set_psi(psi0[1], A0)
        for _ in range(10):
            a.step(4, 0.01)
            b.step(4, 0.01)
        assert np.array_equal(a.get_psi(), alone[0]) and np.array_equal(b.get_psi(), alone[1])


@pytest.mark.parametrize("prec,n", [("fp32", 96), ("fp64", 96), ("mixed", 96), ("fp32", 128)])
def test_batch_record_in_half_groups(prec, n):
    # boxes that fill the device alone record and sweep with two planes a CTA
    # when a batch holds several: the same bits as one box by itself
    psis = [zeldovich_psi(n, seed=n + i) for i in range(3)]
    rng = np.random.default_rng(n)
    cot = [rng.standard_normal((n,) * 3) + 1j * rng.standard_normal((n,) * 3) for _ in psis]
    want = []
    sims = [ifdm.Simulation(MFDM, 0.0, XMAX, n, precision=prec) for _ in psis]
    for s, p, c in zip(sims, psis, cot):
        s.set_psi(p, A0)
        s.record_steps(5, 0.01, 2)
        psi, g = s.get_psi(), np.empty_like(c)
        s.adjoint(c, g)
        want.append((psi, g))
        s.set_psi(p, A0)
    got = [np.empty_like(c) for c in cot]
    with ifdm.Batch(sims) as b:
        b.record_steps(5, 0.01, 2)
        psi = [s.get_psi() for s in sims]
        b.adjoint(cot, got)
    for i, s in enumerate(sims):
        assert np.array_equal(psi[i], want[i][0]) and np.array_equal(got[i], want[i][1]), i
        s.set_psi(psis[i], A0)
        s.step(5, 0.01)  # whole groups again
        assert s.state()["device_error"] == 0 and np.array_equal(s.get_psi(), want[i][0]), i
        s.close()


@pytest.mark.parametrize("prec,n", [("fp32", 96), ("fp64", 96), ("mixed", 96), ("fp32", 128)])
def test_full_boxes_side_by_side(prec, n):
    # boxes of a CTA an SM take half groups while another one has work in
    # flight, whole ones alone: the same bits, with the group changing between
    # the calls of one box
    psis = [zeldovich_psi(n, seed=n + i) for i in range(4)]
    want = []
    for p in psis:
        with ifdm.Simulation(MFDM, 0.0, XMAX, n, precision=prec) as s:
            s.set_psi(p, A0)
            s.step(24, 0.01)
            want.append((s.get_psi(), s.get_phi()))
    sims = [ifdm.Simulation(MFDM, 0.0, XMAX, n, precision=prec) for _ in psis]
    for s, p in zip(sims, psis):
        s.set_psi(p, A0)
    for _ in range(5):
        for s in sims:
            s.step(4, 0.01)
    for s, w in zip(sims, want):
        s.synchronize()
        s.step(4, 0.01)
        assert s.state()["device_error"] == 0
        assert np.array_equal(s.get_psi(), w[0]) and np.array_equal(s.get_phi(), w[1])
        s.close()
