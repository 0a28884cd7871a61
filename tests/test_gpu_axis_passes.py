"""Pipelined axis passes over a caller's own field, and the diagnostics built
on one-axis passes (needs a B200).

From 256 points on ifdm_fft3d and ifdm_fft_slab run the ring-fed kernels of the
steps when the field starts on a 16-byte boundary (bulk copies); any other field
keeps the plain kernels.  Both are checked against torch's FFT; tolerances are a
few rounding steps per stage (1e-13, 2e-6) as in the 3-D transform tests.
"""

import numpy as np
import pytest

import ifdm_code_b200 as ifdm
from ifdm_code_b200.synthetic_ic import zeldovich_psi

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-13, "fp32": 2e-6, "mixed": 2e-7}


def _rel(a, b):
    return float((a - b).abs().norm() / b.abs().norm())


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("n,planes", [(256, 1), (256, 19), (256, 256), (512, 3)])
def test_slab_axes_256_and_up(n, planes, prec):
    import torch

    from ifdm_code_b200.slab import library_axis_op

    op = library_axis_op(prec)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n + planes)
    dt = torch.complex128 if prec == "fp64" else torch.complex64
    for axis, shape, dim in ((2, (planes, n, n), 2), (1, (planes, n, n), 1), (0, (n, planes, n), 0)):
        for sign in (-1, +1):
            x = torch.randn(shape, generator=gen, device="cuda", dtype=torch.complex128).to(dt)
            ref = x.to(torch.complex128)
            ref = torch.fft.fft(ref, dim=dim) if sign < 0 else torch.fft.ifft(ref, dim=dim) * n
            got = op(x.clone(), axis, sign, n, planes)
            assert _rel(got.to(torch.complex128), ref) <= TOL[prec], (axis, sign)


@pytest.mark.parametrize("n", [32, 256])
def test_fft3d_of_a_field_off_the_16_byte_grid(n):
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    buf = torch.randn(n**3 + 1, generator=gen, device="cuda", dtype=torch.complex64)
    x = buf[1:].view(n, n, n)
    assert x.data_ptr() % 16 == 8
    ref = torch.fft.fftn(x.to(torch.complex128))
    first = buf[0].clone()
    ifdm.fft3d_(x, -1)
    assert _rel(x.to(torch.complex128), ref) <= TOL["fp32"]
    assert torch.equal(buf[0], first)


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("n", [16, 48, 128, 256])
def test_diagnostics_against_numpy(n, prec):
    psi0 = zeldovich_psi(n, seed=n, rms_delta=0.3)
    with ifdm.Simulation(2.5e-24, 1e-63, 5.0, n, precision=prec) as s:
        s.set_psi(psi0, 0.05)
        s.step(2, 0.01)
        psi, phi = s.get_psi(), s.get_phi()
        e = s.energies()
        edges = np.linspace(0.0, 0.9 * n, 23)  # k = 0 in the first bin, the corners in the last ones
        ps = s.power_spectrum(22, edges)
        again = s.power_spectrum(22, edges)
    rho = np.abs(psi) ** 2
    k = np.arange(n)
    k = np.where(k < n // 2, k, k - n).astype(float)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    L = 10.0 / 0.677
    power = np.abs(np.fft.fftn(rho / rho.mean() - 1.0)) ** 2
    b = np.digitize(np.sqrt(k2), edges) - 1
    for i in range(22):
        m = b == i
        assert ps["modes"][i] == m.sum()
        if m.any():
            assert ps["k"][i] == pytest.approx(np.sqrt(k2[m]).mean() * 2 * np.pi / L, rel=1e-12)
            assert ps["pk"][i] == pytest.approx(power[m].mean() * L**3 / n**6, rel=1e-9)
    assert all(np.array_equal(ps[q], again[q]) for q in ("k", "pk", "modes"))
    grad2 = (k2 * np.abs(np.fft.fftn(psi)) ** 2).sum() / n**6 * (2 * np.pi / L) ** 2
    want = {"mean_rho": rho.mean(), "mean_grad2": grad2, "mean_phi_rho": (phi * rho).mean(), "mean_rho2": (rho**2).mean()}
    for q, w in want.items():
        assert e[q] == pytest.approx(w, rel=1e-11), q
    assert ps["mean_rho"] == pytest.approx(rho.mean(), rel=1e-12)


@pytest.mark.parametrize("n,prec", [(128, "fp64"), (128, "mixed"), (256, "fp64"), (256, "fp32"), (256, "mixed")])
def test_adjoint_on_ring_passes(n, prec, monkeypatch):
    # the adjoint drift's z transforms on the ring-fed kernels against the plain
    # ones: a step and its adjoint are 12 transforms each, three steps, every
    # transform to TOL
    psi0 = zeldovich_psi(n, seed=n)
    rng = np.random.default_rng(n)
    cot = rng.standard_normal((n,) * 3) + 1j * rng.standard_normal((n,) * 3)
    out = []
    for plain in (False, True):
        if plain:
            monkeypatch.setenv("IFDM_NO_TMA", "1")
        else:
            monkeypatch.delenv("IFDM_NO_TMA", raising=False)
        with ifdm.Simulation(2.5e-24, 0.0, 5.0, n, precision=prec) as s:
            s.set_psi(psi0, 1.0 / 51.0)
            s.record_steps(3, 0.01, 2)
            out.append(np.empty_like(cot))
            s.adjoint(cot, out[-1])
    assert np.linalg.norm(out[0] - out[1]) <= 72 * TOL[prec] * np.linalg.norm(out[1])


@pytest.mark.parametrize("n", [256, 512])
def test_two_rows_per_thread_same_bits(n, monkeypatch):
    # FP32 from 256 points on: two lines a thread, the arithmetic of the
    # one-line kernels
    psi0 = zeldovich_psi(n, seed=n)
    out = []
    for plain in (False, True):
        if plain:
            monkeypatch.setenv("IFDM_NO_PAIR", "1")
        else:
            monkeypatch.delenv("IFDM_NO_PAIR", raising=False)
        with ifdm.Simulation(2.5e-24, 1e-63, 5.0, n, precision="fp32") as s:
            s.set_psi(psi0, 1.0 / 51.0)
            s.step(4, 0.01)
            out.append((s.get_psi(), s.get_phi()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
