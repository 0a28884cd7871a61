"""Loading a wave function behind queued steps (needs a B200)."""

import numpy as np
import pytest

import ifdm_code_b200 as ifdm
from ifdm_code_b200.synthetic_ic import zeldovich_psi

pytestmark = pytest.mark.gpu

MFDM, XMAX, A0 = 2.5e-24, 5.0, 1.0 / 51.0


@pytest.mark.parametrize("prec,n", [("fp64", 16), ("fp32", 64), ("fp32", 128), ("mixed", 128), ("fp64", 128), ("fp32", 256)])
def test_device_psi_is_free_once_set(prec, n):
    # the one-launch boxes and the pass-by-pass ones (128^3 in FP64 arithmetic,
    # 256^3): a tensor overwritten right after set_psi, while steps are queued
    import torch

    x = torch.from_numpy(zeldovich_psi(n, seed=n)).cuda()
    torch.cuda.synchronize()
    with ifdm.Simulation(MFDM, 0.0, XMAX, n, precision=prec) as s:
        s.set_psi(x, A0)
        want = s.get_psi(), s.get_phi()
        s.step(200, 1e-3)
        s.set_psi(x, A0)
        x.zero_()
        got = s.get_psi(), s.get_phi()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("prec", ["fp32", "mixed"])
@pytest.mark.parametrize("n", [16, 48, 64, 128])
@pytest.mark.parametrize("cell0", [0.0, 1000.0])
def test_initial_potential_does_not_depend_on_one_cell(prec, n, cell0):
    # cell (0, 0, 0) empty or in a halo: the other cells' densities must not be
    # rounded relative to it.  Stored psi, the density (to 2^-24 of itself or of
    # its mean) and the transforms' stages then round by some 1e-7, cell by cell
    # at random, against a density of contrast 0.5: below 1e-6 of phi
    psi = zeldovich_psi(n, seed=n, rms_delta=0.5)
    psi[0, 0, 0] = np.sqrt(cell0) * np.abs(psi).mean()
    phi = []
    for p in ("fp64", prec):
        with ifdm.Simulation(MFDM, 0.0, XMAX, n, precision=p) as s:
            s.set_psi(psi, A0)
            phi.append(s.get_phi())
    assert np.linalg.norm(phi[1] - phi[0]) <= 1e-6 * np.linalg.norm(phi[0])
