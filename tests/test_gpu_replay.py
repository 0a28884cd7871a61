"""The adjoint's replay retraces the recorded steps exactly (needs a B200)."""

import numpy as np
import pytest

import ifdm_code_b200 as ifdm
from ifdm_code_b200.synthetic_ic import zeldovich_psi

pytestmark = pytest.mark.gpu

MFDM, XMAX, A0 = 2.5e-24, 5.0, 1.0 / 51.0


@pytest.mark.parametrize("prec", ["mixed", "fp32"])
@pytest.mark.parametrize("n", [16, 64, 128, 256])
def test_replay_of_a_recording_that_follows_steps(n, prec):
    # three steps, then five recorded ones in one segment: the sweep leaves the
    # state before the last recorded step, which is the state of seven steps
    # (stochastic rounding takes its salt from the step counter)
    psi0 = zeldovich_psi(n, seed=n)
    with ifdm.Simulation(MFDM, 0.0, XMAX, n, precision=prec) as s:
        s.set_psi(psi0, A0)
        s.step(7, 0.01)
        want = s.get_psi(), s.get_phi()
        s.set_psi(psi0, A0)
        s.step(3, 0.01)
        s.record_steps(5, 0.01, 5)
        g = np.empty_like(psi0)
        s.adjoint(psi0 / np.abs(psi0).mean(), g)
        assert np.array_equal(s.get_psi(), want[0]) and np.array_equal(s.get_phi(), want[1])
