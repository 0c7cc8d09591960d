"""Linked user fields kept between plans: every simulator runs its own field, however many were linked between."""
import numpy as np
import pytest

import spinsim_b200 as ss

pytestmark = pytest.mark.gpu


def make_field(rate):
    def get_field(time_sample, sweep_parameters, field_sample):
        field_sample[0] = 0
        field_sample[1] = 0
        field_sample[2] = rate
    return get_field


@pytest.mark.parametrize("count", [2, 9])  # within the links kept, and more
def test_each_simulator_runs_its_own_field(count):
    fields = [make_field(1e5 * (k + 1)) for k in range(count)]
    for spin in (ss.SpinQuantumNumber.HALF, ss.SpinQuantumNumber.ONE):
        m = np.array([0.5, -0.5]) if spin.dimension == 2 else np.array([1.0, 0.0, -1.0])
        psi0 = np.full(spin.dimension, spin.dimension ** -0.5, complex)
        for k in list(range(count)) * 2:  # the second time from the kept links, or linked again
            sim = ss.Simulator(fields[k], spin, exponentiation_method=ss.ExponentiationMethod.LIE_TROTTER)
            r = sim.evaluate(0.0, 1e-4, 1e-7, 1e-6, psi0)
            exact = psi0 * np.exp(-1j * np.outer(r.time, m) * 1e5 * (k + 1))
            # 1000 steps, each with a few roundings of 1.1e-16, and phases to 90 rad rounded once: below 1e-12
            np.testing.assert_allclose(r.state, exact, rtol=0, atol=2e-12)
