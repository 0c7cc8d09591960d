"""Field samples at the reference's own times: offsets from the running sum of the fine steps
(spinsim/__init__.py:624-645, :693-752, :759-791, :836), rounded as it rounds them.

A field with edges on the step grid shows which side of an edge a sample falls: Heun samples at the steps' ends and
Euler at their middles, and with decimal steps the rounding of a sample's time decides.  The field is on x alone,
so an output step's operator is exp(-i theta Jx) with theta the weighted sum of its samples, which numpy forms at
the reference's times; one sample on the other side turns theta by dt B / 2, 2e-4 at least.  Tolerance 1e-10, the FP64
contract (and 1e-6, the FP32-bulk one, on the final state).

A fast drive in its rotating frame adds the roundings of its sample times up over a call: states against the oracle
to 1e-10 at a million steps.
"""
import math

import numpy as np
import pytest

import fields as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

B = 2 * math.pi * 25e3


def square_wave(time_sample, sweep_parameters, field_sample):
    """Amplitude on x for every other 7 steps; parameters: half a step, 1 for edges at the steps' middles, amplitude."""
    field_sample[0] = 0.0
    half_steps = math.floor(time_sample / sweep_parameters[0])
    if math.floor(math.floor((half_steps + sweep_parameters[1]) / 2.0) / 7.0) % 2 == 1:
        field_sample[0] = sweep_parameters[2]


def angles(value, integration, t0, dt, dt_out, n, k):
    """theta of every output step, of field value(t) on x."""
    t_c = t0 + dt_out * np.arange(n)
    t_fine, theta = t_c.copy(), np.zeros(n)
    points = [(0.0, 0.5), (dt, 0.5)] if integration == "heun" else [(0.5 * dt, 1.0)]
    for _ in range(k):
        for offset, weight in points:
            theta += weight * dt * value(((t_fine + offset) - t_c) + t_c)
        t_fine = t_fine + dt
    return theta


def operators(theta, dim):
    c, s = np.cos(theta / 2), np.sin(theta / 2)
    if dim == 2:
        return np.stack([c, -1j * s, -1j * s, c], -1).reshape(-1, 2, 2)
    r = -1j * math.sqrt(2.0) * c * s
    return np.stack([c * c, r, -s * s, r, c * c - s * s, r, -s * s, r, c * c], -1).reshape(-1, 3, 3)


def compare(sim_field, value, spin, integration, dt_ns, k, lanes, t0, params=(0.0,)):
    import spinsim_b200 as ss
    sq = ss.SpinQuantumNumber[spin]
    n, dt_out = 600, k * dt_ns * 1e-9
    t1 = t0 + (n + 0.5) * dt_out
    dt, n_found, k_found, _ = O.normalise_steps(t0, t1, dt_ns * 1e-9, dt_out)
    assert (n_found, k_found) == (n, k)
    u = operators(angles(value, integration, t0, dt, dt_out, n, k), sq.dimension)
    final = np.asarray(sq.plus_z, complex)
    for i in range(n - 1):
        final = u[i] @ final
    for precision in (ss.Precision.FP64, ss.Precision.FP32_BULK):
        sim = ss.Simulator(sim_field, sq, integration_method=ss.IntegrationMethod(integration), lanes=lanes,
                           precision=precision, use_rotating_frame=lanes == 1)
        r = sim.evaluate(t0, t1, dt_ns * 1e-9, dt_out, sq.plus_z, params)
        if precision == ss.Precision.FP64:
            assert np.abs(r.time_evolution - u).max() < 1e-10
        assert np.abs(r.state[-1] - final).max() < (1e-10 if precision == ss.Precision.FP64 else 1e-6)


FORMS = [("HALF", "heun", 20.0, 50, 1, 0.0), ("HALF", "heun", 50.0, 20, 4, 0.0), ("ONE", "heun", 50.0, 20, 1, 1e-3),
         ("HALF", "euler", 20.0, 50, 4, 0.0), ("ONE", "euler", 50.0, 20, 1, 0.0), ("HALF", "euler", 30.0, 33, 1, -3e-4)]


@pytest.mark.parametrize("spin,integration,dt_ns,k,lanes,t0", FORMS)
def test_edges_of_a_user_field(cuda, spin, integration, dt_ns, k, lanes, t0):
    half, middles = 0.5e-9 * dt_ns, 1.0 if integration == "euler" else 0.0

    def value(t):
        return np.where(np.floor(np.floor((np.floor(t / half) + middles) / 2.0) / 7.0) % 2 == 1, B, 0.0)

    compare(square_wave, value, spin, integration, dt_ns, k, lanes, t0, (half, middles, B))


@pytest.mark.parametrize("spin,integration,dt_ns,k,lanes,t0", FORMS)
def test_ends_of_an_interpolated_table(cuda, spin, integration, dt_ns, k, lanes, t0):
    """A linear table that is zero outside: its ends, on the grid of sample times, are edges."""
    import spinsim_b200 as ss
    first = 0.5e-9 * dt_ns if integration == "euler" else 0.0
    dt_out = k * dt_ns * 1e-9
    knots = np.array([t0 + first + i * dt_out + 7e-9 * dt_ns for i in (35, 41, 202, 380)])
    amplitude = B * np.array([1.0, 0.25, 1.0, 0.75])

    def value(t):
        return np.where((t >= knots[0]) & (t <= knots[-1]), np.interp(t, knots, amplitude), 0.0)

    compare(ss.TabulatedField({0: (knots, amplitude)}, order=1, zero_boundary=True), value, spin, integration, dt_ns, k,
            lanes, t0)


@pytest.mark.parametrize("spin,mhz,dt_ns,k,steps", [("HALF", 10, 10.0, 100, 1000000), ("HALF", 10, 2.0, 500, 500000),
                                                    ("ONE", 5, 20.0, 50, 200000)])
def test_fast_drive_over_many_steps(cuda, spin, mhz, dt_ns, k, steps):
    import spinsim_b200 as ss
    sq = ss.SpinQuantumNumber[spin]
    field, code = (F.rabi, 2) if spin == "HALF" else (F.rabi_one, 3)
    params = [math.tau * mhz * 1e6, math.tau * 50e3]
    dt_out = k * dt_ns * 1e-9
    end = (steps // k + 0.5) * dt_out
    r = ss.Simulator(field, sq).evaluate(0.0, end, dt_ns * 1e-9, dt_out, sq.plus_z, params)
    time, u, state, _ = O.evaluate(sq.dimension, O.Field(code), params, 0.0, end, dt_ns * 1e-9, dt_out, sq.plus_z)
    assert np.array_equal(r.time, time)
    assert np.abs(r.time_evolution - u).max() < 1e-10
    assert np.abs(r.state - state).max() < 1e-10
