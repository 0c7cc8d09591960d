"""Calls far from time zero, where the rounding of sample times shows: beyond 2^20 steps the samples follow the
reference's running sum of steps, and FP64 tone fields with large phases are sampled one by one, as the oracle does.

Tolerance.  Sample times agree to the last bit, so what is left are an interval's own roundings: its operators agree
to 1e-12 where every sample's phase w t is rounded by up to w t 2^-53, 1e-9 here, in time zero's absence.  The
start time puts whole calls on one side of each line: t0 = 0 below, t0 = 2^21 steps above.
"""
import math

import numpy as np
import pytest

import fields as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DT = 1e-8


@pytest.mark.parametrize("t0", [0.0, 2.0 ** 21 * DT, -(2.0 ** 21) * DT])
@pytest.mark.parametrize("spin,rotating,lanes", [("HALF", True, 1), ("HALF", False, 4), ("ONE", True, 8)])
def test_drive(cuda, spin, rotating, lanes, t0):
    import spinsim_b200 as ss
    sq = ss.SpinQuantumNumber[spin]
    field, code = (F.rabi, 2) if spin == "HALF" else (F.rabi_one, 3)
    params = [math.tau * 7e5, math.tau * 2e3]
    sim = ss.Simulator(field, sq, use_rotating_frame=rotating, lanes=lanes)
    n, k = 40, 64
    end = t0 + (n + 0.5) * k * DT
    r = sim.evaluate(t0, end, DT, k * DT, sq.plus_z, params)
    time, u, _, _ = O.evaluate(sq.dimension, O.Field(code), params, t0, end, DT, k * DT, sq.plus_z, rotating=rotating)
    assert np.array_equal(r.time, time)
    assert np.abs(r.time_evolution - u).max() < 1e-12


@pytest.mark.parametrize("t0", [0.0, 0.1])
def test_tones(cuda, t0):
    """t0 = 0.1 s: phases of 6e5 rad, off the tensor path; t0 = 0: on it."""
    import spinsim_b200 as ss
    p = F.tone_parameters(np.random.default_rng(3))
    tones = {a: p[4 + 24 * a:28 + 24 * a].reshape(8, 3) for a in range(3)}
    half = ss.SpinQuantumNumber.HALF
    sim = ss.Simulator(ss.ToneField(tones), half)
    end = t0 + 60.5e-6
    r = sim.evaluate(t0, end, DT, 1e-6, half.plus_z)
    _, u, _, _ = O.evaluate(2, O.Field(8), p, t0, end, DT, 1e-6, half.plus_z)
    assert np.abs(r.time_evolution - u).max() < 1e-12
