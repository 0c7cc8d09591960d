"""Piecewise constant fields whose frame does not turn, which the table kernels integrate in runs between knots,
against the oracle's step by step: knots on every channel's own times, on sample times exactly (dyadic steps),
several inside one step, before the call's start and after its end, few and many against the output steps,
split over lanes, with the frame on (no z field) and off.

Tolerances: FP64 to 1e-12 (an interval's at most 64 steps each round a few times 2^-53, on operators of size
one; the oracle's squarings 24 times as often), FP32-bulk within the 1e-6 contract on the final state.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DT = 2.0 ** -24
B = 2 * np.pi * 3e5


def tables(kind, seed, n_out, k, with_z):
    rng = np.random.default_rng(seed)
    end = n_out * k * DT
    out = []
    for c in range(3):
        if kind == "on_samples":  # multiples of half a step: Heun's ends and Euler's middles
            t = np.unique(rng.integers(-4, 2 * n_out * k + 8, 40)) * (DT / 2)
        elif kind == "many":  # several knots in one step
            t = np.sort(rng.uniform(-DT, end + DT, 3 * n_out * k))
        else:  # few, none near the end
            t = np.sort(rng.uniform(0.1 * end, 0.7 * end, 7))
        a = rng.uniform(-B, B, t.size) * (1.0 if c < 2 or with_z else 0.0)
        out.append((t, a))
    if kind == "few":
        out[1] = (out[0][0], out[1][1])  # two channels of one time array
    return out


@pytest.mark.parametrize("kind", ["few", "many", "on_samples"])
@pytest.mark.parametrize("zero_boundary", [False, True])
@pytest.mark.parametrize("integration,spin,lanes,k,rotating", [
    ("magnus_cf4", "half", 1, 20, True), ("magnus_cf4", "one", 1, 13, False), ("magnus_cf4", "half", 4, 64, False),
    ("heun", "half", 1, 7, False), ("euler", "one", 2, 9, True)])
def test_runs_against_steps(cuda, kind, zero_boundary, integration, spin, lanes, k, rotating):
    import spinsim_b200 as ss
    sq = ss.SpinQuantumNumber[spin.upper()]
    n_out = 75
    tabs = tables(kind, seed=len(kind) + 10 * k, n_out=n_out, k=k, with_z=not rotating)
    shared = {id(tabs[0][0]): tabs[0][0]}
    field = ss.TabulatedField({c: (shared.get(id(tabs[c][0]), tabs[c][0]), tabs[c][1]) for c in range(3)}, order=0,
                              zero_boundary=zero_boundary)
    end = (n_out + 0.5) * k * DT
    oracle_field = O.Field(9, [(t, a, 0, zero_boundary) for t, a in tabs])
    _, u, st, _ = O.evaluate(sq.dimension, oracle_field, [1.0, 1.0, 0.0, 1.0], 0.0, end, DT, k * DT, sq.plus_x,
                             integration=integration, rotating=rotating)
    for precision in (ss.Precision.FP64, ss.Precision.FP32_BULK):
        sim = ss.Simulator(field, sq, integration_method=ss.IntegrationMethod(integration), use_rotating_frame=rotating,
                           precision=precision, lanes=lanes)
        r = sim.evaluate(0.0, end, DT, k * DT, sq.plus_x)
        assert r.time_evolution.shape == u.shape
        if precision == ss.Precision.FP64:
            assert np.abs(r.time_evolution - u).max() < 1e-12
        assert np.abs(r.state[-1] - st[-1]).max() < (1e-11 if precision == ss.Precision.FP64 else 1e-6)
