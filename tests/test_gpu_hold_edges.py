"""Piecewise constant fields with knots on the grid of sample times of decimal steps, where the rounding of the
reference's running sum (spinsim/__init__.py:836) decides the side of a knot that a sample falls on, and with
several knots inside one step, few enough in all for the table kernels' runs between knots; against the oracle
step by step.  One sample on the other side changes an operator by dt B / 2, 1e-3 at least.

Tolerances: the FP64 contract of 1e-10 (operators and states), FP32-bulk's 1e-6 on the final state.
"""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

B = 2 * math.pi * 25e3


def knots(kind, rng, integration, t0, dt, n_steps):
    if kind == "on_grid":
        at = np.unique(rng.integers(3, n_steps, 40)) + (0.5 if integration == "euler" else 0.0)
        return t0 + at * dt
    groups = np.sort(rng.choice(np.arange(3, n_steps // 400), 4, replace=False)) * 400
    return t0 + np.concatenate([(g + np.sort(rng.uniform(0.05, 0.95, 5))) * dt for g in groups])


@pytest.mark.parametrize("kind", ["on_grid", "several_in_a_step"])
@pytest.mark.parametrize("spin,integration,dt_ns,k,lanes,t0,zero_boundary", [
    ("HALF", "heun", 20.0, 50, 1, 0.0, False), ("HALF", "heun", 50.0, 20, 4, 0.0, True),
    ("ONE", "heun", 50.0, 20, 1, 1e-3, False), ("HALF", "euler", 30.0, 33, 4, -3e-4, False),
    ("ONE", "euler", 50.0, 20, 1, 0.0, True), ("HALF", "heun", 50.0, 20, 1, 0.5, False),
    ("HALF", "magnus_cf4", 20.0, 50, 1, 0.0, True)])
def test_knots_against_the_oracle(cuda, kind, spin, integration, dt_ns, k, lanes, t0, zero_boundary):
    import spinsim_b200 as ss
    sq = ss.SpinQuantumNumber[spin]
    n, dt, dt_out = 600, dt_ns * 1e-9, k * dt_ns * 1e-9
    t1 = t0 + (n + 0.5) * dt_out
    rng = np.random.default_rng(k + lanes)
    tables = []
    for c in range(2):
        t = knots(kind, rng, integration, t0, dt, n * k)
        tables.append((t, rng.uniform(0.5, 1.0, t.size) * np.where(np.arange(t.size) % 2, B, -B)))
    none = (np.array([t0, t1]), np.zeros(2))
    reference = O.Field(9, [(t, a, 0, zero_boundary) for t, a in [*tables, none]])
    _, u, st, _ = O.evaluate(sq.dimension, reference, [1.0, 1.0, 0.0, 1.0], t0, t1, dt, dt_out, sq.plus_z,
                             integration=integration)
    field = ss.TabulatedField(dict(enumerate(tables)), order=0, zero_boundary=zero_boundary)
    for precision in (ss.Precision.FP64, ss.Precision.FP32_BULK):
        sim = ss.Simulator(field, sq, integration_method=ss.IntegrationMethod(integration), lanes=lanes,
                           precision=precision)
        r = sim.evaluate(t0, t1, dt, dt_out, sq.plus_z)
        assert r.time_evolution.shape == u.shape
        if precision == ss.Precision.FP64:
            assert np.abs(r.time_evolution - u).max() < 1e-10
            assert np.abs(r.state - st).max() < 1e-10
        assert np.abs(r.state[-1] - st[-1]).max() < (1e-10 if precision == ss.Precision.FP64 else 1e-6)
