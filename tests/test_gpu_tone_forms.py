"""FP64 tone fields on the tensor path against the same fields sampled one by one, over the forms that the path takes:
step counts around its segments, phases and restarts, starts on both sides of time zero and just before a change of
exponent, units of time, spins, frames, axes without tones.  A ninth tone of no amplitude sends a field to the
per-sample kernel.  Tolerance: the FP64 contract of 1e-10."""
import math
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = [1, 2, 3, 4, 5, 7, 8, 9, 12, 31, 33, 39, 40, 41, 79, 81, 100, 479, 480, 481, 999]


@pytest.mark.parametrize("seed", range(len(STEPS)))
def test_against_single_samples(cuda, seed):
    import spinsim_b200 as ss
    from spinsim_b200.batch import Batch, Instance
    rng, values = random.Random(seed), np.random.default_rng(seed)
    half, one = ss.SpinQuantumNumber.HALF, ss.SpinQuantumNumber.ONE
    k, n = STEPS[seed], rng.choice([1, 7, 8, 31, 33, 64, 100])
    unit = 10.0 ** rng.choice([0, 0, -3, 3])
    dt = rng.choice([1e-8, 2e-8, 2.0 ** -24]) * unit
    t0 = rng.choice([0.0, -1e-4, 2.0 ** -10 - 1e-6]) * unit
    rate, amplitude = rng.choice([1e5, 1e6, 1e7]) / unit, rng.choice([1e3, 6e4, 6e5]) / unit
    tones = {c: np.stack([values.uniform(0, rate, m), values.uniform(0, amplitude, m), values.uniform(0, math.tau, m)], 1)
             for c, m in enumerate((rng.choice([1, 3, 8]), rng.choice([0, 2, 8]), rng.choice([0, 8]))) if m}
    padded = dict(tones)
    padded[0] = np.concatenate([tones[0], np.zeros((9 - len(tones[0]), 3))])
    bias = [0.0, 0.0, rng.choice([0.0, 3e5, 6e6]) / unit]
    spins = rng.choice([[half], [one], [half, one, half]])
    results = []
    for field in (tones, padded):
        insts = [Instance(s, t0, t0 + (max(1, n // (i + 1)) + 0.25) * k * dt, dt, k * dt, s.plus_x,
                          field=ss.ToneField(field, bias=bias)) for i, s in enumerate(spins)]
        # a fixed lane count leaves the tensor path to the fields alone
        batch = Batch(insts, lanes=1, use_rotating_frame=seed % 3 != 0)
        batch.run()
        results.append([batch.result(i) for i in range(len(spins))])
    for a, b in zip(*results):
        assert np.array_equal(a.time, b.time)
        assert np.abs(a.time_evolution - b.time_evolution).max() < 1e-10
        assert np.abs(a.state - b.state).max() < 1e-10
