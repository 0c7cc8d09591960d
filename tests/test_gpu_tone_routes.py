"""FP64 tone calls on either side of the choice between the tensor path and the per-sample kernel (output steps of the
launch, fine steps, tones), against the oracle to 1e-10."""
import numpy as np
import pytest

import fields as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spin,n,k,tones,tensor", [
    ("HALF", 3, 256, (1, 2, 1), False), ("ONE", 3, 255, (1, 2, 1), True), ("HALF", 1024, 256, (0, 0, 1), False),
    ("ONE", 1025, 256, (0, 0, 1), True), ("ONE", 33, 1500, (2, 2, 0), False), ("HALF", 33, 1501, (2, 2, 1), True)])
def test_both_routes(cuda, spin, n, k, tones, tensor):
    import spinsim_b200 as ss
    from spinsim_b200.batch import Batch, Instance
    sq = ss.SpinQuantumNumber[spin]
    p = F.tone_parameters(np.random.default_rng(k), bias=(1e4, 0.0, 2e5, 0.0))
    for axis, count in enumerate(tones):
        p[4 + 24 * axis:28 + 24 * axis].reshape(8, 3)[count:, 1] = 0.0
    field = ss.ToneField({a: p[4 + 24 * a:28 + 24 * a].reshape(8, 3)[:c] for a, c in enumerate(tones) if c},
                         bias=list(p[:4]))
    dt_out = k * 10e-9
    args = (0.0, (n + 0.5) * dt_out, 10e-9, dt_out, sq.plus_z)
    time, u, state, _ = O.evaluate(sq.dimension, O.Field(8), p, *args)
    batch = Batch([Instance(sq, *args, field=field)])
    for lanes, per_sample in ((0, not tensor), (32, not tensor), (16, False)):
        info = Batch([Instance(sq, *args, field=field)], lanes=lanes).launch_info()
        assert info["tile_intervals"] == (1 if per_sample else 32)
    batch.run()
    for r in (batch.result(0), ss.Simulator(field, sq).evaluate(*args)):
        assert np.array_equal(r.time, time)
        assert np.abs(r.time_evolution - u).max() < 1e-10
        assert np.abs(r.state - state).max() < 1e-10
