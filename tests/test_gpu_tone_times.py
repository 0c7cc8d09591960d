"""FP64 tone fields on the tensor path sample at the reference's running-sum times (spinsim/__init__.py:836).

The sum's rounding is the same for all steps of the same exponent, so a resonant drive adds its phases up over a
call: states and operators against the oracle to 1e-10, the FP64 contract.  The phases w t stay below 1e5 rad and
w K t 2^-53 below 2e-9, where fields take this path.
"""
import math

import numpy as np
import pytest

import fields as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def drive(mhz, half_amplitude_hz):
    """F.rabi on the resonance as tones: 2 A cos(w t) on x, w on z."""
    import spinsim_b200 as ss
    w = math.tau * mhz * 1e6
    return ss.ToneField({0: [[w, 2.0 * math.tau * half_amplitude_hz, 0.5 * math.pi]]}, bias=[0.0, 0.0, w])


@pytest.mark.parametrize("spin,mhz,dt_ns,k,n,t0", [
    ("HALF", 10, 2.0, 100, 4000, 0.0), ("HALF", 10, 10.0, 100, 1500, 0.0), ("ONE", 10, 10.0, 101, 1400, 0.0),
    ("HALF", 5, 20.0, 50, 3000, 0.0), ("ONE", 1, 10.0, 100, 10000, 0.0), ("HALF", 10, 2.0, 99, 4000, -4e-4),
    ("ONE", 5, 20.0, 51, 2000, 1e-3), ("HALF", 0.1, 10.0, 2000, 300, 0.0), ("ONE", 0.1, 10.0, 1003, 500, 0.0)])
def test_resonant_drive(cuda, spin, mhz, dt_ns, k, n, t0):
    import spinsim_b200 as ss
    sq = ss.SpinQuantumNumber[spin]
    field, code = drive(mhz, 50e3 if mhz >= 1 else 5e3), 2 if spin == "HALF" else 3
    dt_out = k * dt_ns * 1e-9
    t1 = t0 + (n + 0.5) * dt_out
    args = (t0, t1, dt_ns * 1e-9, dt_out, sq.plus_z)
    r = ss.Simulator(field, sq).evaluate(*args)
    params = [math.tau * mhz * 1e6, math.tau * (50e3 if mhz >= 1 else 5e3)]
    time, u, state, _ = O.evaluate(sq.dimension, O.Field(code), params, t0, t1, dt_ns * 1e-9, dt_out, sq.plus_z)
    assert np.array_equal(r.time, time)
    assert np.abs(r.time_evolution - u).max() < 1e-10
    assert np.abs(r.state - state).max() < 1e-10


@pytest.mark.parametrize("n_pieces", [3, 7])
def test_pieces_round_as_the_whole_call(cuda, n_pieces):
    """Pieces that begin anywhere in a block of eight output steps (1.0 to 1.4 ms: one exponent)."""
    import spinsim_b200 as ss
    from spinsim_b200.batch import Batch, Instance
    from spinsim_b200.shard import Piece, piece_ranges
    sq = ss.SpinQuantumNumber.HALF
    p = F.tone_parameters(np.random.default_rng(5))
    field = ss.ToneField({a: p[4 + 24 * a:28 + 24 * a].reshape(8, 3) for a in range(3)}, bias=list(p[:4]))
    inst = Instance(sq, 1e-3, 1e-3 + 401.5e-6, 10e-9, 1e-6, sq.plus_z, field=field)
    whole = Batch([inst])
    whole.run()
    pieces = [Piece(inst, first, count) for first, count in piece_ranges(401, n_pieces)]
    assert any(x.first % 8 for x in pieces)
    assert np.array_equal(np.concatenate([x.results().time_evolution for x in pieces]), whole.result(0).time_evolution)
