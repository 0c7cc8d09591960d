"""The tile products that the time evolution writes for the state scan, where some tiles of 32 output steps hold SU(2)
elements and others 3 x 3 operators (spin one with a quadratic shift in part of the call), in batches and in long
single calls, and batches of tone fields that take different kernels: the states equal the serial propagation of
the returned operators.

Tolerance: n products of operators, each rounding at most about 16 2^-53, linearly: 2^-49 n.
"""
import math

import numpy as np
import pytest

import fields as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def late_shift(time_sample, sweep_parameters, field_sample):
    """A drive whose quadratic shift is on between two times only."""
    field_sample[0] = sweep_parameters[0] * math.cos(sweep_parameters[1] * time_sample)
    field_sample[1] = 0.0
    field_sample[2] = sweep_parameters[1]
    field_sample[3] = 0.0
    if sweep_parameters[2] < time_sample < sweep_parameters[3]:
        field_sample[3] = 3e4


def check(time_evolution, state, psi0):
    ref = O.state(np.ascontiguousarray(time_evolution), np.asarray(psi0, complex))
    assert np.abs(state - ref).max() < 2.0 ** -49 * len(ref) + 1e-15


@pytest.mark.parametrize("precision", ["FP64", "FP32_BULK"])
@pytest.mark.parametrize("on,off", [(2.0, 1.0), (-1.0, 2.0), (0.3, 0.31), (0.5, 0.9)])
def test_shift_in_part_of_the_call(cuda, on, off, precision):
    import spinsim_b200 as ss
    import spinsim_b200.batch as B
    one, p = ss.SpinQuantumNumber.ONE, ss.Precision[precision]
    n = 9000
    end = (n + 0.5) * 1e-7
    params = [3e4, 4e6, on * end, off * end]
    r = ss.Simulator(late_shift, one, precision=p).evaluate(0.0, end, 2.5e-8, 1e-7, one.plus_x, params)
    check(r.time_evolution, r.state, one.plus_x)
    insts = [B.Instance(one, 0.0, (m + 0.5) * 1e-7, 2.5e-8, 1e-7, one.plus_z,
                        sweep_parameters=[3e4, 4e6, on * m * 1e-7, off * m * 1e-7]) for m in (3000, 1, 33, 700)]
    b = B.Batch(insts, get_field=late_shift, precision=p, lanes=1)
    b.run()
    for k, i in enumerate(insts):
        check(b.result(k).time_evolution, b.result(k).state, i.state_init)


@pytest.mark.parametrize("lanes", [0, 1, 2])
def test_tone_fields_of_both_kernels_in_one_batch(cuda, lanes):
    """FP64 tones: instances of the tensor path, with more than eight tones on an axis, and with a quadratic shift."""
    import spinsim_b200 as ss
    import spinsim_b200.batch as B
    half, one = ss.SpinQuantumNumber.HALF, ss.SpinQuantumNumber.ONE
    insts = []
    for k, (s, n, tones, q) in enumerate([(half, 100, 8, 0.0), (one, 333, 8, 0.0), (half, 64, 11, 0.0),
                                          (one, 200, 3, 2e4), (one, 1, 8, 0.0), (half, 31, 1, 5.0)]):
        rng = np.random.default_rng(k)
        t = {a: np.stack([rng.uniform(0, 6e6, tones), rng.uniform(0, 6e4, tones), rng.uniform(0, 6.28, tones)], 1)
             for a in range(3)}
        insts.append(B.Instance(s, 0.0, (n + 0.5) * 1e-6, 1e-6 / (20 + k), 1e-6, s.plus_x,
                                field=ss.ToneField(t, bias=[0.0, 0.0, 1e5, q])))
    b = B.Batch(insts, lanes=lanes)
    b.run()
    for k, i in enumerate(insts):
        r = b.result(k)
        check(r.time_evolution, r.state, i.state_init)
        alone = B.Batch([i], lanes=1, force_mixed=True)
        alone.run()
        a = alone.result(0)
        assert np.abs(r.time_evolution - a.time_evolution).max() < 1e-12
        if lanes == 1:  # the route depends on the instance alone
            assert np.array_equal(r.time_evolution, a.time_evolution)
