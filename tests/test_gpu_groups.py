"""The host evaluator's groups: at most ``chunks``, of at least GROUP_BYTES of outputs each, contiguous and whole; the
results do not depend on them (bit for bit, with the lanes and the mixed-spin kernel fixed)."""
import numpy as np
import pytest

import fields as F

pytestmark = pytest.mark.gpu


def instances(n):
    import spinsim_b200 as ss
    import spinsim_b200.batch as B
    out = []
    for k in range(n):
        rng = np.random.default_rng(k)
        s = ss.SpinQuantumNumber.ONE if k % 3 == 0 else ss.SpinQuantumNumber.HALF
        p = F.tone_parameters(rng)
        tones = {a: p[4 + 24 * a:28 + 24 * a].reshape(8, 3) for a in range(3)}
        out.append(B.Instance(s, 0.0, float(rng.uniform(20e-6, 400e-6)), 10e-9, 1e-6, s.plus_x, field=ss.ToneField(tones)))
    return out


@pytest.mark.parametrize("group_bytes,expected", [(1, 5), (1 << 40, 1), (200_000, None)])
def test_groups(cuda, monkeypatch, group_bytes, expected):
    import torch
    import spinsim_b200.batch as B
    insts = instances(23)
    monkeypatch.setattr(B.Evaluator, "GROUP_BYTES", group_bytes)
    ev = B.Evaluator(chunks=5, lanes=1, force_mixed=True)
    groups = ev.groups(insts)
    assert groups[0][0] == 0 and groups[-1][1] == 23 and all(a[1] == b[0] for a, b in zip(groups, groups[1:]))
    assert len(groups) == expected if expected else 1 < len(groups) < 5
    ref = B.Batch(insts, lanes=1, force_mixed=True)
    ref.run()
    torch.cuda.synchronize()
    res = ev.evaluate(insts)
    for k in range(23):
        r = ref.result(k)
        assert np.array_equal(res[k].state, r.state) and np.array_equal(res[k].time_evolution, r.time_evolution)
        assert np.array_equal(res[k].time, r.time) and np.array_equal(res[k].spin, r.spin)
