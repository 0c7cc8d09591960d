"""Results in one block: reading an array leaves what a caller has set in another, and arrays that were not read
before the device tensors were handed out show what has been written to those."""
import numpy as np
import pytest

import spinsim_b200 as ss


def results(n=5, d=2):
    block = ss._Block(n, d, False, 256, "cpu")
    block.words.zero_()
    return ss.Results._from_block(block, None, None, 0.0)


@pytest.mark.parametrize("kept", ["time", "time_evolution", "state", "spin"])
def test_reading_keeps_what_was_set(kept):
    r, mine = results(), np.full(3, 7.0)
    setattr(r, kept, mine)
    for name in ("time", "time_evolution", "state", "spin"):
        getattr(r, name)
    assert getattr(r, kept) is mine


def test_device_writes_after_a_read(monkeypatch):
    view = ss._Block.host_arrays  # of a block on the host: a view, where one on the device is copied
    monkeypatch.setattr(ss._Block, "host_arrays", lambda block: {k: v.copy() for k, v in view(block).items()})
    monkeypatch.setattr(ss, "_to_numpy", lambda x: x.numpy().copy())
    r = results()
    assert not r.time.any()
    d = r.device_arrays
    d["time"].fill_(1.0)
    d["state"].fill_(2.0)
    assert not r.time.any()  # read before
    assert (r.state == 2.0).all() and not r.spin.any()
