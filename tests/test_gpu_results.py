"""Results of small calls share one device allocation and reach the host in one copy; those of large calls are
tensors of their own.  Both give the same arrays, on the host and on the device, in any order of access."""
import numpy as np
import pytest

import fields as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["FP64", "FP32_BULK"])
@pytest.mark.parametrize("spin,n", [("HALF", 0), ("HALF", 1), ("ONE", 37), ("HALF", 8191), ("HALF", 8193), ("ONE", 4681),
                                    ("ONE", 4682)])
def test_host_and_device_arrays(cuda, spin, n, precision):
    import torch
    import spinsim_b200 as ss
    sq = ss.SpinQuantumNumber[spin]
    sim = ss.Simulator(F.rabi, sq, precision=ss.Precision[precision])
    args = (0.0, (n + 0.25) * 1e-7, 5e-8, 1e-7, sq.plus_z, [6e5, 2e4])
    first, second, third = (sim.evaluate(*args) for _ in range(3))
    d = second.device_arrays  # before any host read
    assert {k: tuple(v.shape) for k, v in d.items()} == {"time": (n,), "time_evolution": (n, sq.dimension, sq.dimension),
                                                        "state": (n, sq.dimension), "spin": (n, 3)}
    assert all(v.is_contiguous() and v.is_cuda for v in d.values())
    assert d["time"].dtype == d["spin"].dtype == torch.float64 and d["state"].dtype == torch.complex128
    names = ["spin", "state", "time_evolution", "time"]
    for k in names:
        a, b = getattr(first, k), d[k].cpu().numpy()
        assert a.dtype == b.dtype and a.shape == b.shape and a.flags.c_contiguous and a.flags.writeable
        assert np.array_equal(a, b) and np.array_equal(a, getattr(second, k))
        assert getattr(first, k) is a
    assert np.array_equal(third.time, first.time)  # host first, then the device
    assert np.array_equal(third.device_arrays["state"].cpu().numpy(), first.state)
    assert np.array_equal(first.time, np.arange(n) * 1e-7)
    assert (first.error_estimate == 0.0) if precision == "FP64" else (0.0 <= first.error_estimate < 1e-6)
