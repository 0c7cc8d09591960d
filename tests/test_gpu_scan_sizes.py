"""The state scan at the sizes where its launches change: one cluster launch for a short single instance (one to
four output steps per thread, one to eight CTAs), tile products and a cluster prefix for a long one, warp or
cluster prefixes in batches (from operators and from the tensor path's partials).  The states are compared with
the serial propagation (the oracle's) of the same operators.

Tolerance: both sides multiply up to n unitary operators in FP64; a product rounds by at most about 8 2^-53 per
operator, so linear accumulation gives 2^-50 n.
"""
import ctypes

import numpy as np
import pytest

import fields as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def unitaries(n, dim, seed):
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.normal(size=(n, dim, dim)) + 1j * rng.normal(size=(n, dim, dim)))
    psi0 = rng.normal(size=dim) + 1j * rng.normal(size=dim)
    return np.ascontiguousarray(q), psi0 / np.linalg.norm(psi0)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 2047, 2048, 2049, 4100, 6145, 8191, 8192, 8193, 8225,
                               33_001, 270_000])
@pytest.mark.parametrize("dim", [2, 3])
def test_single_instance(cuda, dim, n):
    import torch
    from spinsim_b200 import _lib
    lib = _lib.load()
    q, psi0 = unitaries(n, dim, seed=n + dim)
    u = torch.from_numpy(q).to(cuda)
    state = torch.full((n + 1, dim), np.nan, dtype=torch.complex128, device=cuda)
    spin = torch.full((n + 1, 3), np.nan, dtype=torch.float64, device=cuda)
    product = torch.empty((dim, dim), dtype=torch.complex128, device=cuda)
    size = lib.spinsim_state_workspace_size(dim, n)
    ws = torch.empty(size, dtype=torch.uint8, device=cuda)
    p0 = psi0.ctypes.data_as(ctypes.c_void_p)
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.spinsim_state(dim, u.data_ptr(), n, p0, state.data_ptr(), spin.data_ptr(), ws.data_ptr(), size, stream))
    ref = O.state(q, psi0)
    tol = 2.0 ** -50 * n + 1e-15
    assert np.abs(state[:n].cpu().numpy() - ref).max() < tol
    assert np.abs(spin[:n].cpu().numpy() - O.spin(ref)).max() < 4 * tol
    assert torch.isnan(state[n].real).all() and torch.isnan(spin[n]).all()
    _lib.check(lib.spinsim_piece_product(dim, u.data_ptr(), n, product.data_ptr(), ws.data_ptr(), size, stream))
    last = q[-1] @ ref[-1]
    assert np.abs(product.cpu().numpy() @ psi0 - last).max() < tol + 1e-14


@pytest.mark.parametrize("precision", ["FP64", "FP32_BULK"])
@pytest.mark.parametrize("spins,lengths", [("half", (9000, 1, 40)), ("one", (9000, 64)), ("mixed", (16_500, 9000, 3, 1500)),
                                           ("mixed", (40, 33, 1000))])
def test_batch_of_long_and_short_instances(cuda, spins, lengths, precision):
    import spinsim_b200 as ss
    import spinsim_b200.batch as B
    insts = []
    for j, n in enumerate(lengths):
        s = {"half": ss.SpinQuantumNumber.HALF, "one": ss.SpinQuantumNumber.ONE}.get(
            spins, ss.SpinQuantumNumber.HALF if j % 2 else ss.SpinQuantumNumber.ONE)
        p = F.tone_parameters(np.random.default_rng(j))
        tones = {a: p[4 + 24 * a:28 + 24 * a].reshape(8, 3) for a in range(3)}
        insts.append(B.Instance(s, 0.0, (n + 0.5) * 1e-7, 5e-8, 1e-7, s.plus_x, field=ss.ToneField(tones)))
    b = B.Batch(insts, precision=ss.Precision[precision])
    b.run()
    for k, i in enumerate(insts):
        r = b.result(k)
        ref = O.state(r.time_evolution, np.asarray(i.state_init, complex))
        assert r.state.shape == ref.shape == (lengths[k], i.spin.dimension)
        # FP32-bulk on the tensor path: the scan multiplies the steps' SU(2) pairs, which round apart from
        # their d x d images by one more rounding each
        assert np.abs(r.state - ref).max() < 2.0 ** -49 * lengths[k] + 1e-15, k


def test_sweep_parameters_by_value_and_by_reference(cuda):
    """Up to 64 sweep parameters travel with the launch, more through device memory: the same results."""
    import spinsim_b200 as ss
    sim = ss.Simulator(F.detuned_rabi, ss.SpinQuantumNumber.ONE)
    runs = [sim.evaluate(0.0, 50e-6, 10e-9, 1e-6, ss.SpinQuantumNumber.ONE.plus_z, [1500.0] + [0.0] * extra)
            for extra in (0, 63, 64, 200)]
    for r in runs[1:]:
        assert np.array_equal(r.time_evolution, runs[0].time_evolution) and np.array_equal(r.state, runs[0].state)
    assert np.abs(runs[0].state[-1] - runs[0].state[0]).max() > 1e-3
