"""User-field kernels come in a build of capped registers and an uncapped one: light fields take the capped build by
default, a field of many live values that spills there the uncapped one (as before the cap), and a budget above 168
always does.  Both give the same results."""
import numpy as np
import pytest

import fields as F

pytestmark = pytest.mark.gpu


def many_live_values(n):
    """A field from n x n values of time that are all live at once."""
    lines = ["def field(t, p, f):"]
    lines += [f"    m{i}_{j} = p[{(i * n + j) % 24}] + p[{(i + j * n) % 24}] * t" for i in range(n) for j in range(n)]
    lines += [f"    x{i} = p[{i}]" for i in range(n)] + ["    for k in range(8):"]
    lines += [f"        y{i} = " + " + ".join(f"m{i}_{j} * x{j}" for j in range(n)) for i in range(n)]
    lines += [f"        x{i} = 0.1 * y{i}" for i in range(n)]
    lines += ["    f[0] = 1e4 * x0", "    f[1] = 1e4 * x1", "    f[2] = 1e5 + 1e3 * x2", "    f[3] = 0.0"]
    out = {}
    exec("\n".join(lines), out)
    return out["field"]


@pytest.mark.parametrize("spin,field,capped", [("HALF", F.rabi, True), ("HALF", many_live_values(9), False),
                                               ("ONE", F.rabi_one, True)])
def test_builds(cuda, spin, field, capped):
    import spinsim_b200 as ss
    from spinsim_b200.batch import Batch, Instance
    sq = ss.SpinQuantumNumber[spin]
    p = np.random.default_rng(0).uniform(0.2, 1.0, 24)
    if field in (F.rabi, F.rabi_one):
        p[:2] = 5e6, 2e5
    insts = [Instance(sq, 0.0, 20.5e-6, 2e-8, 1e-6, sq.plus_z, sweep_parameters=p * (1.0 + 1e-3 * i)) for i in range(3)]
    default, wide, tight = (Batch(insts, get_field=field, max_registers=m) for m in (0, 255, 128))
    cap = 96 if spin == "HALF" else 128
    assert tight.launch_info()["registers_per_thread"] <= cap
    assert (default.launch_info()["registers_per_thread"] <= cap) == capped
    if not capped:
        assert wide.launch_info()["registers_per_thread"] > cap
    for b in (default, wide, tight):
        b.run()
    for k in range(3):
        for b in (default, wide):
            assert np.abs(b.result(k).time_evolution - tight.result(k).time_evolution).max() < 1e-13
