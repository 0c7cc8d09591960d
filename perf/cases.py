"""The work that spinsim_b200 is measured on: calls of its public entry points, from one small evaluate() to the
uneven batches of the benchmark, with the sizes, fields, spins, integrators and precisions of the examples, the
tests and the benchmark.

A case says which entry point is called (``Simulator.evaluate``, a prepared ``Batch`` launched again with other
work between, or ``evaluate_many`` into host memory), the spin (half, one, or 70% / 30% mixed), the field, how many
instances, how many output steps each, how many fine steps an output step takes and of what length, and the
numerical options.  ``prepare`` makes what a user's program has in hand (a Simulator and the call's arguments, a
Batch, or the list of instances); ``run`` makes the one call.
"""
import math

import numpy as np
import torch

import spinsim_b200 as ss
from spinsim_b200.batch import Batch, Evaluator, Instance

TAU = 2.0 * math.pi
SQRT3 = math.sqrt(3.0)


# ------------------------------------------------------------------------------------------ the cases
def _case(name, entry, spin, field, count, n_out, k, dt_ns, **more):
    """n_out output steps (with n_min: log-uniform from n_min to n_out over the instances) of k fine steps of dt_ns."""
    c = {"entry": entry, "spin": spin, "field": field, "count": count, "n_min": n_out, "n_out": n_out, "k": k,
         "dt_ns": dt_ns, "precision": "fp64", "integration": "magnus_cf4", "lie_trotter": spin != "half",
         "squares": 24, "rotating": True, "larmor_hz": 300e3, "q_hz": 0.0, "tones": 8, "to_host": False}
    c.update(more)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # One Gaussian pulse in a hundred steps, results read as numpy arrays: what a script that scans a parameter
        # does at each value, bound by the latency of the call.
        _case("simulator pulse small", "simulator", "half", "gaussian", 1, 100, 4, 50.0, to_host=True),
        # Precession over 100 ms at 100 ns / 500 ns: few fine steps and many output steps, so the state propagation
        # counts as much as the integration.
        _case("simulator precession long", "simulator", "half", "drive", 1, 200_000, 5, 100.0, larmor_hz=1e3),
        # One detuning of the spin-one Rabi drive, 10 ms at 10 ns / 100 ns with 28 squarings.
        _case("simulator rabi spin one", "simulator", "one", "drive", 1, 100_000, 10, 10.0, larmor_hz=840e3,
              squares=28),
        # Spin one with the quadratic shift that a real spin-one sample has, an odd number of output steps.
        _case("simulator quadratic shift", "simulator", "one", "drive", 1, 4_001, 50, 20.0, q_hz=64.0),
        # A measured waveform on two axes, cubic interpolation, Heun and the Lie-Trotter exponential, lab frame.
        _case("simulator waveform heun", "simulator", "half", "waveform", 1, 5_003, 37, 20.0, integration="heun",
              lie_trotter=True, rotating=False),
        # A sweep of 64 detunings of the spin-one drive as one batch.
        _case("batch rabi sweep", "batch", "one", "drive", 64, 10_000, 10, 10.0, larmor_hz=840e3, squares=28),
        # The ensemble of 4096 atoms under a Gaussian pulse (1 ms at 20 ns / 1 us), in both precisions.
        _case("batch ensemble", "batch", "half", "gaussian", 4096, 1_000, 50, 20.0),
        _case("batch ensemble fp32-bulk", "batch", "half", "gaussian", 4096, 1_000, 50, 20.0, precision="fp32_bulk"),
        # The benchmark's uneven batch of eight-tone fields (10 us to 10 ms at 10 ns / 1 us, both spins), FP32-bulk,
        # and a quarter of it in FP64.
        _case("batch tones fp32-bulk", "batch", "mixed", "tones", 1024, 10_000, 100, 10.0, n_min=10,
              precision="fp32_bulk"),
        _case("batch tones", "batch", "mixed", "tones", 256, 10_000, 100, 10.0, n_min=10),
        # One launch of the server: pulse-train requests of both spins, 10 us to 100 ms, FP32-bulk.
        _case("batch pulse trains", "batch", "mixed", "pulses", 400, 100_000, 20, 50.0, n_min=10,
              precision="fp32_bulk"),
        # A dozen long instances evaluated into host memory, set-up and copies included.
        _case("evaluate_many tones", "evaluate_many", "mixed", "tones", 12, 10_000, 100, 10.0, n_min=2_500,
              precision="fp32_bulk"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges; no draw costs more than the largest listed case."""
    kind = rng.choice(["simulator", "simulator", "simulator", "batch", "batch", "batch", "evaluate_many"])
    field = rng.choice({"simulator": ["gaussian", "drive", "waveform", "tones"],
                        "batch": ["gaussian", "drive", "tones", "tones", "pulses"],
                        "evaluate_many": ["tones"]}[kind])
    precision = rng.choice(["fp64", "fp32_bulk"])
    mixed = kind != "simulator" and field in ("tones", "pulses")
    spin = "mixed" if mixed else rng.choice(["half", "half", "one"])
    dt_ns = rng.choice([10.0, 20.0, 50.0]) if field != "pulses" else rng.choice([20.0, 50.0, 100.0])
    k = _log_int(rng, 4, 200)
    more = {"precision": precision}
    if spin == "half":
        more["lie_trotter"] = rng.random() < 0.25
    if field == "drive":
        more["larmor_hz"] = rng.choice([1e3, 300e3, 840e3]) if dt_ns <= 20.0 else rng.choice([1e3, 100e3, 300e3])
    if spin == "one" and field == "drive":
        more["q_hz"] = rng.choice([0.0, 0.0, 64.0, 500.0])
    if field == "tones":
        more["tones"] = rng.randint(1, 8)
    if not mixed:
        more["squares"] = rng.choice([24, 24, 28])
        more["rotating"] = rng.random() < 0.75
    if kind == "simulator":
        more["integration"] = rng.choice(["magnus_cf4", "magnus_cf4", "magnus_cf4", "heun", "euler"])
        n_out = _log_int(rng, 30, 200_000)
        n_out = min(n_out, 20_000_000 // k)
        return _case(None, kind, spin, field, 1, n_out, k, dt_ns, to_host=n_out <= 1000, **more)
    # total fine steps of a batch: up to 4e7 (1.2e8 for FP32-bulk tones, the benchmark's own)
    total = _log_int(rng, 2e5, 4e7)
    count = _log_int(rng, 2, 2000) if kind == "batch" else rng.randint(2, 15)
    n_out = max(8, min(100_000, total // (count * k)))
    n_min = max(1, n_out // rng.choice([1, 1, 30, 1000])) if field in ("tones", "pulses") else n_out
    return _case(None, kind, spin, field, count, n_out, k, dt_ns, n_min=n_min, **more)


# ------------------------------------------------------------------------------------------ the fields
def gaussian_pulse(time_sample, sweep_parameters, field_sample):
    """A Gaussian pulse on x over a detuning on z; parameters: detuning, peak, width, centre."""
    x = (time_sample - sweep_parameters[3]) / sweep_parameters[2]
    field_sample[0] = sweep_parameters[1] * math.exp(-0.5 * x * x)
    field_sample[1] = 0.0
    field_sample[2] = sweep_parameters[0]


def drive(time_sample, sweep_parameters, field_sample):
    """A linearly polarised drive; parameters: Larmor, Rabi, drive (rad/s) and, for spin one, the quadratic shift."""
    field_sample[0] = 2.0 * sweep_parameters[1] * math.cos(sweep_parameters[2] * time_sample)
    field_sample[1] = 0.0
    field_sample[2] = sweep_parameters[0]
    field_sample[3] = sweep_parameters[3]


def _parameters(case, rng, spin):
    """The sweep parameters of one instance whose field is a get_field function."""
    if case["field"] == "gaussian":
        span = case["n_out"] * case["k"] * case["dt_ns"] * 1e-9
        width = max(2e-6, 0.05 * span) if case["entry"] == "simulator" else 2e-6
        peak = TAU * 50e3 * rng.uniform(0.9, 1.1) * 2e-6 / width
        return np.array([TAU * rng.normal(0.0, 500.0), peak, width, min(10e-6, 0.5 * span) if width == 2e-6 else 0.5 * span])
    f = case["larmor_hz"] * rng.uniform(0.95, 1.05)
    rabi, detuning = min(2e3, 0.2 * f) * rng.uniform(0.9, 1.1), min(5e3, 0.05 * f) * rng.uniform(-1.0, 1.0)
    return TAU * np.array([f, rabi, f + detuning, case["q_hz"] if spin.dimension == 3 else 0.0])


def _tones(case, rng):
    n = case["tones"]
    tones = {c: np.stack([TAU * rng.uniform(0.0, 1e6, n), rng.uniform(0.0, TAU * 10e3, n), rng.uniform(0.0, TAU, n)], 1)
             for c in range(3)}
    return ss.ToneField(tones, bias=[0.0, 0.0, TAU * rng.uniform(0.0, 50e3)])


def _waveform(case, rng, span):
    """A sampled waveform: two axes of a few harmonics over the call's span, 2001 samples, and a bias on z."""
    t = np.linspace(0.0, span * 1.01, 2001)
    tables = {}
    for c in (0, 1):
        a = np.zeros_like(t)
        for h in range(1, 6):
            a += rng.normal(0.0, TAU * 8e3) * np.sin(math.pi * h * t / span + rng.uniform(0.0, TAU))
        tables[c] = (t, a)
    return ss.TabulatedField(tables, order=3, bias=[0.0, 0.0, TAU * rng.uniform(20e3, 60e3)])


def _pulses(rng, t_end):
    """A train of pi/2 and pi pulses (10 and 20 us at 25 kHz) on x or y with gaps of 1 to 50 us, zero-order hold."""
    m = int(t_end / 35e-6 * 2) + 8
    while True:
        gaps, widths = rng.uniform(1e-6, 50e-6, m), rng.choice([10e-6, 20e-6], m)
        ends = np.cumsum(gaps + widths)
        if ends[-1] >= t_end:
            break
        m *= 2
    m = int(np.searchsorted(ends, t_end)) + 1
    ends, widths, on_y = ends[:m], widths[:m], rng.random(m) < 0.5
    t = np.concatenate([[0.0], np.stack([ends - widths, ends], 1).reshape(-1)])
    x, y = np.zeros(2 * m + 1), np.zeros(2 * m + 1)
    x[1::2] = np.where(on_y, 0.0, TAU * 25e3)
    y[1::2] = np.where(on_y, TAU * 25e3, 0.0)
    return ss.TabulatedField({0: (t, x), 1: (t, y)}, order=0, zero_boundary=False)


# ------------------------------------------------------------------------------------------ prepare and run
HALF, ONE = ss.SpinQuantumNumber.HALF, ss.SpinQuantumNumber.ONE


def _instances(case, seed):
    """The instances of a case, on the host; a Simulator call is an instance of its own."""
    rng = np.random.default_rng([seed, 17])
    shape = np.random.default_rng(23)  # sizes and spins do not change with the seed
    dt = case["dt_ns"] * 1e-9
    dt_out = case["k"] * dt
    out = []
    for i in range(case["count"]):
        spin = {"half": HALF, "one": ONE}.get(case["spin"]) or (HALF if shape.uniform() < 0.7 else ONE)
        n = int(round(math.exp(shape.uniform(math.log(case["n_min"]), math.log(case["n_out"])))))
        psi0 = spin.plus_x if spin is ONE else spin.plus_z
        end = (n + 0.25) * dt_out
        field, params = None, (0.0,)
        if case["field"] == "tones":
            field = _tones(case, rng)
        elif case["field"] == "pulses":
            field = _pulses(rng, end)
        elif case["field"] == "waveform":
            field = _waveform(case, rng, end)
        else:
            params = _parameters(case, rng, spin)
        out.append(Instance(spin, 0.0, end, dt, dt_out, psi0, sweep_parameters=params, field=field))
    return out


def _get_field(case):
    return {"gaussian": gaussian_pulse, "drive": drive}.get(case["field"])


def prepare(case, seed):
    insts = _instances(case, seed)
    precision = ss.Precision.FP64 if case["precision"] == "fp64" else ss.Precision.FP32_BULK
    integration = ss.IntegrationMethod(case["integration"])
    expo = ss.ExponentiationMethod.LIE_TROTTER if case["lie_trotter"] else ss.ExponentiationMethod.ANALYTIC
    state = {"entry": case["entry"], "to_host": case["to_host"]}
    if case["entry"] == "simulator":
        i = insts[0]
        state["sim"] = ss.Simulator(_get_field(case) or i.field, i.spin, integration_method=integration,
                                    exponentiation_method=expo, use_rotating_frame=case["rotating"],
                                    number_of_squares=case["squares"], precision=precision)
        state["args"] = (i.time_start, i.time_end, i.time_step_integration, i.time_step_output, i.state_init,
                         i.sweep_parameters)
        return state
    options = dict(integration_method=integration, use_rotating_frame=case["rotating"],
                   number_of_squares=case["squares"], precision=precision)
    if case["spin"] == "half" and case["lie_trotter"]:
        options["exponentiation_half"] = ss.ExponentiationMethod.LIE_TROTTER
    if case["entry"] == "batch":
        state["batch"] = Batch(insts, get_field=_get_field(case), **options)
    else:
        state["instances"] = insts
        state["evaluator"] = Evaluator(**options)
    return state


def run(state):
    if state["entry"] == "simulator":
        r = state["sim"].evaluate(*state["args"])
        if state["to_host"]:  # a script that plots: numpy arrays
            return {"time": r.time, "u": r.time_evolution, "state": r.state, "spin": r.spin}
        d = r.device_arrays
        return {"time": d["time"], "u": d["time_evolution"], "state": d["state"], "spin": d["spin"]}
    if state["entry"] == "batch":
        b = state["batch"]
        b.run()
        return {"time": b.time, "u": b.u, "state": b.state, "spin": b.spin}
    got = state["evaluator"].evaluate(state["instances"])
    return [[r.time, r.time_evolution, r.state, r.spin] for r in got]


# ------------------------------------------------------------------------------------------ work
def work(case):
    """Descriptors, parameters and tables in; time, operator, state and spin of every output step out.  Per fine step: the
    field's samples (each tone two multiply-adds; a pulse or a drive about ten operations; a table value two, of
    cubic pieces twelve), and for each of the step's exponentials the frame's rotation, the generator, the exponential and
    its product into the step's operator as an SU(2) element (about 60; spin one with a quadratic shift: 3 x 3, about 330)."""
    insts = _shape(case)
    samples = 1 if case["integration"] == "euler" else 2
    field = {"gaussian": 10, "drive": 10, "tones": 3 * 4 * case["tones"], "pulses": 2, "waveform": 24}[case["field"]]
    bytes_, flops = 0.0, 0.0
    for dim, n in insts:
        bytes_ += 200 + n * (8 + 16 * dim * dim + 16 * dim + 24)
        if case["field"] == "tones":
            bytes_ += 72 * case["tones"]
        elif case["field"] == "pulses":
            bytes_ += 24 * 2 * n * case["k"] * case["dt_ns"] * 1e-9 / 40e-6
        elif case["field"] == "waveform":
            bytes_ += 3 * 8 * 2001
        flops += n * case["k"] * samples * (field + (330 if dim == 3 and case["q_hz"] else 60))
    return {"bytes": bytes_, "flops": flops}


def _shape(case):
    """(spin dimension, output steps) of every instance, as _instances draws them."""
    shape = np.random.default_rng(23)
    out = []
    for i in range(case["count"]):
        dim = {"half": 2, "one": 3}.get(case["spin"]) or (2 if shape.uniform() < 0.7 else 3)
        out.append((dim, int(round(math.exp(shape.uniform(math.log(case["n_min"]), math.log(case["n_out"])))))))
    return out


# ------------------------------------------------------------------------------------------ exact
# The same integrators in plain float64 torch on whole arrays of output steps.  The Lie-Trotter exponential with 24
# or more squarings of a step of these sizes is the exponential itself to rounding, and is taken as that.
def _sample(case, insts, which, t):
    """(x, y, z, q) at times t, of instance number which[i] for entry i."""
    dev = t.device
    zero = torch.zeros_like(t)

    def column(v):
        return torch.tensor(np.array(v, np.float64), device=dev)[which]

    if case["field"] in ("gaussian", "drive"):
        p = np.stack([i.sweep_parameters for i in insts])
        if case["field"] == "gaussian":
            x = (t - column(p[:, 3])) / column(p[:, 2])
            return column(p[:, 1]) * torch.exp(-0.5 * x * x), zero, column(p[:, 0]), zero
        return 2.0 * column(p[:, 1]) * torch.cos(column(p[:, 2]) * t), zero, column(p[:, 0]), column(p[:, 3])
    fields = [i.field for i in insts]
    out = [column([f.bias[c] for f in fields]) for c in range(4)]
    if case["field"] == "tones":
        for c in range(3):
            for n in range(case["tones"]):
                w, a, ph = (column([f.tones[c][n, e] for f in fields]) for e in range(3))
                out[c] = out[c] + a * torch.sin(w * t + ph)
        return out
    for c in (0, 1):
        if case["field"] == "pulses":  # zero-order hold, each entry in its own instance's table
            times, values = [f.tables[c][0] for f in fields], [f.tables[c][1] for f in fields]
            ends = torch.tensor(np.cumsum([0] + [x.size for x in times]), device=dev)
            lo, hi = ends[:-1][which], ends[1:][which] - 1
            all_t = torch.tensor(np.concatenate(times), device=dev)
            all_v = torch.tensor(np.concatenate(values), device=dev)
            a, b = lo.clone(), hi.clone()
            for _ in range(20):  # bisection
                m = (a + b + 1) // 2
                below = all_t[m] <= t
                a, b = torch.where(below, m, a), torch.where(below, b, torch.maximum(m - 1, lo))
            out[c] = out[c] + all_v[a]
        else:
            tt, vv = (torch.tensor(x, device=dev) for x in fields[0].tables[c][:2])
            i = (torch.searchsorted(tt, t, right=True) - 1).clamp(0, tt.numel() - 2)
            t0, t1, a0, a1 = tt[i], tt[i + 1], vv[i], vv[i + 1]
            mid = (a1 - a0) / (t1 - t0)
            im, ip = (i - 1).clamp(min=0), (i + 2).clamp(max=tt.numel() - 1)
            left = torch.where(i > 0, 0.5 * ((a0 - vv[im]) / torch.where(i > 0, t0 - tt[im], 1.0) + mid), mid)
            last = i + 2 == tt.numel()
            right = torch.where(last, mid, 0.5 * ((vv[ip] - a1) / torch.where(last, 1.0, tt[ip] - t1) + mid))
            left, right, u = left * (t1 - t0), right * (t1 - t0), (t - t0) / (t1 - t0)
            out[c] = out[c] + (a0 * (2 * u ** 3 - 3 * u ** 2 + 1) + a1 * (3 * u ** 2 - 2 * u ** 3)
                               + left * (u ** 3 - 2 * u ** 2 + u) + right * (u ** 3 - u ** 2))
    return out


def _su2_step(p, x, y, z):
    """exp(-i (x, y, z).sigma / 2) times the SU(2) element p = (alpha - 1, beta), in place of p."""
    r = torch.sqrt(x * x + y * y + z * z)
    s = 0.5 * torch.sinc(r / TAU)  # sin(r / 2) / r
    a = torch.complex(-2.0 * torch.sin(0.25 * r) ** 2, -z * s)
    b = torch.complex(y * s, -x * s)
    am1, beta = p
    alpha = am1 + 1.0
    return am1 + a * alpha - b.conj() * beta, beta + b * alpha + a.conj() * beta


def _spin_one_step(u, x, y, z, q):
    h = torch.zeros(x.shape + (3, 3), dtype=torch.complex128, device=x.device)
    h[..., 0, 0], h[..., 1, 1], h[..., 2, 2] = (v + 0j for v in (z + q / 3, -2 * q / 3, -z + q / 3))
    h[..., 1, 0] = torch.complex(x, y) / math.sqrt(2.0)
    h[..., 2, 1] = h[..., 1, 0]
    h[..., 0, 1] = h[..., 1, 0].conj()
    h[..., 1, 2] = h[..., 0, 1]
    h = -1j * h
    one = torch.eye(3, dtype=torch.complex128, device=x.device)
    e = one
    for n in range(16, 0, -1):  # Horner's form of the series, |h| well below 1
        e = one + (h @ e) / n
    return e @ u


def _operators(case, insts, dim, which, index):
    """The operators of output steps `index` of instances `which` (all of one dimension)."""
    dt = insts[0].time_step_output / case["k"]
    dt_out = insts[0].time_step_output
    t_c = dt_out * index.double()
    quadratic = dim == 3 and case["q_hz"] != 0.0
    rw = torch.zeros_like(t_c)
    if case["rotating"]:
        rw = _sample(case, insts, which, t_c + dt_out / 2)[2]
    lo, hi = 0.5 * dt * (1 - 1 / SQRT3), 0.5 * dt * (1 + 1 / SQRT3)
    w0, w1 = (1.5 + SQRT3) / 6, (1.5 - SQRT3) / 6
    points, weights = {"magnus_cf4": ((lo, hi), ((w0, w1), (w1, w0))), "heun": ((0.0, dt), ((0.5, 0.0), (0.0, 0.5))),
                       "euler": ((0.5 * dt,), ((1.0,),))}[case["integration"]]
    if quadratic:
        u = torch.eye(3, dtype=torch.complex128, device=t_c.device).repeat(t_c.numel(), 1, 1)
    else:
        u = (torch.zeros(t_c.shape, dtype=torch.complex128, device=t_c.device),) * 2
    for j in range(case["k"]):
        samples = []
        for off in points:
            tau = j * dt + off
            x, y, z, q = _sample(case, insts, which, t_c + tau)
            xy = torch.complex(x, y) * torch.exp(-1j * (rw * tau))
            samples.append((xy.real, xy.imag, z - rw, q))
        for w in weights:
            g = [dt * sum(a * s[c] for a, s in zip(w, samples)) for c in range(4)]
            u = _spin_one_step(u, *g) if quadratic else _su2_step(u, *g[:3])
    out = torch.exp(-0.5j * rw * dt_out)  # leaving the frame, of spin half
    if quadratic:
        u[:, 0] *= (out * out)[:, None]
        u[:, 2] *= (out * out).conj()[:, None]
        return u
    a, b = (u[0] + 1.0) * out, u[1] * out.conj()
    if dim == 2:
        return torch.stack([a, -b.conj(), b, a.conj()], -1).view(-1, 2, 2)
    r2 = math.sqrt(2.0)
    ac, bc = a.conj(), b.conj()
    mid = (a * ac - b * bc).real + 0j
    return torch.stack([a * a, -r2 * a * bc, bc * bc, r2 * a * b, mid, -r2 * ac * bc, b * b, r2 * ac * b, ac * ac], -1).view(-1, 3, 3)


def _states(u, index, psi0):
    """state[i] = U[i-1] ... U[0] psi0 for instances back to back; index[i]: the output step of entry i in its instance."""
    d = u.shape[-1]
    p = torch.cat([torch.eye(d, dtype=u.dtype, device=u.device)[None], u[:-1]])
    p[index == 0] = torch.eye(d, dtype=u.dtype, device=u.device)
    s, longest = 1, int(index.max()) + 1
    while s < longest:
        at = torch.nonzero(index >= s).view(-1)
        new = [torch.bmm(p[c], p[c - s]) for c in at.split(1 << 20)]
        p[at] = torch.cat(new)
        s *= 2
    return (p @ psi0[:, :, None])[:, :, 0]


def _spins(st):
    if st.shape[1] == 2:
        p = st[:, 0] * st[:, 1].conj()
        return torch.stack([p.real, -p.imag, 0.5 * (st[:, 0].abs() ** 2 - st[:, 1].abs() ** 2)], 1)
    a = st[:, 1].conj() * (st[:, 0] + st[:, 2])
    b = st[:, 1].conj() * (st[:, 0] - st[:, 2])
    return torch.stack([math.sqrt(2.0) * a.real, -math.sqrt(2.0) * b.imag, st[:, 0].abs() ** 2 - st[:, 2].abs() ** 2], 1)


def exact(case, seed):
    insts = _instances(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    sizes = [n for _, n in _shape(case)]
    results = [None] * len(insts)
    for dim in (2, 3):
        ids = [k for k, i in enumerate(insts) if i.spin.dimension == dim]
        if not ids:
            continue
        mine = [insts[k] for k in ids]
        n = torch.tensor([sizes[k] for k in ids], device=dev)
        which = torch.repeat_interleave(torch.arange(len(ids), device=dev), n)
        start = torch.cumsum(n, 0) - n
        index = torch.arange(which.numel(), device=dev) - start[which]
        u = torch.cat([_operators(case, mine, dim, w, i) for w, i in zip(which.split(1 << 21), index.split(1 << 21))])
        psi0 = torch.tensor(np.stack([np.asarray(i.state_init, complex) for i in mine]), device=dev)[which]
        st = _states(u, index, psi0)
        parts = (mine[0].time_step_output * index.double(), u, st, _spins(st))
        for k, *r in zip(ids, *(v.split(n.tolist()) for v in parts)):
            results[k] = r
    if case["entry"] == "evaluate_many":
        return [[v.cpu().numpy() for v in r] for r in results]
    if case["entry"] == "batch":  # flat, instance after instance
        return {"time": torch.cat([r[0] for r in results]), "u": torch.cat([r[1].reshape(-1) for r in results]),
                "state": torch.cat([r[2].reshape(-1) for r in results]), "spin": torch.cat([r[3] for r in results])}
    out = dict(zip(("time", "u", "state", "spin"), results[0]))
    return {k: v.cpu().numpy() for k, v in out.items()} if case["to_host"] else out
