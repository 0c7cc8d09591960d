// Field sources for the time-evolution kernels.
//
//  FIELD_USER   the user's get_field(time_sample, sweep_parameters, field_sample) (the reference's
//               only extension point, spinsim/__init__.py:381-389, :620), compiled by numba to
//               LTO-IR behind a C-ABI shim and linked into the kernel with nvJitLink.
//  FIELD_TABLE  per-channel interpolation tables (the reference's generate_interpolation_sampler,
//               I:1941-2147): zero-order hold, linear or cubic Hermite, zero or held boundaries.
//  FIELD_TONES  per-channel bias + sum of sinusoids A sin(w t + phi).
#pragma once
#include "common.cuh"

#ifdef SPINSIM_USER_FIELD
// Provided by the numba-compiled shim: writes field_sample[0..8) (pre-zeroed by the caller).
extern "C" __device__ void spinsim_user_field(double time_sample, double* sweep_parameters, int64_t n_parameters,
                                              double* field_sample);
#endif

namespace spinsim {

// find_time_index (I:2026-2061): guess the index from equal spacing, bisect if the guess is wrong.
// Returns -1 outside the table (or after `size` bisection steps, as the reference does).
SS_D int64_t table_find(const TableChannel& tb, double ts, double* u) {
    const double* time = tb.time;
    const int64_t size = tb.size;
    *u = 0.0;
    const double first = __ldg(time), last = __ldg(time + size - 1);
    if (!(first <= ts && ts <= last)) return -1;
    int64_t idx = (int64_t)((ts - first) / (__ldg(time + 1) - first));
    bool low_enough = false, high_enough = true;
    if (idx + 1 < size) {
        low_enough = __ldg(time + idx) <= ts;
        high_enough = ts <= __ldg(time + idx + 1);
    } else {
        idx = size;
    }
    if (!(low_enough && high_enough)) {
        int64_t idx_max = size - 1, idx_min = 0, get_out = size;
        while (!(low_enough && high_enough)) {
            if (!low_enough) idx_max = idx;
            else idx_min = idx;
            idx = (idx_max + idx_min) >> 1;  // the reference's int((max + min) / 2), never negative
            low_enough = false;
            high_enough = true;
            if (idx + 1 < size) {
                low_enough = __ldg(time + idx) <= ts;
                high_enough = ts <= __ldg(time + idx + 1);
            }
            if (--get_out == 0) return -1;
        }
    }
    const double t_lo = __ldg(time + idx), t_hi = __ldg(time + idx + 1);
    *u = (ts - t_lo) / (t_hi - t_lo);
    return idx;
}

// Interpolation given the interval index i and parameter u (the sampler bodies of I:2065-2140).
SS_D double table_value(const TableChannel& tb, int64_t i, double u) {
    const double* time = tb.time;
    const double* amp = tb.amplitude;
    const int64_t size = tb.size;
    if (tb.order == 0) return i >= 0 ? __ldg(amp + i) : 0.0;
    if (!(i >= 0 && i + 1 < size)) return 0.0;
    const double a0 = __ldg(amp + i), a1 = __ldg(amp + i + 1);
    if (tb.order == 1) return a0 * (1 - u) + a1 * u;
    const double t0 = __ldg(time + i), t1 = __ldg(time + i + 1);
    const double g_mid = (t0 != t1) ? (a1 - a0) / (t1 - t0) : 0.0;
    double g_left;
    if (i == 0) {
        g_left = g_mid;
    } else {
        const double tm = __ldg(time + i - 1);
        g_left = (tm != t0) ? 0.5 * ((a0 - __ldg(amp + i - 1)) / (t0 - tm) + g_mid) : 0.0;
    }
    g_left *= (t1 - t0);
    double g_right;
    if (i + 2 == size) {
        g_right = g_mid;
    } else {
        const double tp = __ldg(time + i + 2);
        g_right = (t1 != tp) ? 0.5 * ((__ldg(amp + i + 2) - a1) / (tp - t1) + g_mid) : 0.0;
    }
    g_right *= (t1 - t0);
    const double u2 = u * u, u3 = u2 * u;
    return a0 * (2 * u3 - 3 * u2 + 1) + a1 * (-2 * u3 + 3 * u2) + g_left * (u3 - 2 * u2 + u) + g_right * (u3 - u2);
}

// The sampler of I:2065-2140 with the reference's search.
SS_D double table_sample(const TableChannel& tb, double ts) {
    if (!tb.zero_boundary) {
        if (ts <= __ldg(tb.time)) return __ldg(tb.amplitude);
        if (ts >= __ldg(tb.time + tb.size - 1)) return __ldg(tb.amplitude + tb.size - 1);
    }
    double u;
    const int64_t i = table_find(tb, ts, &u);
    return table_value(tb, i, u);
}

// A per-lane cursor over one table for sample times that only increase (the fine steps of an
// output interval).  The interval [time[i], time[i+1]] that holds a sample strictly inside it is
// unique, so advancing the cursor finds the same index as the reference's search; a sample that
// lands exactly on a table time (or outside the table) goes to the reference's search, which picks
// among the touching intervals as the reference does.  The cursor removes the bisection's chain of dependent loads.
//
// A cursor also keeps the channel (gain and bias included) on (t_lo, t_hi): its constant value (a zero-order
// hold, or a channel without a table, on the whole line), or the coefficients of its linear or cubic piece in
// x = (t - t_lo) * inv.  A sample strictly inside then takes no search, no memory read and no division, where
// the interpolation formula divides four times for a cubic value; the value agrees with the formula's to
// rounding.  A sample on a knot goes to the formula.  A call of 5003 x 37 Heun steps over two cubic channels
// takes 25.7 us, 32.7 with the formula at every sample.
struct TableCursor {
    int32_t i = -1;    // -1: not positioned
    int32_t kept = 0;  // 1: constant c0 on (t_lo, t_hi); 2: c0 + x (c1 + x (c2 + x c3))
    double t_lo = 0.0, t_hi = 0.0;
    double inv = 0.0, c0 = 0.0, c1 = 0.0, c2 = 0.0, c3 = 0.0;

    SS_D double at(double t) const {
        if (kept == 1) return c0;
        const double x = (t - t_lo) * inv;
        return fma(x, fma(x, fma(x, c3, c2), c1), c0);
    }

    // Move to the interval that holds t strictly inside; false where there is none.
    SS_D bool seek(const TableChannel& tb, double t) {
        if (!tb.zero_boundary && (t <= __ldg(tb.time) || t >= __ldg(tb.time + tb.size - 1))) return false;
        if (i >= 0) {
            while (t >= t_hi && i + 2 < tb.size) {
                i++;
                t_lo = t_hi;
                t_hi = __ldg(tb.time + i + 1);
                kept = 0;
            }
            if (t > t_lo && t < t_hi) return true;
        }
        double u;
        const int64_t k = table_find(tb, t, &u);
        if (!(k >= 0 && k + 1 < tb.size && k < INT32_MAX)) return false;
        i = (int32_t)k;
        t_lo = __ldg(tb.time + k);
        t_hi = __ldg(tb.time + k + 1);
        kept = 0;
        return t > t_lo && t < t_hi;
    }

    // The piece on (t_lo, t_hi): the sampler bodies of I:2065-2140 as a polynomial (table_value).
    SS_D void keep(const TableChannel& tb, double gain, double bias) {
        const double a0 = __ldg(tb.amplitude + i);
        c0 = fma(gain, a0, bias);
        if (tb.order == 0) {
            kept = 1;
            return;
        }
        kept = 2;
        const double a1 = __ldg(tb.amplitude + i + 1), step = t_hi - t_lo;
        inv = 1.0 / step;
        c2 = c3 = 0.0;
        c1 = gain * (a1 - a0);
        if (tb.order == 1) return;
        // the ends' slopes times the interval: the mean of the neighbouring differences
        double left = a1 - a0, right = a1 - a0;
        if (i > 0) {
            const double tm = __ldg(tb.time + i - 1);
            left = tm != t_lo ? 0.5 * ((a0 - __ldg(tb.amplitude + i - 1)) / (t_lo - tm) * step + (a1 - a0)) : 0.0;
        }
        if (i + 2 < tb.size) {
            const double tp = __ldg(tb.time + i + 2);
            right = t_hi != tp ? 0.5 * ((__ldg(tb.amplitude + i + 2) - a1) / (tp - t_hi) * step + (a1 - a0)) : 0.0;
        }
        c1 = gain * left;
        c2 = gain * (3.0 * (a1 - a0) - 2.0 * left - right);
        c3 = gain * (left + right - 2.0 * (a1 - a0));
    }
};

// The last index whose time lies before t (-1: none), by a search of a whole warp, 32 probes at a time: three
// rounds of loads for a table of 5000 times, where a lane's bisection takes thirteen.
SS_D int64_t warp_seek(const TableChannel& tb, double t) {
    const int lane = threadIdx.x & 31;
    int64_t lo = -1, hi = tb.size;  // time[lo] < t <= time[hi]
    while (hi - lo > 1) {
        const int64_t step = (hi - lo + 31) / 32;
        const int64_t p = lo + (lane + 1) * step;
        const int n = __popc(__ballot_sync(0xffffffffu, p < hi && __ldg(tb.time + p) < t));
        hi = min(hi, lo + (n + 1) * step);
        lo += n * step;
    }
    return lo;
}

// A channel of a piecewise constant field (a zero-order hold, or no table) for sample times that only
// increase: its value val (gain and bias included), for times before `clear`, its next knot less the sample
// times' slack.
struct HoldChannel {
    int32_t i;  // the value is that of (time[i], time[i + 1])
    double clear, val;

    SS_D void load(const FieldDesc& f, int c, double slack) {
        const TableChannel& tb = f.tables[c];
        double v = 0.0;
        if (i >= 0 && i + 1 < tb.size) v = __ldg(tb.amplitude + i);
        else if (!tb.zero_boundary) v = __ldg(tb.amplitude + (i < 0 ? 0 : tb.size - 1));
        val = fma(f.gain[c], v, f.bias[c]);
        clear = i + 1 < tb.size ? __ldg(tb.time + i + 1) - slack : INFINITY;
    }
    // The value at t (not before the last one's); `near` is set when a knot lies within the slack of t.
    SS_D double at(const FieldDesc& f, int c, double t, double slack, bool& near) {
        if (t >= clear) {
            const TableChannel& tb = f.tables[c];
            while (i + 1 < tb.size && t > __ldg(tb.time + i + 1) + slack) i++;
            load(f, c, slack);
            near |= t >= clear;
        }
        return val;
    }
};

// Position a warp's three channels before t_first, the warp's first sample time; false (for the whole warp)
// where the field is not piecewise constant in its first three channels, has a fourth (`used` of them count),
// or has many knots before t_end, the end of the warp's intervals, to walk.
constexpr int kHoldKnots = 32;

SS_D bool hold_channels(const FieldDesc& f, int used, double t_first, double t_end, double slack,
                        HoldChannel (&ch)[3]) {
    if (used > 3 && (f.tables[3].size > 0 || f.bias[3] != 0.0)) return false;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const TableChannel& tb = f.tables[c];
        ch[c].i = -1;
        ch[c].clear = INFINITY;
        ch[c].val = f.bias[c];
        if (tb.size <= 0) continue;
        if (tb.order != 0 || tb.size >= INT32_MAX) return false;
        if (c > 0 && f.tables[c - 1].time == tb.time && f.tables[c - 1].size == tb.size) {
            ch[c].i = ch[c - 1].i;
        } else {
            ch[c].i = (int32_t)warp_seek(tb, t_first);
            if ((int64_t)ch[c].i + kHoldKnots < tb.size && __ldg(tb.time + ch[c].i + kHoldKnots) < t_end) return false;
        }
        ch[c].load(f, c, slack);
    }
    return true;
}

// Sample the field at time t into out[0..NCH) (entries beyond NCH are left untouched).
// The caller pre-zeroes `out` like the reference does before each sample (I:625-642).  `cursors`
// (FIELD_TABLE, optional) hold one TableCursor per channel for increasing sample times.
template <int FIELD, int NCH>
SS_D void sample_field(const FieldDesc& f, double t, double* out, TableCursor* cursors = nullptr) {
    if constexpr (FIELD == FIELD_USER) {
#ifdef SPINSIM_USER_FIELD
        spinsim_user_field(t, const_cast<double*>(f.params), f.n_params, out);
#endif
    } else if constexpr (FIELD == FIELD_TABLE) {
#pragma unroll
        for (int c = 0; c < NCH; c++) {
            if (cursors && cursors[c].kept && t > cursors[c].t_lo && t < cursors[c].t_hi) {
                out[c] = cursors[c].at(t);
                continue;
            }
            const TableChannel& tb = f.tables[c];
            if (tb.size <= 0) {
                out[c] = f.bias[c];
                if (cursors) {
                    TableCursor& cu = cursors[c];
                    cu.i = 0;
                    cu.kept = 1;
                    cu.t_lo = -INFINITY;
                    cu.t_hi = INFINITY;
                    cu.c0 = out[c];
                }
            } else if (cursors && cursors[c].seek(tb, t)) {
                cursors[c].keep(tb, f.gain[c], f.bias[c]);
                out[c] = cursors[c].at(t);
            } else {
                out[c] = fma(f.gain[c], table_sample(tb, t), f.bias[c]);
            }
        }
    } else {  // FIELD_TONES
#pragma unroll
        for (int c = 0; c < NCH; c++) {
            double acc = f.bias[c];
            const double* tone = f.tones + 3 * f.tone_start[c];
            const int n = f.tone_count[c];
            const double gain = f.gain[c];
            for (int k = 0; k < n; k++) {
                const double w = __ldg(tone + 3 * k), a = gain * __ldg(tone + 3 * k + 1), ph = __ldg(tone + 3 * k + 2);
                acc = fma(a, sin(fma(w, t, ph)), acc);
            }
            out[c] = acc;
        }
    }
}

// The z channel alone (the rotating frame's sample at the middle of an output interval, I:823-829).
template <int FIELD, int NCH>
SS_D double sample_z(const FieldDesc& f, double t) {
    if constexpr (FIELD == FIELD_TABLE) {
        const TableChannel& tb = f.tables[2];
        return tb.size > 0 ? fma(f.gain[2], table_sample(tb, t), f.bias[2]) : f.bias[2];
    } else {
        double s[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        sample_field<FIELD, NCH>(f, t, s);
        return s[2];
    }
}

}  // namespace spinsim
