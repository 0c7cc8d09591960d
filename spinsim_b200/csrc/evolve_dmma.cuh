// Time evolution of tone fields (Magnus CF4) with the field samples formed on the FP64 tensor path, in FP32-bulk
// and in FP64.
//
// The reference samples its field once per Gauss point of every fine step of every output interval
// (get_field_integration_magnus_cf4, spinsim/__init__.py:624-652).  For a tone field, at distances +-delta from
// the middle t_m of an interval,
//     B_c(t_m +- delta) = bias_c + sum_k Im(L_ck) cos(w_k delta) +- sum_k Re(L_ck) sin(w_k delta),
//     L_ck = A_k exp(i (w_k t_m + phi_k)),
// and the Gauss points of the steps lie symmetrically about the middle, so the even and the odd sum at one
// distance give two samples.  The sums of a block of output intervals (rows, through L) at a block of
// distances (columns, through cos and sin) are matrix products with inner dimension (tones per channel) each.
// They run as mma.sync.m8n8k4.f64 (FP64 in, FP64 accumulate: the samples are exact to FP64 rounding), which
// takes eight multiply-adds per lane per instruction.  (Sampling each time by itself takes twice the
// products: inner dimension 2 x tones for one sample.)
//
// Mapping.  A CTA takes a tile of kDmmaTile consecutive output intervals of one instance; warp w
// takes intervals 8 w .. 8 w + 7 (the eight rows of the m8n8k4 product).  The K / 2 steps after the middle
// are split into kDmmaSegments consecutive segments, one per lane of a quad: in the accumulator layout lane
// 4 g + q holds row g, columns 2 q and 2 q + 1, which are made to be the distances of the two Gauss points
// of one step of segment q.  So every lane receives the samples of its own step and of that step's mirror
// image before the middle; it multiplies the first to its product of later steps from the left and the second
// to its product of earlier steps from the right, two independent chains.  The quad's products are combined
// once per interval with shuffles.  For odd K the middle step, its own mirror image, takes one column of one
// more product.
//
// Operands.  A (8 x 4 per k-step): lane 4 g + q holds Im L (even sums) or Re L (odd sums) of interval g for tone
// 4 s + q, computed once per tile with FP64 sincos.  B (4 x 8): lane 4 g + q needs cos or sin (w delta) of that
// tone at column g.  These depend on the instance only, not on the interval, so the CTA builds them in shared
// memory: 192 phasor recurrences exp(i w delta) (channel, tone, column) advanced by exp(i w dt) per pair of steps
// in FP64, written in lane order so that every B load and store is conflict-free.  The table is double-buffered
// in phases of kDmmaPhase pairs (one CTA barrier per phase).  The even sums start at the channel bias.
//
// Step, FP32-bulk.  The reference's Magnus CF4 (I:655-686) composes two exponentials per step; its order-four
// Magnus expansion at the same Gauss points, exp(g), g = (h/2)(b1 + b2) + (sqrt3 h^2 / 12) b2 x b1
// (the commutator [A2, A1] of A = -i b.J is -i (b2 x b1).J; Blanes, Casas and Ros, BIT 40 (2000)),
// is the same map to O(h^5): one SU(2) exponential per step.  A tile takes it when the step is small
// against the field, theta = h (|B|max + w_max) <= kMagnusTheta, and CF4 otherwise.  The frame
// transform, the sum and difference of the samples and the exponential's linear part stay in FP64;
// the commutator and the exponential's O(|g|^2) remainder are FP32, the interval product FP64
// (su2_split).  On the benchmark's longest instances (theta = 0.07) the two compositions agree
// to 1e-11 in the final state.  Instances with more than kBulkTones
// tones on a channel, or spin one with a quadratic shift, take the per-interval path (interval32,
// CF4) inside the same kernel.
//
// Step, FP64.  CF4 with the two FP64 exponentials of evolve64.cuh.  Instances the products do not take, and those
// whose tones' phases are large (tones_on_fp64_tensor_path), run in that file's kernel instead (the host splits the
// batch's tiles).
//
// Scan partials.  A CTA tile is one state scan tile (scan.cuh).  Each interval's lab-frame operator is
// an SU(2) pair (spin one: its representation), so each warp also multiplies its eight rows' pairs
// with three shuffle rounds and writes the product (4 doubles); the scan's prefix kernel combines a
// tile's four warp products and the scan launches no tile products pass over U.
#pragma once
#include "common.cuh"
#include "evolve32.cuh"

namespace spinsim {

constexpr int kDmmaSegments = 4;                             // lanes (time segments) per interval
#ifndef SPINSIM_DMMA_PHASE
#define SPINSIM_DMMA_PHASE 5
#endif
// Steps per segment in one table buffer: 5 divides the 25-step segments of K = 100 (1 us output
// steps of 10 ns), so no phase is a short remainder; 4 was 1% slower there.
constexpr int kDmmaPhase = SPINSIM_DMMA_PHASE;
// FP64: the phasor recurrences restart from sincos every 60 pairs, as the step loop of evolve64.cuh does every 64
// steps: their drift, about a rounding a pair, would grow with K (4e-13 at K = 1e5).
constexpr int kDmmaRestart = 12;  // phases
// Largest step size bound theta = h (|B|max + w_max) for which a tile takes the Magnus step.  The
// Magnus and CF4 steps differ by O(theta^5) per step: measured 4.6e-6 at theta = 6.7 (one 1 us step)
// and 1e-11 over 10^6 steps at theta = 0.07, i.e. about 3e-10 theta^5 per step, so at theta <= 0.1
// below 4e-15 per step, 4e-9 over 10^6 steps.
constexpr double kMagnusTheta = 0.1;
constexpr int kDmmaChunkDoubles = 3 * 4 * 32;  // B operands of one pair: [channel][even, odd][k-step][lane]
static_assert(kDmmaRecurrences == 3 * kBulkTones * kDmmaSegments * 2, "(channel, tone, segment, Gauss point)");
static_assert(kBulkTones == 8 && kDmmaSegments == 4, "two k-steps of four tones, eight columns");
// CF4 generators from samples in units of h / 2: h (w0 b1 + w1 b2) = 2 w0 sa + 2 w1 sb
constexpr double kDmmaW0 = (1.5 + kSqrt3) / 3.0, kDmmaW1 = (1.5 - kSqrt3) / 3.0;

// First pair of segment seg: pair i is the i-th step after the middle of the K and its mirror image.
SS_D int dmma_segment(int K, int seg) { return (int)(((int64_t)(K / 2) * seg) / kDmmaSegments); }

// How the reference's steps of an interval, at the running sum t_c + dt + dt ... (I:836), lie against t_c + j dt: on
// average `shift` later, and spaced (1 + stretch) dt about their middle.
struct StepTimes {
    double shift, stretch;
};

struct __align__(16) DmmaShared {
    double table[2][kDmmaPhase][kDmmaChunkDoubles];
    double2 z[kDmmaRecurrences];   // exp(i w delta) of each recurrence at its next pair
    double2 rot[kToneSlots];       // exp(i w dt)
    double2 middle[kToneSlots];    // exp(i w delta) at the middle step's samples
    double w[kToneSlots];          // the tones' frequencies
    double2 half_step[kToneSlots]; // FP64: exp(i w dt_out / 2)
    StepTimes times[kDmmaTile];    // FP64: the intervals' times (step_times)
    double late[kDmmaTile];        // FP64: how far each middle lies from where L puts it
    Su2p warp_product[kDmmaWarps];
    int32_t tile;
    int32_t magnus;                // 1: the tile takes the one-exponential Magnus step
};

// d[0..1] += a b over the 8 x 8 x 4 product of the warp (FP64 tensor path).
SS_D void dmma_m8n8k4(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

static_assert(kDmmaTile == kScanTile, "a CTA tile is one state scan tile (its warps' row products are its partials)");

// Frequency of tone slot (0 for an absent tone).
SS_D double dmma_frequency(const FieldDesc& f, int slot) {
    const int c = slot / kBulkTones, tone = slot % kBulkTones;
    return tone < f.tone_count[c] ? __ldg(f.tones + 3 * (f.tone_start[c] + tone)) : 0.0;
}

// Pairs before column r's first one (recurrence r = slot * 8 + column), counted from the middle of the interval.
SS_D double dmma_start(int K, int r) { return (double)dmma_segment(K, (r >> 1) & (kDmmaSegments - 1)) + (K & 1 ? 0.5 : 0.0); }

// Pair recurrence r = slot * 8 + column (column = 2 * segment + Gauss point): the phasor exp(i w delta) of its tone
// at the column's first distance from the middle of the interval, and the tone's step rotation exp(i w dt).
SS_D void dmma_recurrence(const FieldDesc& f, int K, double dt, int r, double2* z, double2* rot) {
    const int gauss = r & 1, slot = r >> 3;
    const int c = slot / kBulkTones, tone = slot % kBulkTones;
    *z = make_double2(0.0, 0.0);
    *rot = make_double2(1.0, 0.0);
    if (tone < f.tone_count[c]) {
        const double a = 0.5 * dt * (gauss ? 1.0 + 1.0 / kSqrt3 : 1.0 - 1.0 / kSqrt3);
        const double w = __ldg(f.tones + 3 * (f.tone_start[c] + tone));
        double sn, cs;
        sincos(w * fma(dmma_start(K, r), dt, a), &sn, &cs);
        *z = make_double2(cs, sn);
        sincos(w * dt, &sn, &cs);
        *rot = make_double2(cs, sn);
    }
}

// Recurrence r's phasor at its pair `pair`.  Out of line: the recurrences restart from it so rarely that its code
// should not be the step loop's.
inline __device__ __noinline__ double2 dmma_restart(const FieldDesc& f, int K, double dt, int r, int pair) {
    const int slot = r >> 3;
    if (slot % kBulkTones >= f.tone_count[slot / kBulkTones]) return make_double2(0.0, 0.0);
    const double a = 0.5 * dt * (r & 1 ? 1.0 + 1.0 / kSqrt3 : 1.0 - 1.0 / kSqrt3);
    double sn, cs;
    sincos(dmma_frequency(f, slot) * fma(dmma_start(K, r) + (double)pair, dt, a), &sn, &cs);
    return make_double2(cs, sn);
}

// exp(i w tau) of tone slot (1 for an absent tone).
SS_D double2 dmma_phasor(const FieldDesc& f, int slot, double tau) {
    const int c = slot / kBulkTones, tone = slot % kBulkTones;
    if (tone >= f.tone_count[c]) return make_double2(1.0, 0.0);
    double sn, cs;
    sincos(__ldg(f.tones + 3 * (f.tone_start[c] + tone)) * tau, &sn, &cs);
    return make_double2(cs, sn);
}

// 1 when the instance takes the Magnus step: theta = dt (|B|max + w_max) <= kMagnusTheta, |B|max from
// the channels' biases and amplitudes summed in a fixed order (every launch takes the same branch).
SS_D int32_t dmma_magnus(const FieldDesc& f, double dt) {
    double bsq = 0.0, wmax = 0.0;
    for (int c = 0; c < 3; c++) {
        double bc = fabs(f.bias[c]);
        for (int k = 0; k < f.tone_count[c] && k < kBulkTones; k++) {
            const double* tn = f.tones + 3 * (f.tone_start[c] + k);
            bc += fabs(f.gain[c] * __ldg(tn + 1));
            wmax = fmax(wmax, fabs(__ldg(tn)));
        }
        bsq = fma(bc, bc, bsq);
    }
    return dt * (sqrt(bsq) + wmax) <= kMagnusTheta ? 1 : 0;
}

#ifdef SPINSIM_DMMA_CONSTS_KERNEL
// The per-instance constants of the tensor path (DmmaConsts), one CTA of kDmmaRecurrences threads
// per instance, launched before the time evolution so its tiles load them instead of recomputing
// them (384 FP64 sincos and the step test per tile).  A single call (inst_out not null): the instance and
// field come with the arguments and are also written to device memory for the time evolution.
__global__ void __launch_bounds__(kDmmaRecurrences) dmma_consts_kernel(const __grid_constant__ EvolveArgs a,
                                                                       DmmaConsts* out, int32_t n, Instance* inst_out,
                                                                       FieldDesc* field_out) {
    grid_dependency_release();  // the time evolution may start its tiles' set-up meanwhile
    const int32_t i = blockIdx.x;
    if (i >= n) return;
    const Instance& inst = inst_out != nullptr ? a.single : a.instances[i];
    const FieldDesc& f = inst_out != nullptr ? a.single_field : a.fields[inst.field];
    if (inst_out != nullptr && threadIdx.x == 0) {
        *inst_out = a.single;
        *field_out = a.single_field;
    }
    if (!tones_on_tensor_path(f, inst.dim)) return;
    DmmaConsts& c = out[i];
    const int r = threadIdx.x;
    double2 z, rot;
    dmma_recurrence(f, inst.n_fine, inst.dt_int, r, &z, &rot);
    c.z[r] = z;
    if ((r & 7) == 0) c.rot[r >> 3] = rot;
    if (r < kToneSlots) {
        c.half_step[r] = dmma_phasor(f, r, 0.5 * inst.dt_out);
        c.middle[r] = dmma_phasor(f, r, inst.dt_int * (0.5 / kSqrt3));
    }
    if (r == 0) c.magnus = dmma_magnus(f, inst.dt_int);
}
#endif


// The interval's lab-frame operator from its SU(2) pair: itself (spin half) or its representation.
template <int D>
SS_D void store_interval_operator(const Su2p& v, double* u_out, int64_t idx) {
    const Mat<D> u = su2p_to_mat<D>(v);
    double2* dst = reinterpret_cast<double2*>(u_out) + idx * (D * D);
#pragma unroll
    for (int r = 0; r < D; r++)
#pragma unroll
        for (int k = 0; k < D; k++) dst[r * D + k] = make_double2(u.a[r][k].re, u.a[r][k].im);
}

// How far an output step's start, rounded as the reference rounds it (I:818), lies from t0 + dt_out i.
SS_D double time_rounding(double t0, double dt_out, double i) {
    const double p = __dmul_rn(dt_out, i), ep = __fma_rn(dt_out, i, -p);
    const double s = __dadd_rn(t0, p), b = __dsub_rn(s, t0);
    return -(__dadd_rn(__dsub_rn(t0, __dsub_rn(s, b)), __dsub_rn(p, b)) + ep);
}

inline __device__ __noinline__ StepTimes step_times(double t_c, double dt, int K) {
    StepTimes s;
    double step;
    if (even_steps(t_c, dt, K, &step)) {
        s.shift = 0.5 * (double)(K - 1) * (step - dt);
        s.stretch = (step - dt) / dt;
        return s;
    }
    // The few intervals in which the sum changes its exponent: the line through its deviations from t_c + j dt, a run
    // of steps of one exponent at a time.
    double t = t_c, off = 0.0, sum = 0.0, moment = 0.0;
    const double middle = 0.5 * (double)(K - 1);
    for (int j = 0; j < K;) {
        const double next = t + dt, d = ((next + dt) - next) - dt;
        const long long power = __double_as_longlong(t) & (long long)0xfff0000000000000ull;  // the power of two below |t|
        const double edge = __longlong_as_double(t < 0.0 ? power : power + 0x0010000000000000ll);
        const double room = (edge - t) / (dt + d);
        const int more = room >= (double)(K - 1 - j) ? K - 1 - j : max(0, (int)room);
        const double n = (double)more, c = n + 1.0;
        const double run = c * fma(0.5 * n, d, off);  // steps j .. j + more are late by off, off + d, ...
        sum += run;
        moment += fma((double)j - middle, run, 0.5 * n * c * fma((2.0 * n + 1.0) * (1.0 / 3.0), d, off));
        const double last = fma(n, dt + d, t);
        t = last + dt;
        off = fma(n, d, off) + ((t - last) - dt);
        j += more + 1;
    }
    const double n = (double)K;
    s.shift = K > 0 ? sum / n : 0.0;
    s.stretch = K > 1 ? 12.0 * moment / (n * (n * n - 1.0) * dt) : 0.0;
    return s;
}

template <bool B>
struct Flag {
    static constexpr bool value = B;
};

// One step's element from its samples in units of h / 2, FP32-bulk: the Magnus step or the reference's CF4
// (I:655-686).
template <bool MAGNUS>
SS_D Su2d dmma_step32(const double* sa, const double* sb, float* nsq) {
    if constexpr (MAGNUS) {
        // g = (h / 2)(b1 + b2) + (sqrt3 h^2 / 12) b2 x b1, with (h / 2) b in sa, sb: the linear part
        // g_lin = sa + sb stays FP64; the commutator (sqrt3 / 6) d x g_lin, d = (h / 2)(b2 - b1), and
        // the exponential's remainder are FP32.
        double gl64[3];
        float gl[3], dd[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            gl64[c] = sa[c] + sb[c];
            gl[c] = __double2float_rn(gl64[c]);
            dd[c] = __double2float_rn(sb[c] - sa[c]);
        }
        constexpr float kComm = 0.28867513459481287f;  // sqrt3 / 6
        const float cx = kComm * fmaf(dd[1], gl[2], -dd[2] * gl[1]);
        const float cy = kComm * fmaf(dd[2], gl[0], -dd[0] * gl[2]);
        const float cz = kComm * fmaf(dd[0], gl[1], -dd[1] * gl[0]);
        Su2f rest = su2_exp_rest(gl[0] + cx, gl[1] + cy, gl[2] + cz);
        rest.am1.im = fmaf(-0.5f, cz, rest.am1.im);  // the commutator's linear part
        rest.beta.re = fmaf(0.5f, cy, rest.beta.re);
        rest.beta.im = fmaf(-0.5f, cx, rest.beta.im);
        *nsq = fmaf(gl[0], gl[0], fmaf(gl[1], gl[1], fmaf(gl[2], gl[2], *nsq)));
        return su2_split(gl64[0], gl64[1], gl64[2], rest);
    } else {
        double ga[3], gb[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            ga[c] = fma(kDmmaW0, sa[c], kDmmaW1 * sb[c]);
            gb[c] = fma(kDmmaW1, sa[c], kDmmaW0 * sb[c]);
        }
        return su2_cf4_element(ga, gb, nsq);
    }
}

// The quad's four lanes hold products of consecutive pair segments; lane 0 of the quad gets the whole product:
// of steps after the middle (later segments from the left) and of mirrored steps before it (from the right).
template <bool MIRRORED>
SS_D void combine_segments(Su2d& p, int q) {
#pragma unroll
    for (int s = 1; s < kDmmaSegments; s <<= 1) {
        Su2d other = shfl_down_su2(p, s);
        if ((q & (2 * s - 1)) != 0) continue;
        if (MIRRORED) {
            su2_apply64(other, p);
            p = other;
        } else {
            su2_apply64(p, other);
        }
    }
}

// partial_out (may be null): the tile's scan partials, where this warp writes the lab-frame SU(2) pair of
// its rows' product (later rows from the left; rows past the tile's end are the identity); product_out (may be
// null): the tile's product as a d x d operator instead.  The spin dimension enters only the frame winding, the
// exponentiator and the stored operator, so a mixed-spin launch (DIMS 0) runs one copy of the step loop for
// both spins.
template <int DIMS, int PREC>
SS_D void tile_dmma(const MethodConfig& m, const Instance& inst, const FieldDesc& f, const Tile& tile, DmmaShared& sh,
                    double* time_out, double* u_out, float* norms_out, double* partial_out, double* product_out,
                    const DmmaConsts* cst, double* rows_out) {
    const int D = DIMS != 0 ? DIMS : inst.dim;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, q = lane & 3;
    const int row = (threadIdx.x >> 5) * kDmmaRows + g;
    const bool active = row < tile.count;
    const int64_t idx = tile.first + (active ? row : 0);
    const double dt = inst.dt_int, dt_out = inst.dt_out;
    const int K = inst.n_fine;
    const int seg_start = dmma_segment(K, q);
    const int seg_len = dmma_segment(K, q + 1) - seg_start;
    const int n_steps = (K / 2 + kDmmaSegments - 1) / kDmmaSegments;  // pairs of the longest segment
    const double a_lo = 0.5 * dt * (1.0 - 1.0 / kSqrt3);
    const double a_hi = 0.5 * dt * (1.0 + 1.0 / kSqrt3);
    const double half_dt = 0.5 * dt;
    const double t_c = __dadd_rn(inst.t0, __dmul_rn(dt_out, (double)(inst.interval0 + idx)));  // I:818, unfused

    // The instance's constants (dmma_consts_kernel, which may still be running: it lets this launch start early).
    grid_dependency_wait();
    for (int r = threadIdx.x; r < kDmmaRecurrences; r += kDmmaThreads) sh.z[r] = cst->z[r];
    if (threadIdx.x < kToneSlots) {
        sh.rot[threadIdx.x] = cst->rot[threadIdx.x];
        sh.middle[threadIdx.x] = cst->middle[threadIdx.x];
        if constexpr (PREC == PREC_FP64) sh.half_step[threadIdx.x] = cst->half_step[threadIdx.x];
    }
    if (threadIdx.x == 0) sh.magnus = cst->magnus;

    // L of every tone at the middle of every interval of the tile (buffer 1 of the table holds it until the first
    // refill): thread 4 slot + quarter takes intervals 8 quarter .. 8 quarter + 7, stepping with exp(i w dt_out) from
    // the call's every eighth interval, so that a piece of a call rounds as the whole does.
    double2* lval = reinterpret_cast<double2*>(&sh.table[1][0][0]);  // [slot][interval of the tile]
    static_assert(sizeof(sh.table[1]) >= sizeof(double2) * kToneSlots * kDmmaTile, "L table fits one buffer");
    if (threadIdx.x < 4 * kToneSlots) {
        const int slot = threadIdx.x >> 2, quarter = threadIdx.x & 3;
        const int c = slot / kBulkTones, tone = slot % kBulkTones;
        const int64_t i0 = inst.interval0 + tile.first + kDmmaRows * quarter;
        const bool present = tone < f.tone_count[c];
        const double* tn = f.tones + (present ? 3 * (f.tone_start[c] + tone) : 0);
        const double w = dmma_frequency(f, slot);
        c64 l = c64{0.0, 0.0}, h = c64{1.0, 0.0};
        if (present) {
            const double2 hs = cst->half_step[slot];
            h = c64{hs.x, hs.y};
        }
        const c64 gstep = h * h;
        if (quarter == 0) sh.w[slot] = w;
#pragma unroll 1
        for (int64_t i = i0 & ~(int64_t)(kDmmaRows - 1); i < i0 + kDmmaRows; i++) {
            if (present && (i & (kDmmaRows - 1)) == 0) {
                const double amp = f.gain[c] * __ldg(tn + 1);
                const double tq = __dadd_rn(inst.t0, __dmul_rn(dt_out, (double)i));  // as the intervals' own t_c
                // the phase w tq + phi to twice the precision: its rounding, of which each of the reference's samples has
                // its own, would be that of all steps of eight intervals
                const double p = __dmul_rn(w, tq), phi = __ldg(tn + 2), phase = __dadd_rn(p, phi);
                const double b = __dsub_rn(phase, p);
                const double rest = __dadd_rn(__dsub_rn(p, __dsub_rn(phase, b)), __dsub_rn(phi, b)) + __fma_rn(w, tq, -p);
                double sn, cs;
                sincos(phase, &sn, &cs);
                l = half_dt * amp * c64{fma(-rest, sn, cs), fma(rest, cs, sn)} * h;
            }
            if (i >= i0) lval[slot * kDmmaTile + kDmmaRows * quarter + (int)(i - i0)] = make_double2(l.re, l.im);
            l = l * gstep;
        }
    } else if constexpr (PREC == PREC_FP64) {  // the last warp meanwhile: each interval's times
        static_assert(4 * kToneSlots + kDmmaTile == kDmmaThreads, "a thread per interval beside the tones'");
        const int r = threadIdx.x - 4 * kToneSlots;
        const int64_t index = inst.interval0 + tile.first + r, from = index & ~(int64_t)(kDmmaRows - 1);
        const StepTimes times = step_times(__dadd_rn(inst.t0, __dmul_rn(dt_out, (double)index)), dt, K);
        sh.times[r] = times;
        sh.late[r] = time_rounding(inst.t0, dt_out, (double)index) - time_rounding(inst.t0, dt_out, (double)from) + times.shift;
    }
    __syncthreads();  // producer phasors, rotations, step choice and L in place

    // A operands: L of this lane's interval for tone 4 s + q, its imaginary part for the even sums, real for the
    // odd.
    //
    // In FP64 corrected for the reference's times.  Its samples are taken at the running sum of the steps (I:836), whose
    // rounding is the same for all steps of the same exponent and for whole stretches of a call, so that a resonant
    // drive shows it (1 MHz at 100 steps of 10 ns, states 1.1e-8 off at 10 ms, 5e-12 so; 64 mixed instances 551 -> 572 us).
    // An interval's samples then lie `shift` later and are stretched about their middle.  The shift, with how the interval's start is rounded relative to the one
    // whose phase was taken at its rounded start, is a small turn of L.  Evolving with H(t_m + (1 + stretch) tau) is
    // evolving with H / (1 + stretch) over (1 + stretch) times as long: L and the bias take the factor here, the ends'
    // extra time is two small elements below.  Both are the interval's own, so pieces of a call round as the whole does.
    double late = 0.0, scale = 1.0;
    if constexpr (PREC == PREC_FP64) {
        late = sh.late[row];
        scale = 1.0 - sh.times[row].stretch;
    }
    double even_a[3][2], odd_a[3][2];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const double2 lv = lval[(c * kBulkTones + 4 * s + q) * kDmmaTile + row];
            if constexpr (PREC == PREC_FP64) {
                const double turn = late * sh.w[c * kBulkTones + 4 * s + q];
                even_a[c][s] = active ? scale * fma(turn, lv.x, lv.y) : 0.0;
                odd_a[c][s] = active ? scale * fma(-turn, lv.y, lv.x) : 0.0;
            } else {
                even_a[c][s] = active ? lv.y : 0.0;
                odd_a[c][s] = active ? lv.x : 0.0;
            }
        }
    // Rotating frame (I:823-829): Bz at the middle of the interval, sum_k Im L_zk + bias, over the quad's
    // tones.  prw: P times the frame's rate (for either spin).
    double prw = 0.0;
    if (m.rotating) {
        double part = even_a[2][0] + even_a[2][1];
        part += __shfl_xor_sync(0xffffffffu, part, 1);
        part += __shfl_xor_sync(0xffffffffu, part, 2);
        prw = f.bias[2] + part / half_dt;
    }
    // (h / 2) bias, the starting value of the even sums; in the rotating frame z also carries the frame's
    // -P rw (I:582-618), added once here instead of to every sample
    double bias[3];
#pragma unroll
    for (int c = 0; c < 3; c++) bias[c] = __dmul_rn(half_dt, f.bias[c]);
    bias[2] = __fma_rn(-half_dt, prw, bias[2]);
    if constexpr (PREC == PREC_FP64)
#pragma unroll
        for (int c = 0; c < 3; c++) bias[c] *= scale;
    // Frame phasors at the Gauss points of this segment's steps after the middle: exp(-i P rw delta); those of
    // the mirrored steps before it are their conjugates
    const double start = (double)seg_start + (K & 1 ? 0.5 : 0.0);
    c64 wa = c64{1.0, 0.0}, wb = c64{1.0, 0.0}, wrot = c64{1.0, 0.0};
    if (m.rotating) {
        sincos_small(-prw * dt, &wrot.im, &wrot.re);
        sincos_small(-prw * fma(start, dt, a_lo), &wa.im, &wa.re);
        sincos_small(-prw * fma(start, dt, a_hi), &wb.im, &wb.re);
    }

    // Fill table buffer (ph & 1) with the B operands of pairs [ph kDmmaPhase, ...) of every segment.
    auto fill = [&](int ph) {
        const int m0 = ph * kDmmaPhase;
        const int mc = min(kDmmaPhase, n_steps - m0);
        for (int r = threadIdx.x; r < kDmmaRecurrences; r += kDmmaThreads) {
            const int col = r & 7, slot = r >> 3;
            const int c = slot / kBulkTones, tone = slot % kBulkTones;
            // consumer lane 4 col + tone % 4 of k-step tone / 4: cosines (even sums), then sines
            double* dst = &sh.table[ph & 1][0][(c * 4 + (tone >> 2)) * 32 + 4 * col + (tone & 3)];
            double2 z = sh.z[r];
            const double2 rt = sh.rot[slot];
            for (int mm = 0; mm < mc; mm++) {
                dst[mm * kDmmaChunkDoubles] = z.x;
                dst[mm * kDmmaChunkDoubles + 64] = z.y;
                z = make_double2(fma(z.x, rt.x, -z.y * rt.y), fma(z.x, rt.y, z.y * rt.x));
            }
            sh.z[r] = z;
        }
    };

    Su2d after = Su2d{c64{0.0, 0.0}, c64{0.0, 0.0}};   // this lane's steps after the middle
    Su2d before = Su2d{c64{0.0, 0.0}, c64{0.0, 0.0}};  // and their mirrored steps before it
    float nsq = 0.0f;  // sum of |g|^2 over this lane's steps (the error statement's scale)
    const bool lie_trotter = D == 3 || m.expo_half == EXPO_LIE_TROTTER;
    // An xy sample in the rotating frame (I:582-618; z: in the bias)
    auto rotate = [&](double* s, c64 w) {
        const c64 x = c64{s[0], s[1]} * w;
        s[0] = x.re;
        s[1] = x.im;
    };
    // p <- step p (a step after p's), or p step (a mirrored step, before p's)
    auto apply = [&](auto magnus, Su2d& p, double* sa, double* sb, bool mirrored) {
        Su2d e;
        if constexpr (PREC == PREC_FP32_BULK) {
            e = dmma_step32<decltype(magnus)::value>(sa, sb, &nsq);
        } else {  // the reference's CF4 (I:655-686) with FP64 exponentials
            double ga[3], gb[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                ga[c] = fma(kDmmaW0, sa[c], kDmmaW1 * sb[c]);
                gb[c] = fma(kDmmaW1, sa[c], kDmmaW0 * sb[c]);
            }
            e = su2_step_element64(m, lie_trotter, ga);
            const Su2d eb = su2_step_element64(m, lie_trotter, gb);
            if (!mirrored) {
                su2_apply64(p, e);
                e = eb;
            } else {
                su2_apply64(e, eb);
            }
        }
        if (mirrored) {
            su2_apply64(e, p);
            p = e;
        } else {
            su2_apply64(p, e);
        }
    };

    fill(0);  // buffer 0; buffer 1 (the L table) is first refilled after the barrier below
    if (K & 1) {  // the middle step, whose two samples mirror each other: column 0 of one more product
        double ev[3], od[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            double e0 = bias[c], e1 = 0.0, o0 = 0.0, o1 = 0.0;
#pragma unroll
            for (int s = 0; s < 2; s++) {
                const double2 z = sh.middle[c * kBulkTones + 4 * s + q];
                dmma_m8n8k4(e0, e1, even_a[c][s], g == 0 ? z.x : 0.0);
                dmma_m8n8k4(o0, o1, odd_a[c][s], g == 0 ? z.y : 0.0);
            }
            ev[c] = e0;
            od[c] = o0;
        }
        if (active && q == 0) {
            double sa[3], sb[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                sa[c] = ev[c] - od[c];
                sb[c] = ev[c] + od[c];
            }
            if (m.rotating) {
                c64 w;
                sincos_small(-prw * (dt * (0.5 / kSqrt3)), &w.im, &w.re);
                rotate(sa, conj(w));
                rotate(sb, w);
            }
            if (PREC == PREC_FP32_BULK && sh.magnus != 0) apply(Flag<true>(), after, sa, sb, false);
            else apply(Flag<false>(), after, sa, sb, false);
        }
    }
    __syncthreads();
    const int n_phases = (n_steps + kDmmaPhase - 1) / kDmmaPhase;
    // The step loop, one copy for each kind of step (both inside one loop do not fit the instruction cache).
    auto steps = [&](auto magnus, int from, int to) {
        for (int ph = from; ph < to; ph++) {
            if (ph + 1 < n_phases) fill(ph + 1);
            const int m0 = ph * kDmmaPhase;
            const int mc = min(kDmmaPhase, n_steps - m0);
            const double* tb = &sh.table[ph & 1][0][lane];
            // Even and odd sums at the two distances of pair mm (tensor path), issued at the end of pair mm - 1, so
            // they are in flight while the next pair begins.
            double e0[3], e1[3], o0[3], o1[3];
            auto sums = [&](int mm) {
    #pragma unroll
                for (int c = 0; c < 3; c++) {
                    e0[c] = e1[c] = bias[c];
                    o0[c] = o1[c] = 0.0;
                    const double* t = tb + mm * kDmmaChunkDoubles + c * 128;
    #pragma unroll
                    for (int s = 0; s < 2; s++) {
                        dmma_m8n8k4(e0[c], e1[c], even_a[c][s], t[32 * s]);
                        dmma_m8n8k4(o0[c], o1[c], odd_a[c][s], t[64 + 32 * s]);
                    }
                }
            };
            sums(0);
            for (int mm = 0; mm < mc; mm++) {
                if (active && m0 + mm < seg_len) {
                    double sa[3], sb[3], ma[3], mb[3];  // the step after the middle, and its mirror image
    #pragma unroll
                    for (int c = 0; c < 3; c++) {
                        sa[c] = e0[c] + o0[c];
                        sb[c] = e1[c] + o1[c];
                        ma[c] = e1[c] - o1[c];
                        mb[c] = e0[c] - o0[c];
                    }
                    if (m.rotating) {
                        rotate(sa, wa);
                        rotate(sb, wb);
                        rotate(ma, conj(wb));
                        rotate(mb, conj(wa));
                        wa = wa * wrot;
                        wb = wb * wrot;
                    }
                    apply(magnus, after, sa, sb, false);
                    apply(magnus, before, ma, mb, true);
                }
                // the next pair's sums, issued after this pair's arithmetic (all lanes: mma.sync is
                // warp-collective); measured 0.7% faster than issuing them before it
                if (mm + 1 < mc) sums(mm + 1);
            }
            __syncthreads();  // buffer (ph & 1) is refilled in phase ph + 1
        }
    };
    if constexpr (PREC == PREC_FP64) {
        for (int from = 0; from < n_phases; from += kDmmaRestart) {
            if (from > 0) {
                // buffer (from & 1) is filled: the table's recurrences restart at the next phase (each thread's own)
                for (int r = threadIdx.x; r < kDmmaRecurrences; r += kDmmaThreads)
                    sh.z[r] = dmma_restart(f, K, dt, r, (from + 1) * kDmmaPhase);
                if (m.rotating) {
                    const double at = start + (double)(from * kDmmaPhase);
                    const PhasorPair p = phasor_pair(-prw * fma(at, dt, a_lo), -prw * fma(at, dt, a_hi));
                    wa = p.a;
                    wb = p.b;
                }
            }
            steps(Flag<false>(), from, min(from + kDmmaRestart, n_phases));
        }
    } else {
        if (sh.magnus != 0) steps(Flag<true>(), 0, n_phases);
        else steps(Flag<false>(), 0, n_phases);
    }

    // The interval's product, in lane 0 of the quad
    combine_segments<false>(after, q);
    combine_segments<true>(before, q);
    c64 half_frame = c64{1.0, 0.0};  // the frame's turn over half an output step
    if (m.rotating) sincos_small(-0.5 * prw * dt_out, &half_frame.im, &half_frame.re);
    if constexpr (PREC == PREC_FP64) {
        // The ends' extra time: 1 - i (stretch T / 2) B.sigma / 2, T = K dt, with the ends' samples summed over the quad
        // (one column would leave seven eighths of a tensor product idle).
        double first[3], last[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double2 z0 = sh.half_step[c * kBulkTones + q], z1 = sh.half_step[c * kBulkTones + 4 + q];
            double even = fma(even_a[c][0], z0.x, even_a[c][1] * z1.x);
            double odd = fma(odd_a[c][0], z0.y, odd_a[c][1] * z1.y);
#pragma unroll
            for (int s = 1; s < kDmmaSegments; s <<= 1) {
                even += __shfl_xor_sync(0xffffffffu, even, s);
                odd += __shfl_xor_sync(0xffffffffu, odd, s);
            }
            first[c] = bias[c] + even - odd;
            last[c] = bias[c] + even + odd;
        }
        if (m.rotating) {
            rotate(first, conj(half_frame));
            rotate(last, half_frame);
        }
        const double n = 0.5 * sh.times[row].stretch * (double)K;
        Su2d p = Su2d{c64{0.0, -n * first[2]}, c64{n * first[1], -n * first[0]}};
        su2_apply64(p, before);
        before = p;
        su2_apply64(after, Su2d{c64{0.0, -n * last[2]}, c64{n * last[1], -n * last[0]}});
    }
    su2_apply64(before, after);
    if constexpr (PREC == PREC_FP32_BULK) {
#pragma unroll
        for (int s = 1; s < kDmmaSegments; s <<= 1) nsq += __shfl_down_sync(0xffffffffu, nsq, s);
    }
    // The interval's lab-frame operator as an SU(2) pair.  With the frame's phases counted from the middle of the
    // interval, entering and leaving the frame (I:839-852) multiply alpha by exp(-i P rw dt_out / 2) and leave
    // beta (spin one: the same element's representation).  Rows past the tile's end and the other lanes of a quad
    // hold the identity.
    Su2p v = su2p_identity();
    if (active && q == 0) {
        v.a = c64{1.0 + before.am1.re, before.am1.im};
        v.b = before.beta;
        if (m.rotating) {
            v.a = v.a * half_frame;
            if constexpr (PREC == PREC_FP64) {  // the phases counted from half an output step and the middle's shift
                const double x = -prw * sh.times[row].shift;
                v.b = c64{fma(-x, v.b.im, v.b.re), fma(x, v.b.re, v.b.im)};
            }
        }
        time_out[idx] = t_c;
        if (norms_out != nullptr) norms_out[idx] = nsq;
        if (D == 2) store_interval_operator<2>(v, u_out, idx);
        else store_interval_operator<3>(v, u_out, idx);
        if (rows_out != nullptr) {  // the same operator as its SU(2) pair, for the state scan
            double2* r = reinterpret_cast<double2*>(rows_out) + 2 * idx;
            r[0] = make_double2(v.a.re, v.a.im);
            r[1] = make_double2(v.b.re, v.b.im);
        }
    }
    if (partial_out == nullptr && product_out == nullptr) return;
#pragma unroll
    for (int sft = kDmmaSegments; sft < 32; sft <<= 1) {  // the warp's product of its rows (lanes 4 g), later rows from the left
        const Su2p later = shfl_down_su2p(v, sft);
        if ((lane & (2 * sft - 1)) == 0) v = su2p_mul(later, v);
    }
    if (partial_out != nullptr && lane == 0) {
        double2* dst = reinterpret_cast<double2*>(partial_out) + 2 * (threadIdx.x >> 5);
        dst[0] = make_double2(v.a.re, v.a.im);
        dst[1] = make_double2(v.b.re, v.b.im);
    }
    if (product_out != nullptr) {
        if (lane == 0) sh.warp_product[threadIdx.x >> 5] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < kDmmaWarps; w++) v = su2p_mul(sh.warp_product[w], v);
            if (D == 2) store_interval_operator<2>(v, product_out, 0);
            else store_interval_operator<3>(v, product_out, 0);
        }
    }
}

// More tones than the products take, or a quadratic shift: one interval per thread (not inlined, so its
// registers do not weigh on the tensor path's step loop).
template <int DIMS>
__device__ __noinline__ void dmma_tile_fallback(const MethodConfig& m, const Instance& inst, const FieldDesc& f,
                                                int64_t interval, bool active, double* time_out, double* u_out,
                                                float* norms_out) {
    interval32<DIMS, INTEG_CF4, FIELD_TONES>(m, inst, f, interval, active, 0, time_out, u_out, norms_out, nullptr);
}

// Persistent launch: CTAs pull tiles of kDmmaTile intervals from the queue (or, without a queue, CTA
// b takes tile b of a single instance).
template <int DIMS, int PREC>
SS_D void evolve_dmma_body(const EvolveArgs& a, DmmaShared& sh) {
    int64_t tile_id = blockIdx.x;
    if (a.tiles == nullptr) grid_dependency_wait();  // a single call: its descriptors come from dmma_consts_kernel
    int32_t reserved = -1;  // thread 0: the next tile, taken from the queue while this one runs
    for (;;) {
        if (a.tile_counter != nullptr) {
            if (threadIdx.x == 0) sh.tile = reserved >= 0 ? reserved : atomicAdd(a.tile_counter, 1);
            __syncthreads();
            tile_id = sh.tile;
            // Away from the end of the queue, take the next tile now (its atomic's latency then passes
            // during this tile); near the end tiles are taken only when a CTA is free, so no CTA holds
            // a tile that another could have run.
            if (threadIdx.x == 0)
                reserved = tile_id + 2 * (int64_t)gridDim.x < a.n_tiles ? atomicAdd(a.tile_counter, 1) : -1;
        }
        if (tile_id >= a.n_tiles) {
            grid_dependency_release();  // no tiles left for this CTA: the scan may start launching
            return;
        }
        Tile tile;
        if (a.tiles != nullptr) {
            tile = a.tiles[tile_id];
        } else {
            const int64_t n = a.instances[0].n_out;
            tile.instance = 0;
            tile.first = tile_id * kDmmaTile;
            tile.count = (int)((n - tile.first) < kDmmaTile ? (n - tile.first) : kDmmaTile);
        }
        const Instance& inst = a.instances[tile.instance];
        const FieldDesc& f = a.fields[inst.field];
        double* time_out = a.time + inst.out_offset;
        double* u_out = a.u + inst.u_offset;
        float* norms_out = a.step_norms != nullptr ? a.step_norms + inst.out_offset : nullptr;
        const int dim = (DIMS == 0) ? inst.dim : DIMS;
        if (PREC == PREC_FP64 || tones_on_tensor_path(f, dim)) {
            const int64_t k = (a.scan_begin != nullptr ? a.scan_begin[tile.instance] : 0) + tile.first / kScanTile;
            double* partial_out = a.tile_partials != nullptr ? a.tile_partials + k * kScanMat : nullptr;
            double* product_out = a.tile_products != nullptr ? a.tile_products + k * kScanMat : nullptr;
            double* rows_out = a.rows != nullptr ? a.rows + 4 * inst.out_offset : nullptr;
            tile_dmma<DIMS, PREC>(a.m, inst, f, tile, sh, time_out, u_out, norms_out, partial_out, product_out,
                                  a.dmma_consts + tile.instance, rows_out);
        } else if constexpr (PREC == PREC_FP32_BULK) {
            if (threadIdx.x < kDmmaTile) {  // one warp
                const bool active = (int)threadIdx.x < tile.count;
                dmma_tile_fallback<DIMS>(a.m, inst, f, tile.first + (active ? threadIdx.x : 0), active, time_out, u_out,
                                         norms_out);
            }
        }
        __syncthreads();  // shared memory and the tile slot are reused by the next tile
        if (a.tile_counter == nullptr) return;
    }
}

// MINB: minimum resident CTAs per SM for the register allocation (6: 80 registers, 5: 96, 4: 128, 3: 168).
template <int DIMS, int PREC, int MINB>
__global__ void __launch_bounds__(kDmmaThreads, MINB) evolve_dmma_kernel(EvolveArgs a) {
    __shared__ DmmaShared sh;
    evolve_dmma_body<DIMS, PREC>(a, sh);
}

}  // namespace spinsim
