// Plain FP64 time evolution of one output interval: the reference's get_time_evolution_loop
// (spinsim/__init__.py:797-852) with its integrators (I:622-794), frame transforms (I:582-618) and
// step composition (I:561-580).  All operators live in registers.
//
// An interval's K fine steps may be shared by `lanes` consecutive lanes of a warp: lane l runs
// steps [l K / lanes, (l + 1) K / lanes) and the partial products are combined in step order with
// warp shuffles (the later product multiplies from the left, as append_exponentiation does).
#pragma once
#include "common.cuh"
#include "expo64.cuh"
#include "fields.cuh"

namespace spinsim {

// Components of the field vector (I:547-554); spin half in a mixed-spin kernel (DIMS 0) ignores the fourth.
template <int DIMS, int EXPO_ONE>
struct LieDim {
    static constexpr int value = DIMS == 2 ? 3 : EXPO_ONE == EXPO_LIE_TROTTER_8 ? 8 : 4;
};

// transform_frame_* for the eight-generator exponential (I:582-618).  Division by the unit winding w is
// written as multiplication by its conjugate.
SS_D void transform_frame_lt8(double* s, double rw, c64 w) {
    const c64 wc = conj(w);
    c64 X = c64{s[0], s[1]} * wc;
    s[0] = X.re;
    s[1] = X.im;
    s[2] = s[2] - rw;
    X = (c64{s[4], s[5]} * wc) * wc;
    s[4] = X.re;
    s[5] = X.im;
    X = c64{s[6], s[7]} * wc;
    s[6] = X.re;
    s[7] = X.im;
}

// Frame phasors restart from sincos after this many steps of their recurrence (a power of two), so that their
// drift (about one rounding a step) stays far below the phase's own argument rounding.
constexpr int kPhasorSteps = 64;

struct PhasorPair {
    c64 a, b;
};

// exp(i x) and exp(i y).  Out of line: the step loops restart their phasors so rarely that its code and registers
// should not be theirs.
__attribute__((const)) inline __device__ __noinline__ PhasorPair phasor_pair(double x, double y) {
    PhasorPair p;
    sincos_small(x, &p.a.im, &p.a.re);
    sincos_small(y, &p.b.im, &p.b.re);
    return p;
}

// Where an interval's steps sample the field and how they weight the samples: the interval's start, the
// reference's sample offsets and weights of an integrator for steps of dt (I:624-686 Magnus CF4 at the two
// Gauss points, I:693-752 Heun at the step's ends, I:759-791 Euler at its middle).  Samples are taken at the
// reference's own times, rounded as it rounds them: offsets from the running sum of the steps (I:836), in FP64 at
// the steps' ends and middles also by way of their distance from the interval's start (I:705-716, another
// rounding only next to time zero; no edge lies on a Gauss point).  Which side of a field's edge a sample on it falls
// depends on that, and with a fast field the roundings add up over a call (10 MHz, 10 ns, 10^6 steps: states
// 8e-9 from those of times j dt).  The frame's phase is taken at the same times (FP64; the FP32-bulk frame turns
// uniformly), so that the part of the field's phase that is common with it cancels.
struct StepRule {
    double t_c, dt, off_a, off_b, c0, c1;

    // A sample's time from the running sum plus its offset.
    template <int INTEG, bool FP64>
    SS_D double sample_time(double t) const {
        return FP64 && INTEG != INTEG_CF4 ? (t - t_c) + t_c : t;
    }
};

template <int INTEG>
SS_D StepRule step_rule(double t_c, double dt) {
    const double a_lo = 0.5 * dt * (1.0 - 1.0 / kSqrt3);
    const double a_hi = 0.5 * dt * (1.0 + 1.0 / kSqrt3);
    const double w0 = (1.5 + kSqrt3) / 6.0, w1 = (1.5 - kSqrt3) / 6.0;
    StepRule r;
    r.t_c = t_c;
    r.dt = dt;
    r.off_a = INTEG == INTEG_CF4 ? a_lo : INTEG == INTEG_HEUN ? 0.0 : 0.5 * dt;
    r.off_b = INTEG == INTEG_CF4 ? a_hi : dt;
    r.c0 = INTEG == INTEG_CF4 ? dt * w0 : INTEG == INTEG_HEUN ? 0.5 * dt : dt;
    r.c1 = INTEG == INTEG_CF4 ? dt * w1 : 0.0;
    return r;
}

// Whether the running sum t + dt + dt ... takes n equal steps: while it keeps its sign and exponent, each rounds to
// the same multiple of its last place (*step), but for a first one halfway between two.  The sum after j steps is
// then t + j *step exactly.
SS_D bool even_steps(double t, double dt, int n, double* step) {
    const double next = t + dt;
    *step = (next + dt) - next;
    const double end = fma((double)n, *step, t);
    return *step == next - t && ((__double2hiint(t) ^ __double2hiint(end)) & 0xfff00000) == 0;
}

// What a step loop's field samples need: the rule, the step's start, the frame phasors exp(-i prw tau), prw = P rw
// with P the power of the frame winding in the xy transform (I:599-613: 2 for spin half, 1 for spin one), at the
// step's two samples and their rotation by one step, and the table cursors.
//
// The phasors turn by the running sum's own step (even_steps), and restart at the sum itself.  Measured against
// correcting the phasors of uniform steps to the sum: the pulse ensemble 3075 -> 2823 us (2784 at uniform times).
template <int L>
struct Steps : StepRule {
    c64 wa, wb, wrot;
    double prw, t_fine;
    bool rotating;
    int restart_steps;
    TableCursor cur[L];

    SS_D Steps(const StepRule& rule) : StepRule(rule) {}

    template <int INTEG>
    SS_D void start_phasors() {
        const PhasorPair p = phasor_pair(-prw * ((t_fine + off_a) - t_c),
                                         INTEG != INTEG_EULER ? -prw * ((t_fine + off_b) - t_c) : 0.0);
        wa = p.a;
        wb = p.b;
    }
    // Steps first .. end - 1 of an interval.
    template <int INTEG>
    SS_D void begin(const MethodConfig& m, double interval_prw, int first, int end) {
        prw = interval_prw;
        t_fine = t_c;
        for (int k = 0; k < first; k++) t_fine += dt;
        rotating = m.rotating;
        restart_steps = kPhasorSteps;
        wa = wb = wrot = c64{1.0, 0.0};
        if (m.rotating && end > first && prw != 0.0) {
            // Where the steps are not even and that shows, the phasors restart at every one.
            double step;
            if (!even_steps(t_fine, dt, end - first, &step) &&
                fabs(prw) * fma((double)(end - first), dt, fabs(t_fine)) * (0x1p-52 * (double)(end - first)) > 1e-14)
                restart_steps = 1;
            sincos_small(-prw * step, &wrot.im, &wrot.re);
            start_phasors<INTEG>();
        }
#pragma unroll
        for (int c = 0; c < L; c++) cur[c] = TableCursor{};  // for the increasing sample times of the steps
    }
    // Before the samples of step n of a lane that began at step n0.
    template <int INTEG>
    SS_D void restart(int n, int n0) {
        if (rotating && prw != 0.0 && ((n - n0) & (restart_steps - 1)) == 0) start_phasors<INTEG>();
    }
};

// One step's field samples (FP64) -> frame transform -> the integrator's generators (FP64); the
// step's start and the frame phasors move on.
template <int FIELD, int L, int INTEG, bool FP64>
SS_D void step_generators(const FieldDesc& f, Steps<L>& st, double* ga, double* gb) {
    double s0[8], s1[8];  // a user field writes all eight channels
#pragma unroll
    for (int k = 0; k < 8; k++) {
        s0[k] = 0.0;
        s1[k] = 0.0;
    }
    const double at_a = st.template sample_time<INTEG, FP64>(st.t_fine + st.off_a);
    const double at_b = st.template sample_time<INTEG, FP64>(st.t_fine + st.off_b);
    st.t_fine += st.dt;
    sample_field<FIELD, L>(f, at_a, s0, st.cur);
    if (INTEG != INTEG_EULER) sample_field<FIELD, L>(f, at_b, s1, st.cur);
    if (st.rotating) {  // xy times exp(-i prw tau), z minus prw
        const c64 xa = c64{s0[0], s0[1]} * st.wa;
        s0[0] = xa.re;
        s0[1] = xa.im;
        s0[2] -= st.prw;
        st.wa = st.wa * st.wrot;
        if (INTEG != INTEG_EULER) {
            const c64 xb = c64{s1[0], s1[1]} * st.wb;
            s1[0] = xb.re;
            s1[1] = xb.im;
            s1[2] -= st.prw;
            st.wb = st.wb * st.wrot;
        }
    }
#pragma unroll
    for (int k = 0; k < L; k++) {  // Euler: the one generator in ga (gb zero)
        ga[k] = fma(st.c0, s0[k], st.c1 * s1[k]);
        gb[k] = INTEG == INTEG_HEUN ? st.c0 * s1[k] : fma(st.c1, s0[k], st.c0 * s1[k]);
    }
}

struct Generators4 {
    double a[4], b[4];
};

// Steps j0 .. j1 - 1 of an interval whose field is piecewise constant and whose frame does not turn (pulse
// trains), as runs: the steps between two knots share one element, and their product is its power by
// squarings; a step with a knot between its samples is a run of its own.  element(ga, gb, n) is the element of
// n steps of these generators.  Every lane of the warp calls this.  False, and p of no use, for lanes that do not
// take this form: all of them, or those with a sample so near to a knot that its time's roundings decide the side
// it falls on (a knot on the sample times of Heun or Euler), which only the running sum tells.  Bound by
// latency (the knots' search and the runs' divergence).  A launch of 400 pulse trains (4.1e6 output steps of 20,
// FP32-bulk, 128 registers), time evolution and scan: 3059 us step by step, 777 so, 899 with the running sum in here.
template <int INTEG, typename Element>
SS_D bool hold_steps(const FieldDesc& f, int dim, bool turns, const StepRule& st, int j0, int j1, double dt_out, Su2d& p,
                     Element element) {
    if (__any_sync(0xffffffffu, turns)) return false;
    HoldChannel ch[3];
    const double first = __shfl_sync(0xffffffffu, st.t_c, 0);
    const double dt = st.dt, last = INTEG == INTEG_EULER ? st.off_a : st.off_b;
    // twice as far as the roundings of a time here and of the running sum (I:836) may be apart
    const double slack = (double)(j1 + 4) * 0x1p-51 * (fabs(st.t_c) + dt_out);
    if (!hold_channels(f, dim == 2 ? 3 : 4, first, first + 33.0 * dt_out, slack, ch)) return false;
    bool near = false;
    for (int j = j0, n; j < j1 && !near; j += n) {
        const double ta = st.t_c + fma((double)j, dt, st.off_a), tb = st.t_c + fma((double)j, dt, last);
        double sa[3], ga[3], gb[3];
        double until = INFINITY;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            sa[c] = ch[c].at(f, c, ta, slack, near);
            until = fmin(until, ch[c].clear);
        }
        n = 1;
        if (tb < until) {
            // an estimate, made safe below: a run cut short goes on as another one
            const float more = __fdividef((float)(until - tb), (float)dt);
            n = more >= (float)(j1 - j) ? j1 - j : 1 + (int)more;
            while (n > 1 && !(st.t_c + fma((double)(j + n - 1), dt, last) < until)) n--;
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double sb = INTEG == INTEG_EULER ? 0.0 : tb < until ? sa[c] : ch[c].at(f, c, tb, slack, near);
            ga[c] = fma(st.c0, sa[c], st.c1 * sb);
            gb[c] = INTEG == INTEG_HEUN ? st.c0 * sb : fma(st.c1, sa[c], st.c0 * sb);
        }
        su2_apply_power64(p, element(ga, gb, n), n);
    }
    return !near;
}

// Steps j .. j1 - 1 of a spin-one interval whose quadratic shift is non-zero: full 3 x 3 exponentials
// and products, from the product u of the steps before.  On entry step j's generators are in g and st is at
// step j + 1.  Out of line, its state passed by value, so that the registers of the common
// SU(2) loop are allocated without this path's; loops are kept rolled, since a user field's kernel is linked when
// its simulator is made (with the other rolled loops of the 3 x 3 path an image of 567 -> 455 KB, linked in 0.8 ->
// 0.3 to 0.7 s, and no slower: 4001 x 50 steps 37.6 -> 37.0 us).
template <int INTEG, int FIELD>
__device__ __noinline__ Mat<3> spin_one_quadratic_steps64(const MethodConfig& m, const FieldDesc& f, Steps<4> st,
                                                          Mat<3> u, Generators4 g, int j0, int j, int j1) {
    for (;;) {
#pragma unroll 1
        for (int e = 0; e < (INTEG == INTEG_EULER ? 1 : 2); e++) {
            spin_one_step64(m, u, g.a);
#pragma unroll
            for (int c = 0; c < 4; c++) g.a[c] = g.b[c];
        }
        if (++j >= j1) return u;
        st.template restart<INTEG>(j, j0);
        step_generators<FIELD, 4, INTEG, true>(f, st, g.a, g.b);
    }
}

// The operator of one output interval by the eight-generator Lie-Trotter exponential (spin one,
// I:1810-1925), which is not unitary and has no SU(2) form: 3 x 3 products.
template <int INTEG, int FIELD>
SS_D Mat<3> interval_lt8(const MethodConfig& m, const FieldDesc& f, double t_c, double dt, double rw, int j0, int j1) {
    constexpr int L = 8;
    Mat<3> u;
    set_identity(u);
    TableCursor cur[L];  // per-channel table cursors for the increasing sample times of the steps
#pragma unroll
    for (int c = 0; c < L; c++) cur[c] = TableCursor{};
    const StepRule st = step_rule<INTEG>(t_c, dt);
    double t_fine = t_c;
    for (int j = 0; j < j0; j++) t_fine += dt;
    auto sample = [&](double* s, double off) {
#pragma unroll
        for (int k = 0; k < L; k++) s[k] = 0.0;
        const double tau = (t_fine + off) - t_c;
        c64 w = c64{1.0, 0.0};
        if (m.rotating) sincos(rw * tau, &w.im, &w.re);
        sample_field<FIELD, L>(f, tau + t_c, s, cur);
        if (m.rotating) transform_frame_lt8(s, rw, w);
    };
    for (int j = j0; j < j1; j++) {
        double s0[L], s1[L], g[L];
        sample(s0, st.off_a);
        if constexpr (INTEG != INTEG_EULER) sample(s1, st.off_b);
#pragma unroll
        for (int k = 0; k < L; k++) g[k] = INTEG == INTEG_CF4 ? st.c0 * s0[k] + st.c1 * s1[k] : st.c0 * s0[k];
        u = matmul(expo_lt8_one(g, m.hypercubes, m.precision), u);
        if constexpr (INTEG != INTEG_EULER) {
#pragma unroll
            for (int k = 0; k < L; k++) g[k] = INTEG == INTEG_CF4 ? st.c1 * s0[k] + st.c0 * s1[k] : st.c0 * s1[k];
            u = matmul(expo_lt8_one(g, m.hypercubes, m.precision), u);
        }
        t_fine += dt;
    }
    return u;
}

// Leave the rotating frame (I:839-852): the operator of an SU(2) pair, or a d x d operator.
template <int D>
SS_D void leave_frame(Su2p& v, double rw, double dt_out) {
    c64 w;  // spin one, whose representation doubles the phase: half of it
    sincos_small(rw * dt_out * (D == 2 ? 1.0 : 0.5), &w.im, &w.re);
    v.a = v.a * conj(w);
    v.b = v.b * w;
}

template <int D>
SS_D void leave_frame(Mat<D>& u, double rw, double dt_out) {
    c64 w;
    sincos(rw * dt_out, &w.im, &w.re);
    const c64 wc = conj(w);
#pragma unroll
    for (int k = 0; k < D; k++) {
        u.a[0][k] = u.a[0][k] * wc;
        u.a[D - 1][k] = u.a[D - 1][k] * w;
    }
}

SS_D void identity_of(Su2p& v) { v = su2p_identity(); }
template <int D>
SS_D void identity_of(Mat<D>& u) {
    set_identity(u);
}
template <int D>
SS_D Mat<D> operator_of(const Su2p& v) {
    return su2p_to_mat<D>(v);
}
template <int D>
SS_D Mat<D> operator_of(const Mat<D>& u) {
    return u;
}
SS_D Su2p shfl_down_operator(const Su2p& v, int s) { return shfl_down_su2p(v, s); }
template <int D>
SS_D Mat<D> shfl_down_operator(const Mat<D>& u, int s) {
    return shfl_down_mat(u, s);
}
SS_D Su2p later_times(const Su2p& later, const Su2p& v) { return su2p_mul(later, v); }
template <int D>
SS_D Mat<D> later_times(const Mat<D>& later, const Mat<D>& u) {
    return matmul(later, u);
}

// An interval's outputs, from its rotating-frame operator v: an SU(2) pair, or a d x d operator.  With
// product_out (a warp's 32 intervals are then one tile of the state scan) also the product of the warp's
// operators, in five shuffle rounds, which saves the scan a pass over U: 56 + 63 us of a launch of 400
// pulse trains (4.1e6 output steps).
template <int D, typename V>
SS_D void finish_interval(const MethodConfig& m, V v, double rw, double dt_out, bool writes, double t_c, int64_t index,
                          double* time_out, double* u_out, double* product_out) {
    if (!writes) identity_of(v);
    else if (m.rotating && rw != 0.0) leave_frame<D>(v, rw, dt_out);
    if (writes) {
        const Mat<D> u = operator_of<D>(v);
        time_out[index] = t_c;
        double2* dst = reinterpret_cast<double2*>(u_out) + index * (D * D);
#pragma unroll
        for (int i = 0; i < D; i++)
#pragma unroll
            for (int k = 0; k < D; k++) dst[i * D + k] = make_double2(u.a[i][k].re, u.a[i][k].im);
    }
    if (product_out == nullptr) return;
    const int lane = threadIdx.x & 31;
    // unrolled for the pairs (400 pulse trains 789 -> 777 us); 3 x 3 products would be most of a kernel's code
    constexpr int kUnroll = sizeof(V) == sizeof(Su2p) ? 5 : 1;
#pragma unroll kUnroll
    for (int s = 1; s < 32; s <<= 1) {
        const V later = shfl_down_operator(v, s);
        if ((lane & (2 * s - 1)) == 0) v = later_times(later, v);
    }
    if (lane == 0) {
        const Mat<D> u = operator_of<D>(v);
        double2* dst = reinterpret_cast<double2*>(product_out);
#pragma unroll
        for (int i = 0; i < D; i++)
#pragma unroll
            for (int k = 0; k < D; k++) dst[i * D + k] = make_double2(u.a[i][k].re, u.a[i][k].im);
    }
}

// Combine the lanes' partial products in step order: later steps multiply from the left.
template <typename V>
SS_D void combine_lanes(V& v, int lanes, int lane_in_group) {
    for (int s = 1; s < lanes; s <<= 1) {
        const V later = shfl_down_operator(v, s);
        if ((lane_in_group & (2 * s - 1)) == 0) v = later_times(later, v);
    }
}

// The end of an interval whose lanes hold SU(2) products p, or, where a step with a quadratic shift was met
// (spin one), 3 x 3 products u.  Every lane of the warp calls this.
template <int DIMS>
SS_D void finish_steps(const MethodConfig& m, int dim, const Su2d& p, Mat<3>& u, bool quadratic, int lanes,
                       int lane_in_group, double rw, double dt_out, bool writes, double t_c, int64_t index,
                       double* time_out, double* u_out, double* product_out) {
    Su2p pair = Su2p{c64{1.0 + p.am1.re, p.am1.im}, p.beta};
    if (DIMS != 2 && __any_sync(0xffffffffu, quadratic)) {
        if (!quadratic) u = su2p_to_mat<3>(pair);
        combine_lanes(u, lanes, lane_in_group);
        finish_interval<3>(m, u, rw, dt_out, writes, t_c, index, time_out, u_out, product_out);
        return;
    }
    combine_lanes(pair, lanes, lane_in_group);
    if (DIMS != 3 && dim == 2)
        finish_interval<2>(m, pair, rw, dt_out, writes, t_c, index, time_out, u_out, product_out);
    else if (DIMS != 2)
        finish_interval<3>(m, pair, rw, dt_out, writes, t_c, index, time_out, u_out, product_out);
}

// The product of an interval's steps: an SU(2) element p, or, where a step with a quadratic shift was met (spin
// one), the 3 x 3 operator u; FP32-bulk: the sum of |g|^2.
struct StepsResult {
    Su2d p;
    Mat<3> u;
    float nsq;
    bool quadratic;
};

// Steps j0 .. j1 - 1 of an interval, one after another.
template <int DIMS, int INTEG, bool LT_HALF, int FIELD>
SS_D StepsResult steps64(const MethodConfig& m, const FieldDesc& f, const StepRule& rule, double prw, int dim, int j0, int j1) {
    constexpr int L = LieDim<DIMS, EXPO_LIE_TROTTER>::value;
    const bool lie_trotter = dim == 3 || LT_HALF;
    Steps<L> st(rule);
    st.template begin<INTEG>(m, prw, j0, j1);
    StepsResult r;
    r.p = Su2d{c64{0.0, 0.0}, c64{0.0, 0.0}};
    r.quadratic = false;
    for (int j = j0; j < j1; j++) {
        Generators4 g;
        if (j != j0) st.template restart<INTEG>(j, j0);
        step_generators<FIELD, L, INTEG, true>(f, st, g.a, g.b);
        if constexpr (DIMS != 2) {
            if (dim == 3 && (g.a[3] != 0.0 || (INTEG != INTEG_EULER && g.b[3] != 0.0))) {
                r.quadratic = true;
                r.u = spin_one_quadratic_steps64<INTEG, FIELD>(
                    m, f, st, su2_to_spin_one(c64{1.0 + r.p.am1.re, r.p.am1.im}, r.p.beta), g, j0, j, j1);
                break;
            }
        }
        su2_apply64(r.p, su2_step_element64(m, lie_trotter, g.a));
        if constexpr (INTEG != INTEG_EULER) su2_apply64(r.p, su2_step_element64(m, lie_trotter, g.b));
    }
    return r;
}

// For table fields out of line, so that their cursors' registers are not the piecewise constant path's too.
template <int DIMS, int INTEG, bool LT_HALF, int FIELD>
__device__ __noinline__ StepsResult steps64_call(const MethodConfig& m, const FieldDesc& f, StepRule rule, double prw, int dim,
                                                 int j0, int j1) {
    return steps64<DIMS, INTEG, LT_HALF, FIELD>(m, f, rule, prw, dim, j0, j1);
}

// Evolve one output interval.  Every lane of the warp must call this (shuffles use the full mask);
// lanes with `active == false` do no steps and write nothing.
//
// Bound by the FP64 pipe.  The step's exponentials are SU(2) elements for both spins (su2_step_element64; spin one
// with a quadratic shift: spin_one_step64), its frame phasors come from a recurrence, and the fine
// steps' product is kept in SU(2) residual form: about 120 FP64 operations a step besides the field
// (600 with a quadratic shift), where the 3 x 3 squarings took over 5000.  Measured against that form,
// a launch of each: spin-one Rabi sweep of 6.4e6 steps 3157 -> 185 us, 4001 x 50 steps with a
// quadratic shift 149 -> 35 us, spin-half pulse ensemble of 2.05e8 steps 3832 -> 2880 us.
//
// DIMS 0: a mixed-spin batch.  The spin enters only the frame winding, the exponentiator and the stored
// operator, so both spins run one copy of the step loop.
template <int DIMS, int INTEG, int EXPO_H, int EXPO_O, int FIELD>
SS_D void interval64(const MethodConfig& m, const Instance& inst, const FieldDesc& f, int64_t index, bool active,
                     int lane_in_group, double* time_out, double* u_out, double* product_out) {
    constexpr int L = LieDim<DIMS, EXPO_O>::value;
    const int dim = DIMS != 0 ? DIMS : inst.dim;
    const int lanes = m.lanes;
    const double dt = inst.dt_int, dt_out = inst.dt_out;
    // I:818, rounded as the reference rounds it (no fused multiply-add), so time[] is bit-exact
    const double t_c = __dadd_rn(inst.t0, __dmul_rn(dt_out, (double)(inst.interval0 + index)));
    double prw = 0.0;  // Bz at the middle of the interval (I:823-829): P rw for either spin
    if (active && m.rotating) prw = sample_z<FIELD, L>(f, t_c + dt_out / 2);
    const double rw = dim == 2 ? prw / 2 : prw;
    const int K = active ? inst.n_fine : 0;
    const int j0 = (int)(((int64_t)K * lane_in_group) / lanes);
    const int j1 = (int)(((int64_t)K * (lane_in_group + 1)) / lanes);
    const bool writes = active && lane_in_group == 0;

    if constexpr (DIMS == 3 && EXPO_O == EXPO_LIE_TROTTER_8) {
        Mat<3> u = interval_lt8<INTEG, FIELD>(m, f, t_c, dt, rw, j0, j1);
        combine_lanes(u, lanes, lane_in_group);
        finish_interval<3>(m, u, rw, dt_out, writes, t_c, index, time_out, u_out, product_out);
    } else {
        constexpr bool kLieTrotterHalf = EXPO_H == EXPO_LIE_TROTTER;
        const StepRule rule = step_rule<INTEG>(t_c, dt);
        StepsResult r;
        if constexpr (FIELD == FIELD_TABLE) {
            r.p = Su2d{c64{0.0, 0.0}, c64{0.0, 0.0}};
            r.quadratic = false;
            auto element = [&](const double* ga, const double* gb, int) {
                const bool lie_trotter = dim == 3 || kLieTrotterHalf;
                Su2d e = su2_step_element64(m, lie_trotter, ga);
                if constexpr (INTEG != INTEG_EULER) su2_apply64(e, su2_step_element64(m, lie_trotter, gb));
                return e;
            };
            if (!hold_steps<INTEG>(f, dim, m.rotating && prw != 0.0, rule, j0, j1, dt_out, r.p, element))
                r = steps64_call<DIMS, INTEG, kLieTrotterHalf, FIELD>(m, f, rule, prw, dim, j0, j1);
        } else {
            r = steps64<DIMS, INTEG, kLieTrotterHalf, FIELD>(m, f, rule, prw, dim, j0, j1);
        }
        finish_steps<DIMS>(m, dim, r.p, r.u, r.quadratic, lanes, lane_in_group, rw, dt_out, writes, t_c, index, time_out,
                           u_out, product_out);
    }
}

}  // namespace spinsim
