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

// Lie-algebra dimension of the field vector (I:547-554).
template <int D, int EXPO>
struct LieDim {
    static constexpr int value = (D == 2) ? 3 : (EXPO == EXPO_LIE_TROTTER_8 ? 8 : 4);
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

// Frame phasors restart from sincos after this many steps of their recurrence, so that their drift
// (about one rounding a step) stays far below the phase's own argument rounding.
constexpr int kPhasorSteps = 64;

// What a step loop's field samples need: the frame phasors exp(-i P rw tau) at the step's two samples
// and their rotation by one step, the interval's start and the step's number, the sample offsets and
// weights, and the table cursors.  A sample's time is t_c + tau with tau = j dt + offset, rounded once
// each: the reference's running sum of steps (I:836) agrees with it to its own rounding, and the frame's
// phase (at tau) stays consistent with the field's (at t_c + tau), whose common part cancels in the
// rotating frame.
template <int L>
struct Steps {
    c64 wa, wb, wrot;
    double rw, t_c, j, dt, off_a, off_b, c0, c1;
    bool rotating;
    TableCursor cur[L];

    SS_D double tau(double off) const { return fma(j, dt, off); }

    template <int P, int INTEG>
    SS_D void start_phasors() {
        sincos(-(double)P * rw * tau(off_a), &wa.im, &wa.re);
        if (INTEG != INTEG_EULER) sincos(-(double)P * rw * tau(off_b), &wb.im, &wb.re);
    }
    // Steps from number `first` of an interval that starts at t (steps: how many it has; 0: none).
    template <int P, int INTEG>
    SS_D void begin(const MethodConfig& m, double interval_rw, double t, int first, int steps) {
        rw = interval_rw;
        t_c = t;
        j = (double)first;
        rotating = m.rotating;
        wa = wb = wrot = c64{1.0, 0.0};
        if (m.rotating && steps > 0) {
            sincos(-(double)P * rw * dt, &wrot.im, &wrot.re);
            start_phasors<P, INTEG>();
        }
#pragma unroll
        for (int c = 0; c < L; c++) cur[c] = TableCursor{};  // for the increasing sample times of the steps
    }
    // Before the samples of step n of a lane that began at step n0: the phasors from sincos every
    // kPhasorSteps steps.
    template <int P, int INTEG>
    SS_D void restart(int n, int n0) {
        if (rotating && (n - n0) % kPhasorSteps == 0) start_phasors<P, INTEG>();
    }
};

// One step's field samples (FP64) -> frame transform -> the integrator's generators (FP64); the
// step number and the frame phasors move on.
template <int FIELD, int L, int P, int INTEG>
SS_D void step_generators(const FieldDesc& f, Steps<L>& st, double* ga, double* gb) {
    double s0[8], s1[8];  // a user field writes all eight channels
#pragma unroll
    for (int k = 0; k < 8; k++) {
        s0[k] = 0.0;
        s1[k] = 0.0;
    }
    sample_field<FIELD, L>(f, st.t_c + st.tau(st.off_a), s0, st.cur);
    if (INTEG != INTEG_EULER) sample_field<FIELD, L>(f, st.t_c + st.tau(st.off_b), s1, st.cur);
    st.j += 1.0;
    if (st.rotating) {  // xy times exp(-i P rw tau), z minus P rw
        const c64 xa = c64{s0[0], s0[1]} * st.wa;
        s0[0] = xa.re;
        s0[1] = xa.im;
        s0[2] -= (double)P * st.rw;
        st.wa = st.wa * st.wrot;
        if (INTEG != INTEG_EULER) {
            const c64 xb = c64{s1[0], s1[1]} * st.wb;
            s1[0] = xb.re;
            s1[1] = xb.im;
            s1[2] -= (double)P * st.rw;
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

// The reference's sample offsets and weights of an integrator for steps of dt (I:624-686 Magnus CF4 at
// the two Gauss points, I:693-752 Heun at the step's ends, I:759-791 Euler at its middle).
template <int INTEG, int L>
SS_D void set_integrator(Steps<L>& st, double dt) {
    const double a_lo = 0.5 * dt * (1.0 - 1.0 / kSqrt3);
    const double a_hi = 0.5 * dt * (1.0 + 1.0 / kSqrt3);
    const double w0 = (1.5 + kSqrt3) / 6.0, w1 = (1.5 - kSqrt3) / 6.0;
    st.dt = dt;
    st.off_a = INTEG == INTEG_CF4 ? a_lo : INTEG == INTEG_HEUN ? 0.0 : 0.5 * dt;
    st.off_b = INTEG == INTEG_CF4 ? a_hi : dt;
    st.c0 = INTEG == INTEG_CF4 ? dt * w0 : INTEG == INTEG_HEUN ? 0.5 * dt : dt;
    st.c1 = INTEG == INTEG_CF4 ? dt * w1 : 0.0;
}

// Steps j .. j1 - 1 of a spin-one interval whose quadratic shift is non-zero: full 3 x 3 exponentials
// and products, from the product u of the steps before.  On entry step j's generators are in g and st is at
// step j + 1.  Out of line, its state passed by value, so that the registers of the common
// SU(2) loop are allocated without this path's.
template <int INTEG, int FIELD>
__device__ __noinline__ Mat<3> spin_one_quadratic_steps64(const MethodConfig& m, const FieldDesc& f, Steps<4> st,
                                                          Mat<3> u, Generators4 g, int j0, int j, int j1) {
    for (;;) {
        spin_one_step64(m, u, g.a);
        if constexpr (INTEG != INTEG_EULER) spin_one_step64(m, u, g.b);
        if (++j >= j1) return u;
        st.template restart<1, INTEG>(j, j0);
        step_generators<FIELD, 4, 1, INTEG>(f, st, g.a, g.b);
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
    Steps<L> st;
    set_integrator<INTEG>(st, dt);
    st.j = (double)j0;
    auto sample = [&](double* s, double off) {
#pragma unroll
        for (int k = 0; k < L; k++) s[k] = 0.0;
        const double tau = st.tau(off);
        c64 w = c64{1.0, 0.0};
        if (m.rotating) sincos(rw * tau, &w.im, &w.re);
        sample_field<FIELD, L>(f, t_c + tau, s, cur);
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
        st.j += 1.0;
    }
    return u;
}

// Evolve one output interval.  Every lane of the warp must call this (shuffles use the full mask);
// lanes with `active == false` do no steps and write nothing.
//
// Bound by the FP64 pipe.  The step's exponentials are SU(2) elements for both spins (su2_step64; spin one
// with a quadratic shift: spin_one_step64), its frame phasors come from a recurrence, and the fine
// steps' product is kept in SU(2) residual form: about 120 FP64 operations a step besides the field
// (600 with a quadratic shift), where the 3 x 3 squarings took over 5000.  Measured against that form,
// a launch of each: spin-one Rabi sweep of 6.4e6 steps 3157 -> 185 us, 4001 x 50 steps with a
// quadratic shift 149 -> 35 us, spin-half pulse ensemble of 2.05e8 steps 3832 -> 2880 us.
template <int D, int INTEG, int EXPO, int FIELD>
SS_D void interval64(const MethodConfig& m, const Instance& inst, const FieldDesc& f, int64_t index, bool active,
                     int lane_in_group, double* time_out, double* u_out) {
    constexpr int L = LieDim<D, EXPO>::value;
    constexpr int P = (D == 2) ? 2 : 1;  // power of the frame winding in the xy transform (I:599-613)
    const int lanes = m.lanes;
    const double dt = inst.dt_int, dt_out = inst.dt_out;
    // I:818, rounded as the reference rounds it (no fused multiply-add), so time[] is bit-exact
    const double t_c = __dadd_rn(inst.t0, __dmul_rn(dt_out, (double)(inst.interval0 + index)));
    double rw = 0.0;
    if (active && m.rotating) {  // I:823-829
        double s[8];
#pragma unroll
        for (int k = 0; k < 8; k++) s[k] = 0.0;
        sample_field<FIELD, L>(f, t_c + dt_out / 2, s);
        rw = s[2];
        if (D == 2) rw /= 2;
    }
    const int K = active ? inst.n_fine : 0;
    const int j0 = (int)(((int64_t)K * lane_in_group) / lanes);
    const int j1 = (int)(((int64_t)K * (lane_in_group + 1)) / lanes);

    Mat<D> u;
    if constexpr (EXPO == EXPO_LIE_TROTTER_8) {
        u = interval_lt8<INTEG, FIELD>(m, f, t_c, dt, rw, j0, j1);
        for (int s = 1; s < lanes; s <<= 1) {  // later steps multiply from the left
            const Mat<D> later = shfl_down_mat(u, s);
            if ((lane_in_group & (2 * s - 1)) == 0) u = matmul(later, u);
        }
    } else {
        Steps<L> st;
        set_integrator<INTEG>(st, dt);
        st.template begin<P, INTEG>(m, rw, t_c, j0, K);
        Su2d p = Su2d{c64{0.0, 0.0}, c64{0.0, 0.0}};
        bool quadratic = false;  // a step with a quadratic shift was met: the product is in u
        for (int j = j0; j < j1; j++) {
            Generators4 g;
            if (j != j0) st.template restart<P, INTEG>(j, j0);
            step_generators<FIELD, L, P, INTEG>(f, st, g.a, g.b);
            if constexpr (D == 3) {
                if (g.a[3] != 0.0 || (INTEG != INTEG_EULER && g.b[3] != 0.0)) {
                    quadratic = true;
                    u = spin_one_quadratic_steps64<INTEG, FIELD>(
                        m, f, st, su2_to_spin_one(c64{1.0 + p.am1.re, p.am1.im}, p.beta), g, j0, j, j1);
                    break;
                }
            }
            su2_step64<EXPO>(m, p, g.a);
            if constexpr (INTEG != INTEG_EULER) su2_step64<EXPO>(m, p, g.b);
        }
        // Combine the lanes' partial products in step order: later steps multiply from the left.
        if (D == 2 || !__any_sync(0xffffffffu, quadratic)) {
            for (int s = 1; s < lanes; s <<= 1) {
                const Su2d later = shfl_down_su2(p, s);
                if ((lane_in_group & (2 * s - 1)) == 0) su2_apply64(p, later);
            }
            u = su2p_to_mat<D>(Su2p{c64{1.0 + p.am1.re, p.am1.im}, p.beta});
        } else {
            if (!quadratic) u = su2p_to_mat<D>(Su2p{c64{1.0 + p.am1.re, p.am1.im}, p.beta});
            for (int s = 1; s < lanes; s <<= 1) {
                const Mat<D> later = shfl_down_mat(u, s);
                if ((lane_in_group & (2 * s - 1)) == 0) u = matmul(later, u);
            }
        }
    }
    if (!active || lane_in_group != 0) return;

    if (m.rotating) {  // leave the rotating frame, I:839-852
        c64 wo;
        sincos(rw * dt_out, &wo.im, &wo.re);
        const c64 woc = conj(wo);
#pragma unroll
        for (int k = 0; k < D; k++) {
            u.a[0][k] = u.a[0][k] * woc;
            u.a[D - 1][k] = u.a[D - 1][k] * wo;
        }
    }
    time_out[index] = t_c;
    double2* dst = reinterpret_cast<double2*>(u_out) + index * (D * D);
#pragma unroll
    for (int i = 0; i < D; i++)
#pragma unroll
        for (int k = 0; k < D; k++) dst[i * D + k] = make_double2(u.a[i][k].re, u.a[i][k].im);
}

}  // namespace spinsim
