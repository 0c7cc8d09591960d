// FP64 matrix exponentials of the reference (Utilities, spinsim/__init__.py:1528-1939), held in
// registers.  The same mathematical formulas as the reference, written so that each needs fewer
// transcendental calls: sin(x) = 2 sin(x/2) cos(x/2) from one sincos, a complex phase exp(i p)
// from (x + i y) / |x + i y| instead of atan2, and phase products by angle addition.  These
// rewrites change results only at the level of double rounding.
#pragma once
#include "common.cuh"

namespace spinsim {

constexpr double kSqrt2 = 1.4142135623730951;
constexpr double kSqrt3 = 1.7320508075688772;

// expm1i(x) = exp(i x) - 1 = -2 sin^2(x/2) + i sin(x)   (I:1557-1559)
SS_D c64 expm1i(double x) {
    double s, c;
    sincos(0.5 * x, &s, &c);
    return c64{-2.0 * (s * s), 2.0 * s * c};
}

// cos_exp_m1(c, e) = (expm1i(c + e) + expm1i(-c + e)) / 2 = cos(c) exp(i e) - 1   (I:1561-1563)
SS_D c64 cos_exp_m1(double c, double e) {
    const c64 a = expm1i(c + e), b = expm1i(-c + e);
    return c64{0.5 * (a.re + b.re), 0.5 * (a.im + b.im)};
}

// cos_m1(t) = cos(t) - 1 = -2 sin^2(t/2)   (I:1565-1567)
SS_D double cos_m1(double t) {
    const double s = sin(0.5 * t);
    return -2.0 * (s * s);
}

// ------------------------------------------------------------------ SU(2) elements
// Spin half, and spin one without a quadratic shift: every exponential of the reference is then an
// SU(2) element or its spin-one representation, and so are their products, so a step costs two
// SU(2) exponentials and products (about 35 FP64 operations each) whatever the spin.  Residual form:
// alpha = 1 + am1, U = [[alpha, -conj(beta)], [beta, conj(alpha)]].
struct Su2d {
    c64 am1, beta;
};

// Series coefficients of the step loops, in constant memory: a multiply-add then takes its coefficient as an
// operand, where a literal costs two moves into registers every time (the loops have no registers to
// keep them in).  Half the pulse ensemble's instructions were not FP64 ones.
static __constant__ double kCosHalf[6] = {-0.125, 1.0 / 384.0, -1.0 / 46080.0, 1.0 / 10321920.0, -1.0 / 3715891200.0,
                                          1.0 / 1961990553600.0};  // (-1)^k / ((2k)! 4^k), k = 1 ...
static __constant__ double kSinHalf[6] = {0.5, -1.0 / 48.0, 1.0 / 3840.0, -1.0 / 645120.0, 1.0 / 185794560.0,
                                          -1.0 / 81749606400.0};   // (-1)^k / (2 (2k+1)! 4^k), k = 0 ...
static __constant__ double kInvFact[16] = {1.0,
                                           1.0,
                                           1.0 / 2.0,
                                           1.0 / 6.0,
                                           1.0 / 24.0,
                                           1.0 / 120.0,
                                           1.0 / 720.0,
                                           1.0 / 5040.0,
                                           1.0 / 40320.0,
                                           1.0 / 362880.0,
                                           1.0 / 3628800.0,
                                           1.0 / 39916800.0,
                                           1.0 / 479001600.0,
                                           1.0 / 6227020800.0,
                                           1.0 / 87178291200.0,
                                           1.0 / 1307674368000.0};

// matrix_exponential_analytic (I:1618-1642): exp of -i(x Jx + y Jy + z Jz), minus one, with r2 = |(x, y, z)|^2:
// alpha - 1 = cos(r/2) - 1 - i z s, beta = (y - i x) s, s = sin(r/2) / r.  Even Taylor series for r <= 1/2 (the first
// omitted terms are below 2^-56 of the leading ones; no square root, division or argument reduction), else
// sincos.  Not a number: the identity, as the reference's "r > 0" test gives (I:1626).
SS_D Su2d su2_exp_m1(double x, double y, double z, double r2) {
    double c, s;
    if (r2 <= 0.25) {
        c = kCosHalf[5];
        s = kSinHalf[5];
#pragma unroll
        for (int k = 4; k >= 0; k--) {
            c = fma(c, r2, kCosHalf[k]);
            s = fma(s, r2, kSinHalf[k]);
        }
        c *= r2;
    } else if (r2 > 0.0) {
        const double r = sqrt(r2);
        double s4, c4;
        sincos(0.25 * r, &s4, &c4);
        c = -2.0 * (s4 * s4);
        s = 2.0 * s4 * c4 / r;
    } else {
        return Su2d{c64{0.0, 0.0}, c64{0.0, 0.0}};
    }
    return Su2d{c64{c, -z * s}, c64{y * s, -x * s}};
}

// matrix_exponential_lie_trotter (I:1644-1673; spin one without a quadratic shift I:1768-1808): the
// N-th power, N = 4^h, of e^{-i z Jz / 2N} e^{-i (x Jx + y Jy) / N} e^{-i z Jz / 2N}, minus one.  The
// factor is an SU(2) rotation by 2 theta, cos theta = cos A cos Z and sin theta (axis) =
// (sin A, cos A sin Z) with A = a / 2N, Z = z / 2N, so its N-th power is the rotation by 2 N theta.
// Out of line: the steps that need it are those too large for their N (su2_step_element64).
__attribute__((const)) inline __device__ __noinline__ Su2d su2_lie_trotter_m1(double x, double y, double z, double n) {
    const double a = sqrt(x * x + y * y);
    c64 ep = c64{1.0, 0.0};
    if (a > 0) {
        const double inv = 1.0 / a;
        ep = c64{x * inv, y * inv};
    }
    double sa, ca, sz, cz;
    sincos(0.5 * a / n, &sa, &ca);
    sincos(0.5 * z / n, &sz, &cz);
    const double cs = ca * sz;
    const double sn = sqrt(fma(cs, cs, sa * sa));
    double ratio = n, cm1 = 0.0;  // sin(N theta) / sin(theta), cos(N theta) - 1
    if (sn != 0.0) {
        const double half = 0.5 * (n * atan2(sn, ca * cz));
        double sh, ch;
        sincos(half, &sh, &ch);
        cm1 = -2.0 * (sh * sh);
        ratio = 2.0 * sh * ch / sn;
    }
    const double b = sa * ratio;
    return Su2d{c64{cm1, -cs * ratio}, c64{ep.im * b, -ep.re * b}};
}

// p <- (1 + e) p
SS_D void su2_apply64(Su2d& p, const Su2d& e) {
    const c64 alpha = c64{1.0 + p.am1.re, p.am1.im};
    const c64 beta = p.beta;
    // (alpha - 1) + e.am1 alpha - conj(e.beta) beta and beta + e.beta alpha + conj(e.am1) beta, each
    // part one chain of four FMAs
    const c64 a = e.am1, b = e.beta;
    c64 na, nb;
    na.re = fma(-a.im, alpha.im, fma(a.re, alpha.re, fma(-b.im, beta.im, fma(-b.re, beta.re, p.am1.re))));
    na.im = fma(a.im, alpha.re, fma(a.re, alpha.im, fma(b.im, beta.re, fma(-b.re, beta.im, p.am1.im))));
    nb.re = fma(-b.im, alpha.im, fma(b.re, alpha.re, fma(a.im, beta.im, fma(a.re, beta.re, beta.re))));
    nb.im = fma(b.im, alpha.re, fma(b.re, alpha.im, fma(-a.im, beta.re, fma(a.re, beta.im, beta.im))));
    p.am1 = na;
    p.beta = nb;
}

SS_D Su2d shfl_down_su2(const Su2d& v, int delta) {
    Su2d o;
    o.am1.re = __shfl_down_sync(0xffffffffu, v.am1.re, delta);
    o.am1.im = __shfl_down_sync(0xffffffffu, v.am1.im, delta);
    o.beta.re = __shfl_down_sync(0xffffffffu, v.beta.re, delta);
    o.beta.im = __shfl_down_sync(0xffffffffu, v.beta.im, delta);
    return o;
}

// p <- (1 + e)^n p by binary powers.
SS_D void su2_apply_power64(Su2d& p, Su2d e, int n) {
    for (;;) {
        if (n & 1) su2_apply64(p, e);
        n >>= 1;
        if (n == 0) return;
        const Su2d once = e;
        su2_apply64(e, once);
    }
}

// One exponential of a step's generator, minus one.  A Lie-Trotter
// exponential of N = 4^h factors differs from the exponential by less than |g|^3 / (8 N^2) (symmetric
// splitting), so for |g|^2 <= lt_norm2_max (|g|^3 <= 2^-53 N^2, |g| = 0.31 at the default 24
// squarings) the exponential itself is taken, and the N-th power's closed form beyond.
SS_D Su2d su2_step_element64(const MethodConfig& m, bool lie_trotter, const double* g) {
    const double r2 = fma(g[0], g[0], fma(g[1], g[1], g[2] * g[2]));
    if (!lie_trotter || r2 <= m.lt_norm2_max) return su2_exp_m1(g[0], g[1], g[2], r2);
    return su2_lie_trotter_m1(g[0], g[1], g[2], m.precision);
}

// ------------------------------------------------------------------ spin one
// matrix_exponential_lie_trotter for spin one (I:1768-1808); exp(i p) = (x + i y) / a replaces
// p = atan2(y, x).  The exponential minus one.
SS_D Mat<3> expo_lt_one_m1(const double* g, int hypercubes, double precision) {
    double a = sqrt(g[0] * g[0] + g[1] * g[1]);
    c64 ep = c64{1.0, 0.0};  // exp(i p)
    if (a > 0) {
        const double inv = 1.0 / a;
        ep = c64{g[0] * inv, g[1] * inv};
    }
    a = a / precision;
    double sh, ch;
    sincos(0.5 * a, &sh, &ch);
    const double Sa = sh;                                   // sin(a/2)
    const c64 sa = c64{0.0, -(2.0 * sh * ch) / kSqrt2};    // -i sin(a) / sqrt2
    const double z = g[2] / (2.0 * precision);
    const double q = g[3] / (6.0 * precision);
    double sz, cz, sq, cq;
    sincos(z, &sz, &cz);
    sincos(q, &sq, &cq);
    const c64 ez = c64{cz, sz}, eq = c64{cq, sq};
    const c64 epc = conj(ep), ezc = conj(ez), eqc = conj(eq);
    const double Sa2 = Sa * Sa;
    Mat<3> r;
    c64 cem = cos_exp_m1(0.5 * a, -z - q);
    r.a[0][0] = cem * (cem + c64{2.0, 0.0});
    r.a[1][0] = sa * ((eq * ep) * ezc);           // exp(i(q + p - z))
    r.a[2][0] = (-Sa2) * ((ep * ep) * (eqc * eqc));   // exp(2i(p - q))
    r.a[0][1] = sa * ((eq * epc) * ezc);          // exp(i(q - p - z))
    r.a[1][1] = cos_exp_m1(a, 4.0 * q);
    r.a[2][1] = sa * ((eq * ep) * ez);            // exp(i(q + p + z))
    r.a[0][2] = (-Sa2) * ((eq * eq) * (epc * epc));   // exp(2i(q - p))
    r.a[1][2] = sa * ((eq * epc) * ez);           // exp(i(q - p + z))
    cem = cos_exp_m1(0.5 * a, z - q);
    r.a[2][2] = cem * (cem + c64{2.0, 0.0});
#pragma unroll 1
    for (int h = 0; h < 2 * hypercubes; h++) r = square_m1(r);
    return r;
}

// exp(-i H) - 1 for H = x Jx + y Jy + z Jz + q Q, Q = diag(1, -2, 1) / 3 (spin one).  H is traceless,
// so H^3 = p H + d with p = tr(H^2) / 2 and d = det H, and every power of H is a real combination of
// 1, H and H^2 (Cayley-Hamilton): exp(-i H) - 1 = f0 + f1 H + f2 H^2 with the three complex
// coefficients from a real three-term recurrence summed with 1 / n!.  H has eigenvalues of modulus at
// most 2 sqrt(p / 3): for p <= 1/4 the series to n = 15 leaves less than 2^-56, for p <= 1/100 to n = 10
// (a warp takes the longer one when any lane needs it); larger generators are halved until p <= 1/4
// and the result is squared back (the residual squaring of I:1736-1748).  About 120 FP64 operations,
// against 108 for every one of the reference's squarings.
SS_D Mat<3> spin_one_exp_m1_64(double x, double y, double z, double q) {
    double a2 = fma(x, x, y * y);
    double p = fma(z, z, fma(q * q, 1.0 / 3.0, a2));
    int squarings = 0;
    while (p > 0.25 && squarings < 64) {
        x *= 0.5;
        y *= 0.5;
        z *= 0.5;
        q *= 0.5;
        a2 *= 0.25;
        p *= 0.25;
        squarings++;
    }
    const double d = (2.0 / 3.0) * q * (fma(z, z, -0.5 * a2) - q * q * (1.0 / 9.0));
    // (-i)^n / n! times the coefficients (al, be, ga) of H^n, summed into f0, f1, f2
    c64 f0 = c64{0.0, 0.0}, f1 = c64{0.0, -1.0}, f2 = c64{-0.5, 0.0};  // n = 1 and n = 2
    double al = 0.0, be = 0.0, ga = 1.0;                                 // of H^2
    auto term = [&](int n) {                                             // H^n = H H^(n-1)
        const double na = d * ga, nb = fma(p, ga, al), ng = be;
        al = na;
        be = nb;
        ga = ng;
        const double c = kInvFact[n];
        const bool plus = (n & 3) == 0 || (n & 3) == 3;
        if (n & 1) {  // (-i)^3 = i, (-i)^5 = -i
            f0.im = plus ? fma(c, al, f0.im) : fma(-c, al, f0.im);
            f1.im = plus ? fma(c, be, f1.im) : fma(-c, be, f1.im);
            f2.im = plus ? fma(c, ga, f2.im) : fma(-c, ga, f2.im);
        } else {
            f0.re = plus ? fma(c, al, f0.re) : fma(-c, al, f0.re);
            f1.re = plus ? fma(c, be, f1.re) : fma(-c, be, f1.re);
            f2.re = plus ? fma(c, ga, f2.re) : fma(-c, ga, f2.re);
        }
    };
#pragma unroll
    for (int n = 3; n <= 10; n++) term(n);
    if (p > 0.01)
#pragma unroll
        for (int n = 11; n <= 15; n++) term(n);
    constexpr double ir2 = 0.70710678118654752440;
    const double h0 = fma(q, 1.0 / 3.0, z), h1 = q * (-2.0 / 3.0), h2 = fma(q, 1.0 / 3.0, -z);
    const c64 w = c64{x * ir2, y * ir2};  // H[1][0] = H[2][1]
    const double w2 = 0.5 * a2;
    Mat<3> e;
    auto diagonal = [&](double h, double hh) { return c64{fma(f2.re, hh, fma(f1.re, h, f0.re)), fma(f2.im, hh, fma(f1.im, h, f0.im))}; };
    e.a[0][0] = diagonal(h0, fma(h0, h0, w2));
    e.a[1][1] = diagonal(h1, fma(h1, h1, 2.0 * w2));
    e.a[2][2] = diagonal(h2, fma(h2, h2, w2));
    const c64 lo = c64{fma(f2.re, h0 + h1, f1.re), fma(f2.im, h0 + h1, f1.im)};
    const c64 hi = c64{fma(f2.re, h1 + h2, f1.re), fma(f2.im, h1 + h2, f1.im)};
    const c64 ww = w * w;
    e.a[1][0] = w * lo;
    e.a[0][1] = conj(w) * lo;
    e.a[2][1] = w * hi;
    e.a[1][2] = conj(w) * hi;
    e.a[2][0] = ww * f2;
    e.a[0][2] = conj(ww) * f2;
    for (int k = 0; k < squarings; k++) e = square_m1(e);
    return e;
}

// u <- (1 + e) u, column by column in place
SS_D void spin_one_apply64(Mat<3>& u, const Mat<3>& e) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const c64 c0 = u.a[0][j], c1 = u.a[1][j], c2 = u.a[2][j];
#pragma unroll
        for (int i = 0; i < 3; i++)
            u.a[i][j] = cfma(e.a[i][2], c2, cfma(e.a[i][1], c1, cfma(e.a[i][0], c0, u.a[i][j])));
    }
}

// A step by the reference's squarings.  Out of line, the product by value: taken only by steps that are
// too large for their number of squarings, so its registers and stack stay out of the common loop.
inline __device__ __noinline__ Mat<3> spin_one_squarings_step64(Mat<3> u, double x, double y, double z, double q,
                                                               int hypercubes, double precision) {
    const double g[4] = {x, y, z, q};
    spin_one_apply64(u, expo_lt_one_m1(g, hypercubes, precision));
    return u;
}

// One exponential of a spin-one step with a quadratic shift (I:1768-1808), applied to the interval's
// product u.  As in su2_step_element64, the exponential itself where the Lie-Trotter product agrees with it to
// rounding (|g|^2 <= lt_norm2_max; the reversed sign of the shift in the factor's [0][2] phase is
// of the same order as the splitting's error, a^2 q / (6 N^2)), else the reference's squarings.
SS_D void spin_one_step64(const MethodConfig& m, Mat<3>& u, const double* g) {
    const double r2 = fma(g[0], g[0], fma(g[1], g[1], fma(g[2], g[2], g[3] * g[3])));
    if (r2 <= m.lt_norm2_max) spin_one_apply64(u, spin_one_exp_m1_64(g[0], g[1], g[2], g[3]));
    else u = spin_one_squarings_step64(u, g[0], g[1], g[2], g[3], m.hypercubes, m.precision);
}

// matrix_exponential_lie_trotter_8 (I:1810-1925).  As in the reference, the third block
// (generators 4, 5) reuses `sa` from the second block (generators 6, 7) when its amplitude is
// non-zero, and sets it to zero otherwise.
SS_D Mat<3> expo_lt8_one(const double* g, int hypercubes, double precision) {
    Mat<3> r, t1, t2;
    double a = sqrt(g[0] * g[0] + g[1] * g[1]);
    c64 ep, sa;
    double Sa, Cam1;
    if (a > 0) {
        ep = c64{g[0] / a, g[1] / a};
        a = a / precision;
        double sh, ch;
        sincos(0.5 * a, &sh, &ch);
        Sa = sh;
        sa = c64{0.0, -(2.0 * sh * ch) / kSqrt2};
        Cam1 = cos_m1(0.5 * a);
    } else {
        ep = c64{1.0, 0.0};
        Sa = 0;
        sa = c64{0.0, 0.0};
        Cam1 = 0;
    }
    {
        const c64 sep = Sa * ep, sepc = Sa * conj(ep);
        r.a[0][0] = c64{Cam1 * (Cam1 + 2), 0.0};
        r.a[1][0] = sa * ep;
        r.a[2][0] = (-1.0) * (sep * sep);
        r.a[0][1] = sa * conj(ep);
        r.a[1][1] = c64{cos_m1(a), 0.0};
        r.a[2][1] = sa * ep;
        r.a[0][2] = (-1.0) * (sepc * sepc);
        r.a[1][2] = sa * conj(ep);
        r.a[2][2] = c64{Cam1 * (Cam1 + 2), 0.0};
    }
    a = sqrt(g[6] * g[6] + g[7] * g[7]);
    if (a > 0) {
        ep = c64{g[6] / a, g[7] / a};
        a = a / precision;
        double sh, ch;
        sincos(0.5 * a, &sh, &ch);
        Sa = sh;
        sa = c64{0.0, -(2.0 * sh * ch) / kSqrt2};
        Cam1 = cos_m1(0.5 * a);
    } else {
        ep = c64{1.0, 0.0};
        Sa = 0;
        sa = c64{0.0, 0.0};
        Cam1 = 0;
    }
    {
        const c64 sep = Sa * ep, sepc = Sa * conj(ep);
        t1.a[0][0] = c64{Cam1 * (Cam1 + 2), 0.0};
        t1.a[1][0] = sa * ep;
        t1.a[2][0] = (-1.0) * (sep * sep);
        t1.a[0][1] = sa * conj(ep);
        t1.a[1][1] = c64{cos_m1(a), 0.0};
        t1.a[2][1] = (-1.0) * (sa * ep);
        t1.a[0][2] = (-1.0) * (sepc * sepc);
        t1.a[1][2] = (-1.0) * (sa * conj(ep));
        t1.a[2][2] = c64{Cam1 * (Cam1 + 2), 0.0};
    }
    t2 = multiply_m1(r, t1);
    a = sqrt(g[4] * g[4] + g[5] * g[5]);
    if (a > 0) {
        ep = c64{g[4] / a, g[5] / a};
        a = a / precision;
        Sa = sin(a);
        Cam1 = cos_m1(a);
    } else {
        ep = c64{1.0, 0.0};
        Sa = 0;
        sa = c64{0.0, 0.0};
        Cam1 = 0;
    }
    {
        const c64 sep = Sa * ep, sepc = Sa * conj(ep);
        const c64 zero = c64{0.0, 0.0};
        r.a[0][0] = c64{Cam1, 0.0};
        r.a[1][0] = zero;
        r.a[2][0] = (-1.0) * (sep * sep);
        r.a[0][1] = sa * conj(ep);
        r.a[1][1] = zero;
        r.a[2][1] = (-1.0) * (sa * ep);
        r.a[0][2] = (-1.0) * (sepc * sepc);
        r.a[1][2] = zero;
        r.a[2][2] = c64{Cam1, 0.0};
    }
    t1 = multiply_m1(r, t2);
    a = g[2] / precision;
    const double e = g[3] / (3.0 * precision);
    {
        const c64 zero = c64{0.0, 0.0};
        t2.a[0][0] = expm1i(-a - e);
        t2.a[1][0] = zero;
        t2.a[2][0] = zero;
        t2.a[0][1] = zero;
        t2.a[1][1] = expm1i(2.0 * e);
        t2.a[2][1] = zero;
        t2.a[0][2] = zero;
        t2.a[1][2] = zero;
        t2.a[2][2] = expm1i(a - e);
    }
    r = multiply_m1(t1, t2);
    for (int h = 0; h < hypercubes; h++) {
        r = square_m1(r);
        r = square_m1(r);
    }
    r.a[0][0].re += 1.0;
    r.a[1][1].re += 1.0;
    r.a[2][2].re += 1.0;
    return r;
}

}  // namespace spinsim
