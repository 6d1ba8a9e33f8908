// so_fast64.cuh -- branch-free FP64 division, square root and swept angle for the geodesic integrator,
// and the Dormand-Prince attempt built on them.
//
// What bounds the FP64 tracer is the dependent chain of one attempt, and with many rays the issue of its
// instructions: 920 per attempt of a vacuum ray with the IEEE operators, 45 % of them on the FP64 pipe (ncu,
// 65,536 rays).  Every `/` and sqrt() is a range test, a branch and a call behind it, so the scheduler
// cannot overlap the two quotients of a right-hand side, nor the five of the error norm, and the code of
// all of them does not fit the instruction cache.  Here they are straight-line (640, 58 %):
//   1/d, a/b   a 20-bit hardware seed, one third-order (Halley) step to within an ulp, then
//              Markstein's correction q + y (a - b q) with the residual exact in one fma (P. Markstein,
//              "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J.
//              R&D 34, 1990);
//   sqrt       the same with the residual x - g^2.
// How they round, with operands and results in the normal range:
//   1/d        to nearest, but for the one significand that is all ones (an ulp there);
//   sqrt       to nearest, also for the operands whose roots lie nearest to a midpoint of two doubles;
//   a/b        within an ulp.  Markstein's theorem wants y rounded to nearest, and y is good to an ulp: of
//              quotients made to lie next to a midpoint (within 2^-50 ulp of it) one in two hundred goes
//              the wrong way, of random ones none in some millions.  Rounding y first mends that for two
//              more fma a quotient, which cost the thin-disk frame 2.9 %, the FP64 flow frame 1.2 %.
// (tests/fast64_midpoints.cpp, tests/fast64_check.cpp; the device's own: tests/test_gpu_quick_arithmetic.py.)
// The integrator takes the steps of the IEEE form, bit for bit in every test, unless such a quotient or a
// near tie of the error norm (dp54_fast) comes up; that moves one error or derivative by an ulp.  dp54_fast
// looks at its result once, and an attempt with an out-of-range operand anywhere (a pole, a diverging trial
// step) is taken again by dp54.
//
// Measured on the B200, IEEE operators against this form, results identical: 65,536 vacuum rays
// 4.11 -> 3.28 ms, 1,021 of them (the longest ray's chain) 2.08 -> 1.54 ms, 262,144 rays through the
// reference flow 24.7 -> 17.9 ms, the 1280 x 720 x 2 disk frame 30.0 -> 22.6 ms.
#pragma once
#include "so_kerr.cuh"

namespace so {

// Seeds of 1/d and 1/sqrt(x), relative error below 2^-19: the hardware's approximations on the
// device, a rounded quotient cut to 20 bits on the host (the host form serves the checks).
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ double seed_rcp(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    return y;
}
__device__ __forceinline__ double seed_rsqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
#else
inline double seed_rcp(double d) { return bitsd(dbits(1.0 / d) & 0xffffffff00000000ull); }
inline double seed_rsqrt(double x) { return bitsd(dbits(1.0 / std::sqrt(x)) & 0xffffffff00000000ull); }
#endif

// 1/d to within an ulp from a seed y0: with e = 1 - d y0, y0 (1 + e + e^2) leaves e^3 < 2^-57.
SO_HD double near_rcp(double d, double y0) {
    const double e = fma(-d, y0, 1.0);
    return fma(y0, fma(e, e, e), y0);
}
// 1/d rounded to nearest, a/b within an ulp and nearly always to nearest (y: near_rcp of the divisor; see above).
SO_HD double round_rcp(double d, double y) { return fma(y, fma(-d, y, 1.0), y); }
SO_HD double round_quot(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}
SO_HD double fast_rcp(double d) { return round_rcp(d, near_rcp(d, seed_rcp(d))); }
SO_HD double fast_div(double a, double b) { return round_quot(a, b, near_rcp(b, seed_rcp(b))); }

// sqrt(x), x = 0 or normal.  With e = 1 - x y0^2, y0 (1 + e/2 + 3 e^2 / 8) is 1/sqrt(x) to within an
// ulp; g = x y is then corrected by its exact residual.
SO_HD double fast_sqrt(double x) {
    const double y0 = seed_rsqrt(x);
    const double e = fma(-(x * y0), y0, 1.0);
    const double y = fma(y0 * e, fma(0.375, e, 0.5), y0);
    const double g = x * y;
    const double s = fma(fma(-g, g, x), 0.5 * y, g);
    return x > 0.0 ? s : 0.0;
}

// sin(theta) = sqrt(max(1 - u^2, 0)) (0 for a NaN, as fmax gives it); 1 - u^2 in one rounding is 0 or
// at least 2^-106.
SO_HD double sin_of(double u) {
    const double t = fma(-u, u, 1.0);
    return fast_sqrt(t > 0.0 ? t : 0.0);
}

// rhs() with the two quotients above.  A Delta or sin^2 outside the normal range makes d[4] infinite
// or NaN.  1 - u^2 in one rounding is at most 0 or at least 2^-53, so the sign of its high word
// is the test against 1e-300 (a NaN goes through to d[4]).  Without TIME the coordinate time is left out (d[5] = 0): nothing depends
// on it but the emission.
template <bool TIME = true>
SO_HD void rhs_fast(const RayC& c, const double* y, double* d) {
    double r = y[0], u = y[2];
    double r2 = r * r;
    double Delta = fma(r, r - 2.0, c.A2);
    double P = fma(r, r, c.CP);
    d[0] = y[1];
    d[1] = fma(2.0 * r, P, -((r - 1.0) * c.K));
    d[2] = y[3];
    double u2 = u * u;
    d[3] = u * fma(c.A2, fma(-2.0, u2, 1.0), -c.Q3);
    double s2 = 1.0 - u2;
    s2 = (int)(dbits(s2) >> 32) > 0 ? s2 : 1e-300;
    double iD = fast_rcp(Delta);
    d[4] = c.a - fma(c.a * P, iD, fast_div(c.lam, s2));
    d[5] = TIME ? -fma((r2 + c.A2) * P, iD, c.a * fma(-c.a, s2, c.lam)) : 0.0;
}

// The Dormand-Prince coefficients as constant-bank operands: as literals each use costs two moves (a
// 64-bit immediate does not fit an instruction).
struct Tableau {
    double a21, a31, a32, a41, a42, a43, a51, a52, a53, a54, a61, a62, a63, a64, a65, b1, b3, b4, b5, b6, e1, e3, e4, e5, e6, e7;
};
#define SO_TABLEAU_VALUES {A21, A31, A32, A41, A42, A43, A51, A52, A53, A54, A61, A62, A63, A64, A65, B1, B3, B4, B5, B6, E1, E3, E4, E5, E6, E7}
#if defined(__CUDACC__)
static __constant__ Tableau dp_tableau = SO_TABLEAU_VALUES;
#endif
#if defined(__CUDA_ARCH__)
#define SO_TABLEAU(T) const Tableau& T = dp_tableau
#else
#define SO_TABLEAU(T) static const Tableau T = SO_TABLEAU_VALUES
#endif

// dp54() in this arithmetic; *ok says whether every operand stayed in range (else the result is
// not to be used).  The error norm is the largest of five quotients |e_i| / sc_i.  Rounding is
// monotone, so it is the rounded quotient of the largest ratio, found by comparing products; the two
// constant denominators tol and 4 tol share one candidate (the factor 4 is exact).  The products are
// rounded too: of two ratios within 2^-52 of each other the smaller may be taken, and the error be an ulp
// below dp54's.  A NaN candidate is passed over, as fmax does.  Four divisions fewer.
template <bool TIME = true>
SO_HD double dp54_fast(const RayC& c, const double* y, const double* k1, double h, double tol, double* yo,
                       double* k7, bool* ok) {
    SO_TABLEAU(T);
    double k2[6], k3[6], k4[6], k5[6], k6[6], t[6];
    t[4] = y[4];
    t[5] = y[5];
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = fma(h, T.a21 * k1[i], y[i]);
    rhs_fast<TIME>(c, t, k2);  // (the phi and t components of k2 enter nothing)
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = fma(h, fma(T.a32, k2[i], T.a31 * k1[i]), y[i]);
    rhs_fast<TIME>(c, t, k3);
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = fma(h, fma(T.a43, k3[i], fma(T.a42, k2[i], T.a41 * k1[i])), y[i]);
    rhs_fast<TIME>(c, t, k4);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        t[i] = fma(h, fma(T.a54, k4[i], fma(T.a53, k3[i], fma(T.a52, k2[i], T.a51 * k1[i]))), y[i]);
    rhs_fast<TIME>(c, t, k5);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        t[i] = fma(h, fma(T.a65, k5[i], fma(T.a64, k4[i], fma(T.a63, k3[i], fma(T.a62, k2[i], T.a61 * k1[i])))), y[i]);
    rhs_fast<TIME>(c, t, k6);
#pragma unroll
    for (int i = 0; i < (TIME ? 6 : 5); ++i)
        yo[i] = fma(h, fma(T.b6, k6[i], fma(T.b5, k5[i], fma(T.b4, k4[i], fma(T.b3, k3[i], T.b1 * k1[i])))), y[i]);
    if (!TIME) yo[5] = y[5];
    rhs_fast<TIME>(c, yo, k7);
    double e[5];
#pragma unroll
    for (int i = 0; i < 5; ++i)
        e[i] = fabs(h * fma(T.e7, k7[i], fma(T.e6, k6[i], fma(T.e5, k5[i], fma(T.e4, k4[i], fma(T.e3, k3[i], T.e1 * k1[i]))))));
    const double a0 = fabs(y[0]), b0 = fabs(yo[0]), a1 = fabs(y[1]), b1 = fabs(yo[1]);
    const double a3 = fabs(y[3]), b3 = fabs(yo[3]), rr = y[0] * y[0];
    double m1 = b1 > a1 ? b1 : a1;
    m1 = rr > m1 ? rr : m1;
    double m3 = b3 > a3 ? b3 : a3;
    m3 = m3 > 1.0 ? m3 : 1.0;
    const double sc0 = tol * (1e-6 + (b0 > a0 ? b0 : a0));
    const double sc1 = tol * (1e-6 + m1);
    const double sc3 = tol * m3;
    double num = e[2] > 0.0 ? e[2] : 0.0, den = tol;
    const double e4 = 0.25 * e[4];
    num = e4 > num ? e4 : num;
    const bool t0 = e[0] * den > num * sc0;
    num = t0 ? e[0] : num;
    den = t0 ? sc0 : den;
    const bool t1 = e[1] * den > num * sc1;
    num = t1 ? e[1] : num;
    den = t1 ? sc1 : den;
    const bool t3 = e[3] * den > num * sc3;
    num = t3 ? e[3] : num;
    den = t3 ? sc3 : den;
    const double err = fast_div(num, den);
    *ok = err < 1e300 && e[4] < 1e300;
    return err;
}

#if defined(__CUDACC__)
// The attempt again with the IEEE operators, out of line (through memory, so that the caller's state
// stays in registers).
static __device__ __noinline__ double dp54_again(const RayC* c, const double* yk, double h, double tol, double* yo) {
    return dp54(*c, yk, yk + 6, h, tol, yo, yo + 6);
}
// dp54() through the fast form.
template <bool TIME>
__device__ __forceinline__ double dp54_attempt(const RayC& c, const double* y, const double* k1, double h, double tol,
                                               double* yo, double* k7) {
    bool ok;
    double err = dp54_fast<TIME>(c, y, k1, h, tol, yo, k7, &ok);
    if (!ok) {
        double yk[12], out[12];
        const RayC cc = c;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            yk[i] = y[i];
            yk[6 + i] = k1[i];
        }
        err = dp54_again(&cc, yk, h, tol, out);
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            yo[i] = out[i];
            k7[i] = out[6 + i];
        }
    }
    return err;
}
#endif

// rpow5() for 1e-30 <= x <= 1 (the same operations; the exponent is never positive there), and
// accept_step() with it: the growth factor 0.9 err^-0.2 is at least 0.9, so only its upper limit binds.
SO_HD double rpow5_small(double x) {
    const uint64_t b = dbits(x);
    const int n = 1023 - (int)(b >> 52);  // -e
    const double m = bitsd((b & 0x000fffffffffffffULL) | 0x3ff0000000000000ULL);
    const int nq = (int)((unsigned)(n + 4) / 5u);  // -q
    const int r = 5 * nq - n;
    double y = fma(fma(0.05174, m, -0.28294), m, 1.23011);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double y2 = y * y;
        const double y5 = (y2 * y2) * y;
        y = fma(y * 0.2, fma(-m, y5, 1.0), y);
    }
    const double c = r == 0 ? 1.0 : r == 1 ? 0.8705505632961241 : r == 2 ? 0.757858283255199
                   : r == 3 ? 0.6597539553864471 : 0.5743491774985175;
    y = y * c;
    return y * bitsd((uint64_t)(1023 + nq) << 52);
}
SO_HD double accept_step_fast(double hc, double err) {
    const double f = 0.9 * rpow5_small(err > 1e-30 ? err : 1e-30);
    return hc * (f < 5.0 ? f : 5.0);
}

// project_radial() with fast_sqrt (R > r^4 / 4 there).
SO_HD void project_radial_fast(const RayC& c, double* y, double* k) {
    const double r = y[0];
    const double R = radial_pot(c, r);
    const double r2 = r * r;
    if (R > 0.25 * (r2 * r2)) {
        const double v = fast_sqrt(R);
        y[1] = y[1] < 0.0 ? -v : v;
        k[0] = y[1];
    }
}

// Angle of a long step, by the cross and dot products of the two directions.
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
inline
#endif
    double
    long_angle(double u0, double s0, double u1, double s1, double dphi) {
    const double sn = sin(dphi), cs = cos(dphi);
    const double cx = -(u0 * s1) * sn, cy = fma(u0, s1 * cs, -(s0 * u1)), cz = (s0 * s1) * sn;
    return atan2(sqrt(fma(cz, cz, fma(cy, cy, cx * cx))), fma(u0, u1, s0 * s1 * cs));
}

// Angle between the directions (u0, s0) and (u1, s1) (cosine and sine of the polar angle) whose
// azimuths differ by dphi, from the chord: w = (u1-u0)^2 + (s1-s0)^2 + 4 s0 s1 sin^2(dphi/2), angle
// 2 asin(sqrt(w)/2).  dphi/2 is reduced to |g| <= pi/2 (the square does not care for the sign), sin(g)/g
// is a polynomial of degree 7 in g^2 and the angle sqrt(w) times one of degree 9 in w for w <= 1/2
// (minimax fits, relative error 2e-16 and 6e-17: fit_swept_angle.py); a longer step (or a NaN) goes
// to long_angle.
SO_HD double swept_angle(double u0, double s0, double u1, double s1, double dphi) {
    const double magic = 6755399441055744.0;  // 1.5 * 2^52
    const double x = 0.5 * dphi;
    const double q = fma(x, 0x1.45f306dc9c883p-2, magic) - magic;
    double g = fma(-q, 0x1.921fb54442d18p+1, x);
    g = fma(-q, 0x1.1a62633145c07p-53, g);
    const double z = g * g;
    double p = -0x1.9f23bce07d610p-41;
    p = fma(p, z, 0x1.60e724daf2361p-33);
    p = fma(p, z, -0x1.ae63577964c39p-26);
    p = fma(p, z, 0x1.71de38085d206p-19);
    p = fma(p, z, -0x1.a01a019a53600p-13);
    p = fma(p, z, 0x1.1111111109f1cp-7);
    p = fma(p, z, -0x1.555555555547fp-3);
    p = fma(p, z, 0x1.fffffffffffffp-1);
    const double sn = g * p;
    const double du = u1 - u0, ds = s1 - s0;
    const double w = fma(4.0 * (s0 * s1), sn * sn, fma(ds, ds, du * du));
    if (!(w <= 0.5)) return long_angle(u0, s0, u1, s1, dphi);
    double a = 0x1.18ce9eb9bb012p-24;
    a = fma(a, w, 0x1.3366a4ef8bc52p-23);
    a = fma(a, w, 0x1.d49864b02c10ep-21);
    a = fma(a, w, 0x1.1bcdfdec88914p-18);
    a = fma(a, w, 0x1.6e92da456e5c5p-16);
    a = fma(a, w, 0x1.f1c6ddd11a5bbp-14);
    a = fma(a, w, 0x1.6db6dc0928801p-11);
    a = fma(a, w, 0x1.333333326fdf6p-8);
    a = fma(a, w, 0x1.5555555555b45p-5);
    a = fma(a, w, 1.0);
    return fast_sqrt(w) * a;
}

}  // namespace so
