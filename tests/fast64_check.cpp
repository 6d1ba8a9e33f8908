// Host check of so_fast64.cuh (branch-free division, square root, swept angle, Dormand-Prince attempt)
// against the IEEE operators and dp54(), with seeds as far off as the hardware's may be.  Prints
// "name mismatches cases worst"; built and run by tests/test_fast64.py (no device).
#include <cmath>
#include <cstdio>
#include <random>

#include "so_fast64.cuh"
using namespace so;

static std::mt19937_64 g(20240611);
static double uni() { return (double)(g() >> 11) * 0x1p-53; }
static double any(int emax) {  // random significand, exponent in [-emax, emax]
    return bitsd((g() & 0xfffffffffffffull) | ((uint64_t)(1023 + (int)(g() % (2 * emax + 1)) - emax) << 52));
}
static double off() { return 1.0 + (2.0 * uni() - 1.0) * 0x1p-19; }  // a seed's relative error

static void arithmetic() {
    long bad[3] = {0, 0, 0}, n = 3000000;
    for (long i = 0; i < n; ++i) {
        double a = any(300), b = any(300);
        if (i % 5 == 0) b = bitsd(dbits(b) & 0xfffffff000000000ull);       // short significands
        if (i % 7 == 0) a = b * (double)(1 + g() % 1000);                  // quotients near whole numbers
        if (i % 11 == 0) b = bitsd(dbits(b) | 0x000ffffffffff000ull) - 0.0;  // just under a power of two
        if ((dbits(b) & 0xfffffffffffffull) == 0xfffffffffffffull) continue;  // the documented exception
        if (i % 13 == 0) b = 1e-300, a = 40.0 * uni() - 20.0;              // the pole's sin^2
        const double y = near_rcp(b, off() / b);
        bad[0] += round_rcp(b, y) != 1.0 / b;
        bad[1] += round_quot(a, b, y) != a / b;
        const double x = i % 3 ? any(200) : uni() * uni();
        bad[2] += fast_sqrt(x) != std::sqrt(x);
    }
    bad[1] += round_quot(0.0, 3.0, near_rcp(3.0, 1.0 / 3.0)) != 0.0;
    bad[2] += fast_sqrt(0.0) != 0.0 || sin_of(1.0) != 0.0 || sin_of(-1.0) != 0.0 || sin_of(std::nan("")) != 0.0;
    std::printf("rcp %ld %ld 0\ndiv %ld %ld 0\nsqrt %ld %ld 0\n", bad[0], n, bad[1], n, bad[2], n);
}

static void controller() {
    long bad = 0, n = 400000;
    for (long i = 0; i < n; ++i) {
        const double err = i == 0 ? 1.0 : i == 1 ? 0.0 : i == 2 ? 1e-30 : i < 120 ? std::ldexp(1.0, -(int)i + 3) : std::pow(10.0, -33.0 * uni());
        if (err <= 1.0) bad += accept_step(0.7, err) != accept_step_fast(0.7, err);
    }
    std::printf("accept %ld %ld 0\n", bad, n);
}

static void angles() {
    double worst = 0.0;
    long n = 400000;
    for (long i = 0; i < n; ++i) {
        const double th = std::acos(1.0 - 2.0 * uni()), p0 = 50.0 * uni() - 25.0;
        const double far = i % 4 ? 0.3 : 6.0;
        const double t1 = th + (uni() - 0.5) * far, p1 = p0 + (uni() - 0.5) * (i % 4 ? 0.4 : 40.0);
        const double u0 = std::cos(th), u1 = std::cos(t1);
        const double dp = p1 - p0;  // what the function is given
        const long double A = u0, B = u1, S = sqrtl(1 - A * A), T = sqrtl(1 - B * B), D = dp;
        const long double x1 = T * cosl(D), y1 = T * sinl(D);
        const long double cx = -A * y1, cy = A * x1 - S * B, cz = S * y1;
        const long double want = atan2l(sqrtl(cx * cx + cy * cy + cz * cz), S * x1 + A * B);
        const double e = std::fabs((double)(swept_angle(u0, sin_of(u0), u1, sin_of(u1), dp) - want));
        if (e > worst) worst = e;
    }
    std::printf("angle 0 %ld %.3g\n", n, worst);
    const double same = swept_angle(0.3, sin_of(0.3), 0.3, sin_of(0.3), 0.0);
    std::printf("still %d 1 0\nnan %d 1 0\n", same != 0.0, swept_angle(0.3, 0.9, 0.3, 0.9, std::nan("")) == 0.0);
}

// Whole rays by both attempts: every error and state equal, bit for bit, wherever dp54_fast says ok.
static void rays() {
    long steps = 0, bad = 0, notok = 0, polenotok = 0;
    const double spins[] = {1e-6, 0.5, 0.94, 0.9999}, incls[] = {0.5, 17.0, 90.0, 163.0};
    for (double a : spins)
        for (double inc : incls)
            for (int k = 0; k < 24; ++k) {
                so_kerr_point kp;
                kerr_point(a, 1000.0, inc * PI / 180.0, &kp);
                const double al = 16.0 * uni() - 8.0, be = 16.0 * uni() - 8.0;
                const double nx = -1.0, ny = -be / 1000.0, nz = al / 1000.0, il = 1.0 / std::sqrt(nx * nx + ny * ny + nz * nz);
                RayC c;
                double y[6], k1[6], yn[6], k7[6], ym[6], k8[6];
                camera_photon(a, kp, 0.3, 0.0, {nx * il, ny * il, nz * il}, {0.0, 0.0, 0.0}, c, y);
                rhs(c, y, k1);
                double h = initial_step(y);
                const double rs = horizon_radius(a) * 1.000001;
                for (int it = 0; it < 4000; ++it, ++steps) {
                    bool ok;
                    const double err = dp54(c, y, k1, h, 1e-10, yn, k7), e2 = dp54_fast(c, y, k1, h, 1e-10, ym, k8, &ok);
                    if (!ok) ++notok;
                    else {
                        bad += err != e2;
                        for (int i = 0; i < 6; ++i) bad += yn[i] != ym[i] || k7[i] != k8[i];
                    }
                    if (!(err <= 1.0)) {
                        h = reject_step(h, err);
                        continue;
                    }
                    double ka[6];
                    for (int i = 0; i < 6; ++i) {
                        y[i] = ym[i] = yn[i];
                        k1[i] = ka[i] = k7[i];
                    }
                    project_radial(c, y, k1);
                    project_radial_fast(c, ym, ka);
                    for (int i = 0; i < 6; ++i) bad += y[i] != ym[i] || k1[i] != ka[i];
                    h = accept_step(h, err);
                    if (y[0] < rs || (y[0] > 1000.0 && y[1] > 0.0)) break;
                }
            }
    // an overflowing quotient (u past the pole) and a NaN: the fast form must say so
    {
        RayC c;
        ray_consts(c, 0.5, 1e-3, 3.0, 1.0);
        double y[6] = {50.0, -2400.0, 2.0, 0.0, 0.0, 0.0}, k1[6], yn[6], k7[6];
        rhs(c, y, k1);
        c.lam = 1e9;  // lam over 1e-300
        bool ok = true;
        dp54_fast(c, y, k1, 1e-4, 1e-10, yn, k7, &ok);
        polenotok += !ok;
        double bad_y[6] = {50.0, -2400.0, 0.3, std::nan(""), 0.0, 0.0};
        dp54_fast(c, bad_y, k1, 1e-4, 0.0, yn, k7, &ok);  // tolerance 0: no finite error
        polenotok += !ok;
    }
    std::printf("attempts %ld %ld 0\nnotok %ld %ld 0\nflagged %ld 2 0\n", bad, steps, notok, steps, 2 - polenotok);
}

int main() {
    arithmetic();
    controller();
    angles();
    rays();
    return 0;
}
