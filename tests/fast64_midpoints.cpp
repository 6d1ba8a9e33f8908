// Quotients and square roots as near to the midpoint of two doubles as they come (so_fast64.cuh), against the
// IEEE operators, with seeds as far off as the hardware's may be.  Prints "name mismatches cases worst" (worst in
// units in the last place); built and run by tests/test_fast64_midpoints.py (no device).
//   a / b for 53-bit integers a, b: a 2^s - b X = k for an odd X (a midpoint) and a small odd k leaves the
//           quotient |k| / (b 2^s) from it; X = -k / b mod 2^s.  s = 53: a >= b, s = 54: a < b.
//   sqrt(X 2^m / 4) for a 53-bit integer X: r^2 = X 2^m + k for an odd r, a root of k = 1 mod 8 modulo 2^m
//           (found bit by bit), m = 54, 55.
#include <cmath>
#include <cstdio>
#include <random>

#include "so_fast64.cuh"
using namespace so;
typedef unsigned __int128 u128;

static std::mt19937_64 g(53);
static double off() { return 1.0 + (2.0 * ((double)(g() >> 11) * 0x1p-53) - 1.0) * 0x1p-19; }
static bool is53(u128 v) { return v >= (u128)1 << 52 && v < (u128)1 << 53; }

static long apart(double a, double b) { return std::labs((long)(dbits(a) - dbits(b))); }

static void quotients() {
    const uint64_t one = 1;
    long bad = 0, n = 0, worst = 0;
    for (int i = 0; i < 400000; ++i) {
        uint64_t b = (one << 52) | (g() & ((one << 52) - 1)) | 1;
        if (i % 4 == 0) b = (one << 53) - 3 - 2 * (g() % (one << (1 + g() % 40)));  // the top significands
        if (i % 4 == 1) b = (one << 52) + 1 + 2 * (g() % (one << (1 + g() % 40)));
        if (b == (one << 53) - 1) continue;  // the reciprocal's exception
        uint64_t inv = b;
        for (int j = 0; j < 6; ++j) inv *= 2 - b * inv;
        for (int k = -7; k <= 7; k += 2)
            for (int s = 53; s <= 54; ++s) {
                uint64_t X = ((uint64_t)(-(int64_t)k) * inv) & ((one << s) - 1);
                if (s == 53) X += one << 53;
                if (X < (one << 53)) continue;
                const u128 a = ((u128)b * X + (u128)(__int128)k) >> s;
                if (!is53(a)) continue;
                const double x = std::ldexp((double)(uint64_t)a, (int)(g() % 400) - 200);
                const double d = std::ldexp((double)b, (int)(g() % 400) - 200);
                const long e = apart(round_quot(x, d, near_rcp(d, off() / d)), x / d);
                bad += e != 0;
                worst = e > worst ? e : worst;
                ++n;
            }
    }
    std::printf("quotient %ld %ld %ld\n", bad, n, worst);
}

// fast_sqrt from a seed y0.
static double root(double x, double y0) {
    const double e = std::fma(-(x * y0), y0, 1.0);
    const double y = std::fma(y0 * e, std::fma(0.375, e, 0.5), y0);
    const double h = x * y;
    return std::fma(std::fma(-h, h, x), 0.5 * y, h);
}
static void roots() {
    long bad = 0, n = 0;
    for (int m = 54; m <= 55; ++m)
        for (long k = 1 - (1 << 14); k < 1 << 14; k += 8) {
            const u128 mask = ((u128)1 << m) - 1, K = (u128)(__int128)k;
            u128 s = 1;
            for (int b = 3; b < m; ++b)
                if (((s * s - K) >> b) & 1) s += (u128)1 << (b - 1);
            for (int q = 0; q < 4; ++q) {
                u128 r = ((q & 1 ? ~s + 1 : s) + (q & 2 ? (u128)1 << (m - 1) : 0)) & mask;
                if (r < (u128)1 << 53 || r >= (u128)1 << 54 || ((r * r - K) & mask) || !is53((r * r - K) >> m)) continue;
                for (int t = 0; t < 20; ++t, ++n) {
                    const double x = std::ldexp((double)(uint64_t)((r * r - K) >> m), m - 2 + 2 * ((int)(g() % 200) - 100));
                    bad += root(x, off() / std::sqrt(x)) != std::sqrt(x);
                    bad += fast_sqrt(x) != std::sqrt(x);
                }
            }
        }
    std::printf("sqrt %ld %ld 0\n", bad, n);
}

int main() {
    quotients();
    roots();
    return 0;
}
