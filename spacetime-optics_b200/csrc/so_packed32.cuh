// so_packed32.cuh -- FP32 arithmetic two values at a time (fma / add / mul / sub .f32x2 of sm_100): one
// issue slot for two operations, each rounded as the scalar one.
#pragma once
#include <cuda_runtime.h>

namespace so {

struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 both(float a) { return pack2(a, a); }
__device__ __forceinline__ void unpack2(F2 x, float* a, float* b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(*a), "=f"(*b) : "l"(x.v));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

// cos(2 pi t) of two phases in turns, |t| < 2^21, on the FMA pipe: cos_turns (so_kerr.cuh) in FP32.  The nearest
// half turn q/2 is read off 2t + 1.5 * 2^23 (parity in the low mantissa bit), g = t - q/2 is exact, and
// cos(2 pi g), |g| <= 1/4, is a polynomial of degree 4 in g^2 (Chebyshev fit, fit_cos_turns.py: 4.7e-8, with
// coefficients rounded to FP32 1.1e-7, evaluated in FP32 1.9e-7).
__device__ __forceinline__ F2 cos_turns2(F2 t) {
    const F2 s = fma2(t, both(2.f), both(12582912.f));
    const F2 q = add2(s, both(-12582912.f));
    const F2 g = fma2(q, both(-0.5f), t);
    const F2 z = mul2(g, g);
    F2 p = both(0x1.c1e8dcp+5f);
    p = fma2(p, z, both(-0x1.54f5a0p+6f));
    p = fma2(p, z, both(0x1.03bd00p+6f));
    p = fma2(p, z, both(-0x1.3bd3a6p+4f));
    p = fma2(p, z, both(0x1.fffffep-1f));
    float a, b, sa, sb;
    unpack2(p, &a, &b);
    unpack2(s, &sa, &sb);
    return pack2(__int_as_float(__float_as_int(a) ^ (__float_as_int(sa) << 31)),
                 __int_as_float(__float_as_int(b) ^ (__float_as_int(sb) << 31)));
}

// FP32 turbulence sums acc += sum_m a_m cos(k_m . X + p_m) at 2 NP positions (pairs), the modes from
// constant memory.  The SFU's cosine bounds it (16 a clock per SM); the phases and the accumulation are
// packed, which halves their issue slots, and the slots that frees let every TURB_POLY-th mode
// (its k and p folded to turns by turb_modes_fold) take its cosine on the FMA pipe instead.  Which
// modes do is fixed, so a position's sum depends on the position alone.  Measured with 87 M positions and
// 512 modes: scalar 3.64 T cosines/s, packed 4.15, packed with every 8th (16th) mode on the FMA pipe
// 4.51 (4.54), every 6th 4.47; error against 64 bits 1.21e-5 -> 1.14e-5 of the sums' norm (the phase's
// rounding; the FMA-pipe cosine is the more exact one).  k_turb_records on the 2048^2 synchrotron frame:
// 133.7 -> 121.2 ms, SFU pipe 87 %, FMA pipe 73 % (4.6 T cosines/s).
template <int NP>
__device__ __forceinline__ void mode_sums2(const TurbModes& M, const F2* x, const F2* y, const F2* z, F2* acc) {
    const int nm = M.n, grouped = M.grouped;
    auto phase = [&](const float4& k, int q) {
        return fma2(both(k.z), z[q], fma2(both(k.y), y[q], fma2(both(k.x), x[q], both(k.w))));
    };
    auto sfu = [&](int m) {
        const float4 k = M.k[m];
        const F2 am = both(M.a[m]);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            float a, b;
            unpack2(phase(k, q), &a, &b);
            acc[q] = fma2(am, pack2(__cosf(a), __cosf(b)), acc[q]);
        }
    };
    int m = 0;
#pragma unroll 1
    for (; m + TURB_POLY <= grouped; m += TURB_POLY) {
#pragma unroll
        for (int j = 0; j < TURB_POLY - 1; ++j) sfu(m + j);
        const float4 k = M.k[m + TURB_POLY - 1];
        const F2 am = both(M.a[m + TURB_POLY - 1]);
#pragma unroll
        for (int q = 0; q < NP; ++q) acc[q] = fma2(am, cos_turns2(phase(k, q)), acc[q]);
    }
#pragma unroll 1
    for (; m < nm; ++m) sfu(m);
}

}  // namespace so
