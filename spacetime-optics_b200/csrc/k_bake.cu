// k_bake.cu -- bake of the reference flow's turbulence into the frame's 24 retarded-time slices.
//
// Reference: k_bake_turb (blackholes/src/render.cu:449-460), one thread per texel.  Slice k holds
// exp(a n - a^2 / 2) of the sheared noise n (emission.cuh:34-51: two noise generations of four
// octaves) at the retarded time t_ref(r) + delta_k, on cell centres phi = 2 pi (i + 1/2) / 512, ln R
// uniform over [lr0, lr1] (192 cells), z / R uniform over [-zmax, zmax] (48 cells).
//
// What bounds it is the integer pipe: a texel takes 8 lattice cells (2 generations x 4 octaves), each
// with the pcg hashes of its 8 corners, 64 hash chains and their gradients.  But along one row (fixed
// ln R, z / R and slice) the 512 values of phi walk a circle through each lattice, so neighbouring
// texels mostly stand in the same cell: of 32 consecutive texels about 2, 4, 6 and 12 cells per
// octave are distinct at the reference's scale.  Here a warp takes a row, 32 texels at a time: every lane
// finds its cells, a ballot per octave marks where a run of equal cells begins, and each lane then hashes one
// run's eight corners into gradient vectors in shared memory, which all the texels of the run read
// back.  About 24 of 128 cells are hashed per 32 texels and generation.  What depends on the row
// alone (radius, retarded time, shear, generation) is computed once per row, and the sine and cosine
// of phi come from a table turned by the row's shear angle.  113 M texels: 11.3 -> 6.2 ms on the B200
// (integer pipe 72 % -> 46 %, FMA pipe 39 %, issue 77 %).
//
// The float operations of a texel are those of the reference's noise in their order (its gradient is
// a sum of two signed components: the dot product with a vector of two +-1 and a 0 rounds the same).
// Compiled with -fmad=false: every fusion is explicit.
#include <cuda_runtime.h>

#include "so_emission.cuh"
#include "so_launch.h"

namespace so {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int BAKE_WARPS = 4;  // warps (rows) per CTA
constexpr int RUN_CAP = 64;    // runs of one generation's 32 texels that fit the table at once

struct RunTable {
    float4 cell[RUN_CAP];   // lattice cell (x, y, z as floats) and the octave's seed
    float4 grad[RUN_CAP][6];  // eight corner gradients (x fastest), 24 floats
};

// Gradient of lattice corner hash h: grad3's two signed components (so_emission.cuh) as a vector.
__device__ __forceinline__ void corner_grad(uint32_t h, float* g) {
    const uint32_t third = (h >> 2) * 0x55555556u;
    const float su = (h & 1u) ? -1.f : 1.f, sv = (h & 2u) ? -1.f : 1.f;
    g[0] = third < 0xAAAAAAAAu ? su : 0.f;
    g[1] = third < 0x55555555u ? sv : (third < 0xAAAAAAAAu ? 0.f : su);
    g[2] = third < 0x55555555u ? 0.f : sv;
}

// Hash of the table's runs [0, n): lane by lane, the corners in gnoise's nesting (z, then y, then x).
__device__ __forceinline__ void hash_runs(RunTable& T, int n) {
    for (int r = threadIdx.x & 31; r < n; r += 32) {
        const float4 c = T.cell[r];
        const int ix = (int)c.x, iy = (int)c.y, iz = (int)c.z;
        const uint32_t seed = __float_as_uint(c.w);
        float g[24];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t hz = pcg((uint32_t)(iz + k) * 83492791u ^ seed);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint32_t hy = pcg((uint32_t)(iy + j) * 19349663u ^ hz);
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    corner_grad(pcg((uint32_t)(ix + i) * 73856093u ^ hy), g + 3 * (4 * k + 2 * j + i));
            }
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) T.grad[r][q] = make_float4(g[4 * q], g[4 * q + 1], g[4 * q + 2], g[4 * q + 3]);
    }
}

__device__ __forceinline__ float fade(float u) { return u * u * u * (u * (u * 6.f - 15.f) + 10.f); }

// gnoise at (ux, uy, uz) inside a hashed cell.
__device__ __forceinline__ float cell_noise(const float4* __restrict__ gr, float ux, float uy, float uz) {
    float g[24];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const float4 v = gr[q];
        g[4 * q] = v.x;
        g[4 * q + 1] = v.y;
        g[4 * q + 2] = v.z;
        g[4 * q + 3] = v.w;
    }
    const float wx = fade(ux), wy = fade(uy), wz = fade(uz);
    const float vx[2] = {ux, ux - 1}, vy[2] = {uy, uy - 1}, vz[2] = {uz, uz - 1};
    float n[8];
#pragma unroll
    for (int c = 0; c < 8; ++c)
        n[c] = fmaf(g[3 * c], vx[c & 1], fmaf(g[3 * c + 1], vy[(c >> 1) & 1], g[3 * c + 2] * vz[c >> 2]));
    const float x00 = lerpf_(n[0], n[1], wx), x10 = lerpf_(n[2], n[3], wx);
    const float x01 = lerpf_(n[4], n[5], wx), x11 = lerpf_(n[6], n[7], wx);
    return lerpf_(lerpf_(x00, x10, wy), lerpf_(x01, x11, wy), wz);
}

}  // namespace

// One warp per row (j, l, k), grid-stride.  SURF: into slice k's 3-D array through its surface (x =
// phi, y = ln R, z = z / R), for the texture-unit fetch; else into plain memory, phi fastest.
template <bool SURF>
__global__ void __launch_bounds__(32 * BAKE_WARPS) k_bake_turb(const so_scene* __restrict__ Sp,
                                                               const so_frame* __restrict__ Fp, const TurbBake b,
                                                               float* __restrict__ field, const SurfaceSet surf) {
    __shared__ RunTable table[BAKE_WARPS];
    __shared__ double2 turn[TURB_NPHI];  // cos, sin of the cell centres phi
    for (int i = threadIdx.x; i < TURB_NPHI; i += blockDim.x) {
        double s, c;
        sincos((i + 0.5) / TURB_NPHI * 2.0 * PI, &s, &c);
        turn[i] = make_double2(c, s);
    }
    __syncthreads();
    const so_scene& S = *Sp;
    const so_frame& F = *Fp;
    const int lane = threadIdx.x & 31;
    RunTable& T = table[threadIdx.x >> 5];
    const float amp_t = S.flow_turb_amp, scale = S.flow_turb_scale, tcorr = S.flow_tcorr;
    const uint32_t seed = S.seed ^ 0x51f15eedu;
    const int nrows = TURB_NLR * TURB_NZ * TURB_NT, nwarps = gridDim.x * BAKE_WARPS;
    for (int row = blockIdx.x * BAKE_WARPS + (threadIdx.x >> 5); row < nrows; row += nwarps) {
        const int j = row % TURB_NLR, l = (row / TURB_NLR) % TURB_NZ, k = row / (TURB_NLR * TURB_NZ);
        const double R = exp(S.turb_lr0 + (j + 0.5) / TURB_NLR * (S.turb_lr1 - S.turb_lr0));
        const double z = (-1.0 + 2.0 * (l + 0.5) / TURB_NZ) * S.turb_zmax * R;
        const double r = sqrt(fma(R, R, z * z));
        const double t = (F.t - (F.r - r + 2.0 * log(F.r / r))) + b.delta[k];
        // sheared_noise at (R, phi, z, t): generation, blend, and per generation the shear angle
        const double Om = keplerian_omega(S.a, fmax(R, S.r_isco));
        const double P = 6.283185307179586 / Om * (double)tcorr;
        const double s = t / P;
        const double gen = floor(s);
        const float f = (float)(s - gen);
        const float inv = 1.f / (scale * (float)R), zz = (float)z * inv * 2.f;
        const float blend = 1.f / sqrtf((1.f - f) * (1.f - f) + f * f);
        double ca[2], sa[2];
#pragma unroll
        for (int g = 0; g < 2; ++g) sincos(Om * (t - (gen + g) * P), &sa[g], &ca[g]);
        for (int i0 = 0; i0 < TURB_NPHI; i0 += 32) {
            const double2 ph = turn[i0 + lane];
            float acc = 0.f;
#pragma unroll 1
            for (int g = 0; g < 2; ++g) {
                const double cg = g ? ca[1] : ca[0], sg = g ? sa[1] : sa[0];
                const double cp = fma(ph.x, cg, ph.y * sg), sp = fma(ph.y, cg, -(ph.x * sg));  // of phi - angle
                float x = (float)(R * cp) * inv, y = (float)(R * sp) * inv, zc = zz;
                const uint32_t gseed = seed + 7919u * (uint32_t)(long long)(gen + g);
                // cells of the four octaves; a run of equal cells along the lanes gets one entry
                float ux[4], uy[4], uz[4], fx[4], fy[4], fz[4];
                int run[4], total = 0;
                unsigned starts[4];
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    fx[o] = floorf(x);
                    fy[o] = floorf(y);
                    fz[o] = floorf(zc);
                    ux[o] = x - fx[o];
                    uy[o] = y - fy[o];
                    uz[o] = zc - fz[o];
                    const float qx = __shfl_up_sync(FULL, fx[o], 1), qy = __shfl_up_sync(FULL, fy[o], 1),
                                qz = __shfl_up_sync(FULL, fz[o], 1);
                    starts[o] = __ballot_sync(FULL, lane == 0 || qx != fx[o] || qy != fy[o] || qz != fz[o]);
                    run[o] = __popc(starts[o] << (31 - lane)) - 1;
                    total += __popc(starts[o]);
                    const float nx = 0.80f * x + 0.60f * zc, nz = -0.60f * x + 0.80f * zc;
                    x = nx * 2.03f;
                    y = y * 2.03f;
                    zc = nz * 2.03f;
                }
                // all four octaves' runs together where they fit the table (one hashing pass of the
                // lanes, rarely two), else octave by octave (at most 32 each)
                const bool together = total <= RUN_CAP;
                float noise[4];
#pragma unroll
                for (int o0 = 0; o0 < 4; ++o0) {
                    if (o0 > 0 && together) break;
                    int n = 0;
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        if (!together && o != o0) continue;
                        if ((starts[o] >> lane) & 1u)
                            T.cell[n + run[o]] = make_float4(fx[o], fy[o], fz[o],
                                                             __uint_as_float(gseed + 1013u * (uint32_t)o));
                        n += __popc(starts[o]);
                    }
                    __syncwarp();
                    hash_runs(T, n);
                    __syncwarp();
                    n = 0;
#pragma unroll
                    for (int o = 0; o < 4; ++o) {
                        if (!together && o != o0) continue;
                        noise[o] = cell_noise(T.grad[n + run[o]], ux[o], uy[o], uz[o]);
                        n += __popc(starts[o]);
                    }
                    __syncwarp();
                }
                float sum = 0.f, amp = 1.f, norm = 0.f;
#pragma unroll
                for (int o = 0; o < 4; ++o) {
                    sum += amp * noise[o];
                    norm += amp * amp;
                    amp *= 0.55f;
                }
                const float n4 = sum * 2.2f / sqrtf(norm);
                acc += (g == 0 ? 1.f - f : f) * n4;
            }
            const float v = __expf(amp_t * (acc * blend) - 0.5f * amp_t * amp_t);
            if (SURF) surf3Dwrite(v, surf.s[k], (i0 + lane) * (int)sizeof(float), j, l);
            else field[(size_t)row * TURB_NPHI + i0 + lane] = v;
        }
    }
}

namespace {
template <bool SURF>
cudaError_t go(const so_scene* d_scene, const so_frame* d_frame, const TurbBake& b, float* field,
               const SurfaceSet& surf, int num_sms, cudaStream_t st) {
    int per_sm = 1;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bake_turb<SURF>, 32 * BAKE_WARPS, 0);
    if (e != cudaSuccess) return e;
    k_bake_turb<SURF><<<num_sms * (per_sm > 0 ? per_sm : 1), 32 * BAKE_WARPS, 0, st>>>(d_scene, d_frame, b, field, surf);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_bake_turb(const so_scene* d_scene, const so_frame* d_frame, const TurbBake& b, float* field,
                             int num_sms, cudaStream_t st) {
    return go<false>(d_scene, d_frame, b, field, SurfaceSet{}, num_sms, st);
}

cudaError_t launch_bake_turb_surf(const so_scene* d_scene, const so_frame* d_frame, const TurbBake& b,
                                  const SurfaceSet& surf, int num_sms, cudaStream_t st) {
    return go<true>(d_scene, d_frame, b, nullptr, surf, num_sms, st);
}

}  // namespace so
