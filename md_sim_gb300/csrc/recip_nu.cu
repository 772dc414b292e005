// recip_nu.cu - reciprocal-space Ewald sum of the mixed form by gridding (force_fouri,
// src/forcem.f90:827-937): the same sum over the same k vectors as the direct form, with the atoms
// spread onto a grid of M >= 2 (2K + 1) points per box edge by a Kaiser-Bessel window, separable
// discrete Fourier sums between the grid and the 2K + 1 frequencies per direction, and the window's
// transform divided out (nonuniform FFT of types 1 and 2: Dutt and Rokhlin 1993; the window and its
// piecewise polynomials as in Barnett, Magland and af Klinteberg 2019).  The work per atom is that
// of 8^3 grid points instead of one product per k vector.
//
//   S(k) = sum_j q_j e^{ik.r_j} ~ [sum_g G(g) e^{i 2 pi k.g/M}] / phi^(k),
//   G(g) = sum_j q_j phi(g - r_j M/L), phi(t) = prod_d I0(b sqrt(1 - (t_d/4)^2)) / I0(b), |t_d| < 4
//   f_j  = -q_j grad Phi(r_j),  Phi(r) = Re sum_k C(k) e^{ik.r},  C = Ak conj(S + S_wall),
//          Phi on the grid from C / phi^, between grid points by the window, its gradient by the
//          window's derivative.
// With b = 6 pi the window and its aliases leave a relative error of about 1e-6 in the reciprocal
// forces (1e-7 in S(k)); everything between the fixed-point positions and C(k) is FP32, C(k) and
// the energies are FP64 as in the direct form.
//
// The packing of the atom records (pack.cuh) also drops each moving atom's index into the bucket of
// its block of 8 x 8 x 8 cells.  Then, all on one stream:
//   k_nu_spread  two warps per block (more CTAs where blocks hold many atoms): the block's 15 x 15 x 15
//                points in shared memory, each warp the columns of one x parity, one of an atom's 64
//                (x, y) columns and 8 z per lane, then added to the grid with red.v4
//   k_nu_zy      one CTA per (x plane, group of n): sums over z (real input, n >= 0), then over y
//   k_nu_x       one CTA per (n, group of m): sums over x, S(k), energies, C(k), back over l
//   k_nu_yz      one CTA per (x plane, group of y): back over m, then over n to the real Phi
//   k_nu_force   one CTA per block: its 15 x 15 x 15 points of Phi in shared memory, half a warp per atom
// The Fourier sums fold p and M - p (and the frequencies k and -k), which leaves a quarter of the
// multiply-adds of the plain complex sums: 95 M FMAs forward and back at M = 104.
//
// 98,304 atoms, 29,038 k vectors (M = 104): spread 32 us, zy 12, x 13, yz 11, force 30 = 98 us where the
// tensor-core passes take 310 (143 + 11 + 5 + 156); resident step 0.496 -> 0.276 ms, forces of the
// whole evaluation 6.2e-7 off FP64 (tensor cores 1.1e-6), reciprocal energy 2e-7 (1.9e-6).  Spread and
// force are bound by shared-memory wavefronts (79 and 82 % of the L1 pipe), the Fourier sums by them
// and by the few CTAs.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "ctx.h"

namespace mdg {

namespace {

constexpr int kW = 8;       // window width in grid points
constexpr int kDeg = 9;     // degree of the window's polynomial on each unit interval (error 7e-8)
constexpr int kStage = 10;  // atoms a warp prepares at a time (3 lanes each)
constexpr int kPX = 260, kPY = 17;  // pitches of a block's points: 4 x (of one parity) times 8 y hit 32 banks
constexpr int kTile = 15 * kPX;     // x, y from 3 cells below the block, z from 4 (quads aligned to 4)
constexpr int kSplit = 64;  // atoms of a block that one more CTA is given for

// weight of point k (0..7) for an atom at fraction t of its cell: sum_i c[k][i] s^i, s = 2t - 1
struct NuPoly {
    float c[kW][kDeg + 1];
};

__device__ __forceinline__ int wrap(int g, int M) { return g < 0 ? g + M : g >= M ? g - M : g; }

__device__ __forceinline__ void red4(float* p, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// cell (0..M-1) and fraction of a fixed-point coordinate
__device__ __forceinline__ int cell_of(uint32_t u, int M, float& t) {
    const unsigned long long g = (unsigned long long)u * (unsigned)M;
    t = (float)(uint32_t)g * 2.3283064365386963e-10f;  // 2^-32
    return (int)(g >> 32);
}

// The weights w[0..7] (and their derivatives by t) at fraction t.
template <bool GRAD>
__device__ __forceinline__ void weights(const NuPoly& P, float t, float* w, float* dw) {
    const float s = 2.0f * t - 1.0f;
#pragma unroll
    for (int k = 0; k < kW; ++k) {
        float a = P.c[k][kDeg], d = 0.f;
#pragma unroll
        for (int i = kDeg - 1; i >= 0; --i) {
            if (GRAD) d = fmaf(d, s, a);
            a = fmaf(a, s, P.c[k][i]);
        }
        w[k] = a;
        if (GRAD) dw[k] = 2.0f * d;
    }
}

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(float2* dst, const float2* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Offset of an atom's first point in its block's tile: x, y from 3 below the atom's cell, z likewise
// (the tile's z starts 4 below the block).
__device__ __forceinline__ int tile_off(int fx, int fy, int fz) { return fx * kPX + fy * kPY + fz + 1; }

__global__ void __launch_bounds__(64) k_nu_spread(NuView g, const uint4* __restrict__ atoms, const __grid_constant__ NuPoly P) {
    __shared__ __align__(16) float tile[kTile];
    __shared__ __align__(16) float wts[2 * kStage][3][kW];
    __shared__ int off[2 * kStage];
    const int t64 = threadIdx.x, lane = t64 & 31, warp = t64 >> 5, nblk = g.nblk;
    if (blockIdx.x == nblk) {
        // atoms whose block's bucket was full: straight to the grid
        const int n = *g.novf;
        for (int i = 2 * blockIdx.y + warp; i < n; i += 2 * gridDim.y) {
            const uint4 r = atoms[g.ovf[i]];
            float t[3], w[3][kW];
            const int c0 = cell_of(r.x, g.M[0], t[0]), c1 = cell_of(r.y, g.M[1], t[1]), c2 = cell_of(r.z, g.M[2], t[2]);
#pragma unroll
            for (int d = 0; d < 3; ++d) weights<false>(P, t[d], w[d], nullptr);
            for (int e = lane; e < kW * kW; e += 32) {
                const int x = wrap(c0 - 3 + e / kW, g.M[0]), y = wrap(c1 - 3 + e % kW, g.M[1]);
                float wx = 0.f, wy = 0.f;
#pragma unroll
                for (int k = 0; k < kW; ++k) {
                    wx = k == e / kW ? w[0][k] : wx;
                    wy = k == e % kW ? w[1][k] : wy;
                }
                const float v = __uint_as_float(r.w) * wx * wy;
#pragma unroll
                for (int k = 0; k < kW; ++k)
                    atomicAdd(&g.grid[((size_t)x * g.M[1] + y) * g.M[2] + wrap(c2 - 3 + k, g.M[2])], v * w[2][k]);
            }
        }
        return;
    }
    const int n = min(g.cnt[blockIdx.x], g.cap);
    const int i0 = (int)((long)n * blockIdx.y / gridDim.y), i1 = (int)((long)n * (blockIdx.y + 1) / gridDim.y);
    if (i0 >= i1) return;
    const int* bucket = g.bucket + (size_t)blockIdx.x * g.cap;
    // warp w adds to the columns whose x in the tile has parity w: 4 x times 8 y of each atom's 64
    const int si = warp * kStage + lane / 3, sd = lane % 3, xh = lane >> 3, y = lane & 7;
    const bool stager = lane < 3 * kStage;
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    if (stager && i0 + si < i1) r = atoms[bucket[i0 + si]];
    for (int e = t64; e < kTile / 4; e += 64) reinterpret_cast<float4*>(tile)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int b0 = i0; b0 < i1; b0 += 2 * kStage) {
        const int nb = min(2 * kStage, i1 - b0);
        float t, w[kW];
        const int f = cell_of(sd == 0 ? r.x : sd == 1 ? r.y : r.z, g.M[sd], t) & 7;
        weights<false>(P, t, w, nullptr);
        const float q = sd == 0 ? __uint_as_float(r.w) : 1.0f;
        const int fy = __shfl_down_sync(0xffffffffu, f, 1), fz = __shfl_down_sync(0xffffffffu, f, 2);
        if (b0 > i0) __syncthreads();
        if (stager && si < nb) {
            float4* o = reinterpret_cast<float4*>(wts[si][sd]);
            o[0] = make_float4(q * w[0], q * w[1], q * w[2], q * w[3]);
            o[1] = make_float4(q * w[4], q * w[5], q * w[6], q * w[7]);
            if (sd == 0) off[si] = tile_off(f, fy, fz) | f << 16;
        }
        // the next atoms' records load while these are added
        if (stager && b0 + 2 * kStage + si < i1) r = atoms[bucket[b0 + 2 * kStage + si]];
        __syncthreads();
        for (int a = 0; a < nb; ++a) {
            const float(*wa)[kW] = wts[a];
            const int o = off[a], kx = 2 * xh + ((warp ^ (o >> 16)) & 1);
            const float4 za = *reinterpret_cast<const float4*>(wa[2]), zb = *reinterpret_cast<const float4*>(wa[2] + 4);
            const float zw[8] = {za.x, za.y, za.z, za.w, zb.x, zb.y, zb.z, zb.w};
            const float v = wa[0][kx] * wa[1][y];
            float* p = tile + (o & 0xffff) + kx * kPX + y * kPY;
            float s[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) s[k] = p[k];
#pragma unroll
            for (int k = 0; k < 8; ++k) p[k] = fmaf(v, zw[k], s[k]);
            __syncwarp();
        }
    }
    __syncthreads();
    const int bz = blockIdx.x % g.n8[2], by = (blockIdx.x / g.n8[2]) % g.n8[1], bx = blockIdx.x / (g.n8[2] * g.n8[1]);
    #pragma unroll 5
    for (int e = t64; e < 900; e += 64) {
        const int Q = e & 3, X = (e >> 2) / 15, Y = (e >> 2) % 15;
        const float* s = tile + X * kPX + Y * kPY + 4 * Q;
        const int gx = wrap(8 * bx - 3 + X, g.M[0]), gy = wrap(8 * by - 3 + Y, g.M[1]), gz = wrap(8 * bz - 4 + 4 * Q, g.M[2]);
        if (s[0] != 0.f || s[1] != 0.f || s[2] != 0.f || s[3] != 0.f)
            red4(&g.grid[((size_t)gx * g.M[1] + gy) * g.M[2] + gz], s[0], s[1], s[2], s[3]);
    }
}

// ---- Fourier sums ------------------------------------------------------------------------------
// Twiddle tables of a direction: tw[p * (K + 1) + k] and twt[k * (M/2 + 1) + p], both
// (cos, sin)(2 pi k p / M) for p = 0..M/2, k = 0..K.
constexpr int kNGrp = 8;    // most n of one k_nu_zy CTA
constexpr int kMGrp = 8;    // most m of one k_nu_x CTA
constexpr int kYRows = 128; // most y rows staged at a time in k_nu_zy

__device__ __forceinline__ int odd(int n) { return n | 1; }

// A folded pair of terms: (a + b, a - b), or (a, 0) for a term that is its own partner.
__device__ __forceinline__ float4 fold(float2 a, float2 b, bool own) {
    return own ? make_float4(a.x, a.y, 0.f, 0.f) : make_float4(a.x + b.x, a.y + b.y, a.x - b.x, a.y - b.y);
}

// Two folded Fourier sums with one set of twiddles: u = sum e cos, v = sum o sin (complex each);
// u + i v is the sum at the twiddles' frequency (or point), u - i v the one at its negative.
struct Sum2 {
    float2 u[2], v[2];
    __device__ __forceinline__ void run(const float4* __restrict__ a, const float4* __restrict__ b,
                                        const float2* __restrict__ w, int wstride, int n) {
        u[0] = u[1] = v[0] = v[1] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int p = 0; p < n; ++p) {
            const float2 c = w[p * wstride];
            const float4 x = a[p], y = b[p];
            u[0].x = fmaf(x.x, c.x, u[0].x);
            u[0].y = fmaf(x.y, c.x, u[0].y);
            v[0].x = fmaf(x.z, c.y, v[0].x);
            v[0].y = fmaf(x.w, c.y, v[0].y);
            u[1].x = fmaf(y.x, c.x, u[1].x);
            u[1].y = fmaf(y.y, c.x, u[1].y);
            v[1].x = fmaf(y.z, c.y, v[1].x);
            v[1].y = fmaf(y.w, c.y, v[1].y);
        }
    }
    __device__ __forceinline__ float2 plus(int k) const { return make_float2(u[k].x - v[k].y, u[k].y + v[k].x); }
    __device__ __forceinline__ float2 minus(int k) const { return make_float2(u[k].x + v[k].y, u[k].y - v[k].x); }
};

// Sum over z then y of one x plane: H[n][x][m] for n = n0..n0 + nn - 1 (nn <= 8), m = -KM..KM.
// Staged rows are Mz + 4 apart (16-byte rows; 8 of them on different banks).
__global__ void __launch_bounds__(256) k_nu_zy(NuView g) {
    extern __shared__ __align__(16) float sm[];
    const int My = g.M[1], Mz = g.M[2], hz = Mz / 2, hy = My / 2, KM = g.K[1];
    const int x = blockIdx.x, n0 = blockIdx.y * g.ngrp, nn = min(g.ngrp, g.K[2] + 1 - n0);
    const int t = threadIdx.x, pitch = Mz + 4, rb = min(My, g.yrows);
    // z twiddles (hz + 1) x 8 cos | sin, A[n][y], y twiddles [y][m], then the staged rows
    float* cs = sm;
    float2* A = reinterpret_cast<float2*>(cs + (hz + 1) * 2 * kNGrp);
    float2* ty = A + kNGrp * My;
    float* rows = reinterpret_cast<float*>(ty) + ((2 * (hy + 1) * (KM + 1) + 3) & ~3);
    const int q4 = Mz / 4;
    auto stage = [&](int y0, int ny) {
        const float* src = g.grid + ((size_t)x * My + y0) * Mz;
        for (int e = t; e < ny * q4; e += 256) cp_async16(rows + (e / q4) * pitch + 4 * (e % q4), src + 4 * e);
    };
    stage(0, rb);
    for (int e = t; e < (hy + 1) * (KM + 1); e += 256) cp_async8(ty + e, g.tw[1] + e);
    for (int e = t; e < (hz + 1) * kNGrp; e += 256) {
        const int p = e / kNGrp, k = e % kNGrp;
        const float2 w = k < nn ? __ldg(&g.tw[2][p * (g.K[2] + 1) + n0 + k]) : make_float2(0.f, 0.f);
        cs[p * 2 * kNGrp + k] = w.x;
        cs[p * 2 * kNGrp + kNGrp + k] = w.y;
    }
    for (int y0 = 0; y0 < My; y0 += rb) {
        const int ny = min(rb, My - y0);
        if (y0) {
            __syncthreads();
            stage(y0, ny);
        }
        cp_async_wait();
        __syncthreads();
        // two threads per row, each four n
        const int y = t >> 1, nb = (t & 1) * 4;
        if (y < ny && nb < nn) {
            const float* r = rows + y * pitch;
            float re[4] = {0, 0, 0, 0}, im[4] = {0, 0, 0, 0};
            auto add = [&](int p, float e, float o) {
                const float4 c = *reinterpret_cast<const float4*>(cs + p * 2 * kNGrp + nb);
                const float4 s = *reinterpret_cast<const float4*>(cs + p * 2 * kNGrp + kNGrp + nb);
                re[0] = fmaf(e, c.x, re[0]);
                re[1] = fmaf(e, c.y, re[1]);
                re[2] = fmaf(e, c.z, re[2]);
                re[3] = fmaf(e, c.w, re[3]);
                im[0] = fmaf(o, s.x, im[0]);
                im[1] = fmaf(o, s.y, im[1]);
                im[2] = fmaf(o, s.z, im[2]);
                im[3] = fmaf(o, s.w, im[3]);
            };
            add(0, r[0], 0.f);
#pragma unroll 4
            for (int p = 1; p < hz; ++p) {
                const float a = r[p], b = r[Mz - p];
                add(p, a + b, a - b);
            }
            add(hz, r[hz], 0.f);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (nb + k < nn) A[(nb + k) * My + y0 + y] = make_float2(re[k], im[k]);
        }
    }
    __syncthreads();
    // fold y and My - y (over the staged rows): sum and difference side by side
    float4* F = reinterpret_cast<float4*>(rows);
    for (int e = t; e < nn * (hy + 1); e += 256) {
        const int k = e / (hy + 1), y = e % (hy + 1);
        F[k * (hy + 1) + y] = fold(A[k * My + y], A[k * My + (y ? My - y : 0)], y == 0 || y == hy);
    }
    __syncthreads();
    // over y, for m and -m at once, two n per thread
    const int nm = 2 * KM + 1, half = (nn + 1) / 2;
    for (int e = t; e < (KM + 1) * half; e += 256) {
        const int m = e % (KM + 1), k0 = e / (KM + 1), k1 = min(k0 + half, nn - 1);
        Sum2 s;
        s.run(F + k0 * (hy + 1), F + k1 * (hy + 1), ty + m, KM + 1, hy + 1);
        float2* o = g.H + ((size_t)(n0 + k0) * g.M[0] + x) * nm + KM;
        o[m] = s.plus(0);
        if (m) o[-m] = s.minus(0);
        if (k0 + half < nn) {
            o = g.H + ((size_t)(n0 + k1) * g.M[0] + x) * nm + KM;
            o[m] = s.plus(1);
            if (m) o[-m] = s.minus(1);
        }
    }
}

// Over x for one n and up to 8 m: S(k), the energies, C(k), and back over l.  Also clears the grid and
// the buckets' counts for the next evaluation (the force kernel takes its own copy of the counts).
__global__ void __launch_bounds__(256) k_nu_x(NuView g, double* __restrict__ acc_uewa, double* __restrict__ acc_ll) {
    extern __shared__ __align__(16) float sm[];
    const int Mx = g.M[0], hx = Mx / 2, KL = g.K[0], nm = 2 * g.K[1] + 1, nl = 2 * KL + 1, tp = odd(KL + 1);
    const int n = blockIdx.x, m0 = blockIdx.y * g.mgrp, mm = min(g.mgrp, nm - m0);
    const int t = threadIdx.x;
    // columns [m][x]; folded columns [m][x <= hx], later [m][l]; C(k) [m][l + KL]; twiddles [x][l]
    float2* Hs = reinterpret_cast<float2*>(sm);
    float4* F = reinterpret_cast<float4*>(Hs + kMGrp * Mx);
    float2* Cs = reinterpret_cast<float2*>(F + kMGrp * (hx + 1));
    float2* tx = Cs + kMGrp * nl;
    float2* Hn = g.H + (size_t)n * Mx * nm + m0;
    for (int e = t; e < mm * Mx; e += 256) {
        const int x = e / mm, m = e % mm;
        cp_async8(Hs + m * Mx + x, Hn + (size_t)x * nm + m);
    }
    for (int e = t; e < (hx + 1) * (KL + 1); e += 256) cp_async8(tx + (e / (KL + 1)) * tp + e % (KL + 1), g.tw[0] + e);
    {
        const size_t n4 = (size_t)Mx * g.M[1] * g.M[2] / 4, nthr = (size_t)gridDim.x * gridDim.y * 256;
        for (size_t e = (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * 256 + t; e < n4; e += nthr)
            reinterpret_cast<float4*>(g.grid)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (size_t e = (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * 256 + t; e < (size_t)g.nblk + 1; e += nthr) {
            g.cntf[e] = g.cnt[e];
            g.cnt[e] = 0;
        }
    }
    cp_async_wait();
    __syncthreads();
    for (int e = t; e < mm * (hx + 1); e += 256) {
        const int m = e / (hx + 1), x = e % (hx + 1);
        F[e] = fold(Hs[m * Mx + x], Hs[m * Mx + (x ? Mx - x : 0)], x == 0 || x == hx);
    }
    __syncthreads();
    double ew = 0.0, ll = 0.0;
    const int half = (mm + 1) / 2;
    for (int e = t; e < (KL + 1) * half; e += 256) {
        const int l = e % (KL + 1), ma = e / (KL + 1), mb = min(ma + half, mm - 1);
        // k of the set at +l and -l for both m (its index, and bit 0: the conjugate), or -1
        int km[2][2];
        double2 q[2][2];
        double a[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int* kmp = g.kmap + ((size_t)n * nm + m0 + (i ? mb : ma)) * nl + KL;
            const bool on = i == 0 || ma + half < mm;
            km[i][0] = on ? __ldg(kmp + l) : -1;
            km[i][1] = on && l ? __ldg(kmp - l) : -1;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (km[i][h] >= 0) {
                    q[i][h] = __ldg(&g.qw[km[i][h] >> 1]);
                    a[i][h] = __ldg(&g.ak[km[i][h] >> 1]);
                }
        Sum2 s2;
        s2.run(F + ma * (hx + 1), F + mb * (hx + 1), tx + l, tp, hx + 1);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int m = i ? mb : ma, am = abs(m0 + m - g.K[1]);
            const double dec = g.dec[0][l] * g.dec[1][am] * g.dec[2][n];
            const double dec2 = g.dec[0][KL + 1 + l] * g.dec[1][g.K[1] + 1 + am] * g.dec[2][g.K[2] + 1 + n];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if ((h && l == 0) || (i && ma + half >= mm)) break;
                float2 c = make_float2(0.f, 0.f);
                if (km[i][h] >= 0) {
                    const bool cj = km[i][h] & 1;
                    const float2 v = h ? s2.minus(i) : s2.plus(i);
                    double2 s = make_double2((double)v.x * dec, (double)v.y * dec);
                    if (cj) s.y = -s.y;
                    g.S[km[i][h] >> 1] = s;
                    const double2 st = make_double2(s.x + q[i][h].x, s.y + q[i][h].y);
                    const double ak = a[i][h];
                    ll += ak * (s.x * s.x + s.y * s.y);
                    ew += ak * (st.x * st.x + st.y * st.y);
                    c = make_float2((float)(ak * st.x * dec2), (float)((cj ? ak : -ak) * st.y * dec2));
                }
                Cs[m * nl + KL + (h ? -l : l)] = c;
            }
        }
    }
    ew = warp_sum(ew);
    ll = warp_sum(ll);
    if ((t & 31) == 0) {
        if (ew != 0.0) atomicAdd(acc_uewa, ew);
        if (ll != 0.0) atomicAdd(acc_ll, ll);
    }
    __syncthreads();
    for (int e = t; e < mm * (KL + 1); e += 256) {
        const int m = e / (KL + 1), l = e % (KL + 1);
        F[e] = fold(Cs[m * nl + KL + l], Cs[m * nl + KL - l], l == 0);
    }
    __syncthreads();
    for (int e = t; e < (hx + 1) * half; e += 256) {
        const int x = e % (hx + 1), ma = e / (hx + 1), mb = min(ma + half, mm - 1);
        Sum2 s;
        s.run(F + ma * (KL + 1), F + mb * (KL + 1), tx + x * tp, 1, KL + 1);
        // staged in Hs so that the stores below run along m
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float2* o = Hs + (i ? mb : ma) * Mx;
            o[x] = s.plus(i);
            if (x > 0 && x < hx) o[Mx - x] = s.minus(i);
        }
    }
    __syncthreads();
    for (int e = t; e < mm * Mx; e += 256) {
        const int x = e / mm, m = e % mm;
        Hn[(size_t)x * nm + m] = Hs[m * Mx + x];
    }
}

// Back over m and n for one x plane and up to ygrp pairs (y, My - y): the potential on the grid.
__global__ void __launch_bounds__(256) k_nu_yz(NuView g) {
    extern __shared__ __align__(16) float sm[];
    const int My = g.M[1], Mz = g.M[2], hy = My / 2, hz = Mz / 2, KM = g.K[1], KN = g.K[2], nm = 2 * KM + 1;
    const int x = blockIdx.x, y0 = blockIdx.y * g.ygrp, ny = min(g.ygrp, hy + 1 - y0);
    const int t = threadIdx.x;
    float4* F = reinterpret_cast<float4*>(sm);     // folded [n][m]
    float2* Hs = reinterpret_cast<float2*>(F + (size_t)(KN + 1) * (KM + 1));  // [n][m + KM]
    float2* B = Hs + (size_t)(KN + 1) * nm;        // [y pair][2][n]
    float2* ty = B + 2 * g.ygrp * (KN + 1);        // y twiddles [m][y pair]
    float2* tz = ty + (KM + 1) * g.ygrp;           // z twiddles [n][z]
    for (int e = t; e < (KN + 1) * nm; e += 256) {
        const int n = e / nm, m = e % nm;
        cp_async8(Hs + e, g.H + ((size_t)n * g.M[0] + x) * nm + m);
    }
    for (int e = t; e < (KM + 1) * ny; e += 256) cp_async8(ty + e, g.twt[1] + (e / ny) * (hy + 1) + y0 + e % ny);
    for (int e = t; e < (KN + 1) * (hz + 1); e += 256) cp_async8(tz + e, g.twt[2] + e);
    cp_async_wait();
    __syncthreads();
    for (int e = t; e < (KN + 1) * (KM + 1); e += 256) {
        const float2* h = Hs + (e / (KM + 1)) * nm + KM;
        const int m = e % (KM + 1);
        F[e] = fold(h[m], h[-m], m == 0);
    }
    __syncthreads();
    const int half = (KN + 2) / 2;
    for (int e = t; e < half * ny; e += 256) {
        const int yi = e % ny, na = e / ny, nb = min(na + half, KN);
        Sum2 s;
        s.run(F + na * (KM + 1), F + nb * (KM + 1), ty + yi, ny, KM + 1);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            B[(2 * yi) * (KN + 1) + (i ? nb : na)] = s.plus(i);
            B[(2 * yi + 1) * (KN + 1) + (i ? nb : na)] = s.minus(i);
        }
    }
    __syncthreads();
    // over n to z and Mz - z; a thread takes one z and four rows
    const int nrow = 2 * ny, ng = (nrow + 3) / 4;
    for (int e = t; e < (hz + 1) * ng; e += 256) {
        const int z = e % (hz + 1), r0 = (e / (hz + 1)) * 4;
        const float2* b[4];
        float u[4], v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            b[k] = B + min(r0 + k, nrow - 1) * (KN + 1);
            u[k] = b[k][0].x;
            v[k] = 0.f;
        }
#pragma unroll 4
        for (int n = 1; n <= KN; ++n) {
            const float2 w = tz[n * (hz + 1) + z];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 h = b[k][n];
                u[k] = fmaf(h.x, w.x, u[k]);
                v[k] = fmaf(h.y, w.y, v[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = r0 + k;
            if (r >= nrow) break;
            const int yp = y0 + (r >> 1), y = (r & 1) ? My - yp : yp;
            if ((r & 1) && (yp == 0 || yp == hy)) continue;
            float* o = g.pot + ((size_t)x * My + y) * Mz;
            o[z] = u[k] - v[k];
            if (z > 0 && z < hz) o[Mz - z] = u[k] + v[k];
        }
    }
}

// ---- forces ------------------------------------------------------------------------------------
constexpr int kFW = 4;  // warps of a force CTA
constexpr int kFA = 48; // atoms prepared at a time

__global__ void __launch_bounds__(32 * kFW) k_nu_force(NuView g, const uint4* __restrict__ atoms, const __grid_constant__ NuPoly P,
                                                       int natom, double* __restrict__ frc) {
    __shared__ __align__(16) float tile[kTile];
    __shared__ __align__(16) float wts[kFA][3][2 * kW + 4];  // rows 5 x 16 bytes apart
    __shared__ int4 rec[kFA];  // tile offset, atom, charge bits
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, nblk = g.nblk;
    if (blockIdx.x == nblk) {
        // atoms whose block's bucket was full: one warp each, from the grid
        const int n = g.cntf[nblk];
        for (int i = blockIdx.y * kFW + warp; i < n; i += gridDim.y * kFW) {
            const int id = g.ovf[i];
            const uint4 r = atoms[id];
            float t[3], w[3][kW], dw[3][kW];
            const int c0 = cell_of(r.x, g.M[0], t[0]), c1 = cell_of(r.y, g.M[1], t[1]), c2 = cell_of(r.z, g.M[2], t[2]);
#pragma unroll
            for (int d = 0; d < 3; ++d) weights<true>(P, t[d], w[d], dw[d]);
            float ex = 0.f, ey = 0.f, ez = 0.f;
            for (int e = lane; e < kW * kW; e += 32) {
                const int x = wrap(c0 - 3 + e / kW, g.M[0]), y = wrap(c1 - 3 + e % kW, g.M[1]);
                float wx = 0.f, wy = 0.f, dx = 0.f, dy = 0.f, a0 = 0.f, a1 = 0.f;
#pragma unroll
                for (int k = 0; k < kW; ++k) {
                    wx = k == e / kW ? w[0][k] : wx;
                    dx = k == e / kW ? dw[0][k] : dx;
                    wy = k == e % kW ? w[1][k] : wy;
                    dy = k == e % kW ? dw[1][k] : dy;
                    const float p = g.pot[((size_t)x * g.M[1] + y) * g.M[2] + wrap(c2 - 3 + k, g.M[2])];
                    a0 = fmaf(p, w[2][k], a0);
                    a1 = fmaf(p, dw[2][k], a1);
                }
                ex = fmaf(dx * wy, a0, ex);
                ey = fmaf(wx * dy, a0, ey);
                ez = fmaf(wx * wy, a1, ez);
            }
            ex = warp_sum(ex);
            ey = warp_sum(ey);
            ez = warp_sum(ez);
            const float q = -__uint_as_float(r.w);
            if (lane == 0) {
                frc[id] = (double)(q * g.scale[0] * ex);
                frc[natom + id] = (double)(q * g.scale[1] * ey);
                frc[2 * natom + id] = (double)(q * g.scale[2] * ez);
            }
        }
        return;
    }
    const int n = min(g.cntf[blockIdx.x], g.cap);
    const int i0 = (int)((long)n * blockIdx.y / gridDim.y), i1 = (int)((long)n * (blockIdx.y + 1) / gridDim.y);
    if (i0 >= i1) return;
    const int* bucket = g.bucket + (size_t)blockIdx.x * g.cap;
    const int bz = blockIdx.x % g.n8[2], by = (blockIdx.x / g.n8[2]) % g.n8[1], bx = blockIdx.x / (g.n8[2] * g.n8[1]);
    // the block's points: quads along z, all loads of a thread in flight at once
    constexpr int kQ = (900 + 32 * kFW - 1) / (32 * kFW);
    float4 quad[kQ];
#pragma unroll
    for (int k = 0; k < kQ; ++k) {
        const int e = t + k * 32 * kFW, Q = e & 3, X = (e >> 2) / 15, Y = (e >> 2) % 15;
        const int gx = wrap(8 * bx - 3 + X, g.M[0]), gy = wrap(8 * by - 3 + Y, g.M[1]), gz = wrap(8 * bz - 4 + 4 * Q, g.M[2]);
        if (e < 900) quad[k] = __ldg(reinterpret_cast<const float4*>(&g.pot[((size_t)gx * g.M[1] + gy) * g.M[2] + gz]));
    }
#pragma unroll
    for (int k = 0; k < kQ; ++k) {
        const int e = t + k * 32 * kFW;
        if (e < 900) {
            float* o = tile + ((e >> 2) / 15) * kPX + ((e >> 2) % 15) * kPY + 4 * (e & 3);
            o[0] = quad[k].x;
            o[1] = quad[k].y;
            o[2] = quad[k].z;
            o[3] = quad[k].w;
        }
    }
    const int h = lane >> 4, x = lane & 7, y = (lane >> 3) & 1;  // half a warp: one x, y = y, y + 2, .. per lane
    for (int b0 = i0; b0 < i1; b0 += kFA) {
        const int nb = min(kFA, i1 - b0);
        if (b0 > i0) __syncthreads();
        for (int e = t; e < 3 * nb; e += 32 * kFW) {
            const int si = e / 3, sd = e % 3;
            const int id = bucket[b0 + si];
            const uint4 r = atoms[id];
            float tt, w[kW], dw[kW];
            cell_of(sd == 0 ? r.x : sd == 1 ? r.y : r.z, g.M[sd], tt);
            weights<true>(P, tt, w, dw);
            float4* o = reinterpret_cast<float4*>(wts[si][sd]);
            if (sd == 1) {  // even y, odd y
                o[0] = make_float4(w[0], w[2], w[4], w[6]);
                o[1] = make_float4(w[1], w[3], w[5], w[7]);
                o[2] = make_float4(dw[0], dw[2], dw[4], dw[6]);
                o[3] = make_float4(dw[1], dw[3], dw[5], dw[7]);
            } else {
                o[0] = make_float4(w[0], w[1], w[2], w[3]);
                o[1] = make_float4(w[4], w[5], w[6], w[7]);
                o[2] = make_float4(dw[0], dw[1], dw[2], dw[3]);
                o[3] = make_float4(dw[4], dw[5], dw[6], dw[7]);
            }
            if (sd == 0) {
                const int fx = __umulhi(r.x, g.M[0]) & 7, fy = __umulhi(r.y, g.M[1]) & 7, fz = __umulhi(r.z, g.M[2]) & 7;
                rec[si] = make_int4(tile_off(fx, fy, fz), id, (int)(r.w ^ 0x80000000u), 0);
            }
        }
        __syncthreads();
        for (int a0 = 2 * warp; a0 < nb; a0 += 2 * kFW) {
            const int a = min(a0 + h, nb - 1);
            const int4 r = rec[a];
            const float(*w)[2 * kW + 4] = wts[a];
            const float* p = tile + r.x + x * kPX + y * kPY;
            const float4* z = reinterpret_cast<const float4*>(w[2]);
            const float4 za = z[0], zb = z[1], da = z[2], db = z[3];
            const float zw[8] = {za.x, za.y, za.z, za.w, zb.x, zb.y, zb.z, zb.w};
            const float zd[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
            const float4 wy = *reinterpret_cast<const float4*>(w[1] + 4 * y), dy = *reinterpret_cast<const float4*>(w[1] + kW + 4 * y);
            const float wyv[4] = {wy.x, wy.y, wy.z, wy.w}, dyv[4] = {dy.x, dy.y, dy.z, dy.w};
            float s0 = 0.f, s1 = 0.f, sy = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float u0 = 0.f, u1 = 0.f;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float v = p[2 * c * kPY + k];
                    u0 = fmaf(v, zw[k], u0);
                    u1 = fmaf(v, zd[k], u1);
                }
                s0 = fmaf(wyv[c], u0, s0);
                s1 = fmaf(wyv[c], u1, s1);
                sy = fmaf(dyv[c], u0, sy);
            }
            const float wx = w[0][x];
            float s[3] = {w[0][kW + x] * s0, wx * sy, wx * s1};
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
#pragma unroll
                for (int d = 0; d < 3; ++d) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
            const int d = lane & 15;
            if (a0 + h < nb && d < 3)
                frc[d * natom + r.y] = (double)(__int_as_float(r.z) * g.scale[d] * (d == 0 ? s[0] : d == 1 ? s[1] : s[2]));
        }
    }
}

// ---- host: window, its transform and polynomials -----------------------------------------------
double bessel_i0(double x) {
    double s = 1.0, t = 1.0;
    for (int k = 1; k < 200 && t > 1e-18 * s; ++k) {
        t *= (0.5 * x / k) * (0.5 * x / k);
        s += t;
    }
    return s;
}

// Shape of the window: pi w (1 - 1 / (2 sigma)) = 19.5 at w = 8, sigma = 2.2 is best for S(k); the
// gradient by the window's derivative also sees the step that the cut window has at its edge, and is
// best with a higher b there.  In float64 with M = 4K + 8, waters at random orientations: error of the
// reciprocal forces 1.2e-6 with b = 20 for both, 2.8e-7 with these two (S(k): 4e-8).
constexpr double kBetaSpread = 20.0, kBetaForce = 21.5;

double window(double t, double beta) {
    const double a = 1.0 - (2.0 * t / kW) * (2.0 * t / kW);
    return a <= 0.0 ? (a > -1e-12 ? 1.0 / bessel_i0(beta) : 0.0) : bessel_i0(beta * std::sqrt(a)) / bessel_i0(beta);
}

// Monomial coefficients of the interpolant at the kDeg + 1 Chebyshev points of each unit interval.
NuPoly window_poly(double beta) {
    NuPoly P;
    constexpr int n = kDeg + 1;
    const double pi = 3.14159265358979323846;
    for (int k = 0; k < kW; ++k) {
        double cheb[n] = {0}, f[n];
        for (int i = 0; i < n; ++i) {
            const double s = std::cos(pi * (i + 0.5) / n), t = 0.5 * (s + 1.0);
            f[i] = window((double)(k - 3) - t, beta);
        }
        for (int j = 0; j < n; ++j) {
            for (int i = 0; i < n; ++i) cheb[j] += f[i] * std::cos(pi * j * (i + 0.5) / n);
            cheb[j] *= (j ? 2.0 : 1.0) / n;
        }
        // T_0 = 1, T_1 = s, T_{j+1} = 2 s T_j - T_{j-1}
        double c[n] = {0}, a[n] = {0}, b[n] = {0};
        a[0] = 1.0;
        b[1] = 1.0;
        for (int i = 0; i < n; ++i) c[i] = cheb[0] * a[i] + cheb[1] * b[i];
        for (int j = 2; j < n; ++j) {
            double d[n];
            for (int i = 0; i < n; ++i) d[i] = (i ? 2.0 * b[i - 1] : 0.0) - a[i];
            for (int i = 0; i < n; ++i) {
                c[i] += cheb[j] * d[i];
                a[i] = b[i];
                b[i] = d[i];
            }
        }
        for (int i = 0; i < n; ++i) P.c[k][i] = (float)c[i];
    }
    return P;
}

// 1 / phi^(k) of one direction, phi^(k) = integral of phi(t) cos(2 pi k t / M).  The trapezoid rule at
// spacing 1/32 is exact to 2e-10 here: phi is analytic, about a Gaussian of width 0.9, and 1e-8 at
// its ends.
struct WindowTable {
    static constexpr int n = 32 * kW / 2;
    double f[n + 1];
    explicit WindowTable(double beta) {
        for (int i = 0; i <= n; ++i) f[i] = window(i / 32.0, beta) / 16.0 * (i == 0 || i == n ? 0.5 : 1.0);
    }
    double inverse(int k, int M) const {
        const double c = std::cos(2.0 * 3.14159265358979323846 * k / (32.0 * M));
        double a = 1.0, b = c, s = f[0];  // cos(i w) by recurrence
        for (int i = 1; i <= n; ++i) {
            s += f[i] * b;
            const double d = 2.0 * c * b - a;
            a = b;
            b = d;
        }
        return 1.0 / s;
    }
};

}  // namespace

int recip_nu_setup(Ctx& c) {
    View& v = c.v;
    KSet& ks = c.ks;
    NuView& g = c.nu.g;
    if (ks.nk == 0 || v.nmove == 0) return MDG_OK;
    static const WindowTable spread(kBetaSpread), force(kBetaForce);
    const int K[3] = {ks.klmax, ks.kmmax, ks.knmax};
    const double pip[3] = {ks.pipix, ks.pipiy, ks.pipiz}, len[3] = {v.lx, v.ly, v.lz};
    size_t npts = 1, nblk = 1;
    double cell = 1.0;
    for (int d = 0; d < 3; ++d) {
        g.K[d] = K[d];
        g.M[d] = std::max(16, 4 * K[d] + 8);  // 2.1 to 2.5 (2K + 1), a multiple of 4
        g.n8[d] = (g.M[d] + 7) / 8;
        g.scale[d] = (float)(g.M[d] * pip[d] / (2.0 * 3.14159265358979323846));
        npts *= g.M[d];
        nblk *= g.n8[d];
        cell *= 8.0 * len[d] / g.M[d];
    }
    // bucket room: three times the mean, or three times a dense liquid's 0.11 atoms / A^3
    const double want = 3.0 * std::max((double)v.nmove / (double)nblk, 0.11 * cell) + 16.0;
    g.cap = (int)std::min<double>(want, v.nmove);
    g.nblk = (int)nblk;
    g.split = std::max(1, std::min(64, std::max((int)(v.nmove / nblk / kSplit) + 1, (int)(912 / nblk))));
    const int nm = 2 * K[1] + 1, nl = 2 * K[0] + 1;
    std::vector<int> kmap((size_t)(K[2] + 1) * nm * nl, -1);
    for (int r = 0; r < ks.nrow; ++r)
        for (int i = 0; i < ks.h_nlen[r]; ++i) {
            int l = ks.h_row[r].x, m = ks.h_row[r].y, n = ks.h_row[r].z + i, cj = 0;
            if (n < 0) {
                l = -l;
                m = -m;
                n = -n;
                cj = 1;
            }
            kmap[((size_t)n * nm + m + K[1]) * nl + l + K[0]] = 2 * (ks.h_row[r].w + i) + cj;
        }
    auto put = [&](const void* h, size_t bytes) {
        void* p = dalloc(c, bytes);
        if (p && bytes) cudaMemcpy(p, h, bytes, cudaMemcpyHostToDevice);
        return p;
    };
    g.kmap = (int*)put(kmap.data(), sizeof(int) * kmap.size());
    for (int d = 0; d < 3; ++d) {
        const int h = g.M[d] / 2, k1 = K[d] + 1;
        std::vector<float2> a((size_t)(h + 1) * k1), b(a.size());
        std::vector<double> dec(2 * k1);
        for (int p = 0; p <= h; ++p)
            for (int k = 0; k < k1; ++k) {
                const double w = 2.0 * 3.14159265358979323846 * (double)((long)p * k % g.M[d]) / g.M[d];
                a[(size_t)p * k1 + k] = b[(size_t)k * (h + 1) + p] = make_float2((float)std::cos(w), (float)std::sin(w));
            }
        for (int k = 0; k < k1; ++k) {
            dec[k] = spread.inverse(k, g.M[d]);
            dec[k1 + k] = force.inverse(k, g.M[d]);
        }
        g.tw[d] = (float2*)put(a.data(), sizeof(float2) * a.size());
        g.twt[d] = (float2*)put(b.data(), sizeof(float2) * b.size());
        g.dec[d] = (double*)put(dec.data(), sizeof(double) * dec.size());
    }
    g.grid = (float*)dalloc(c, sizeof(float) * npts);
    g.pot = (float*)dalloc(c, sizeof(float) * npts);
    g.H = (float2*)dalloc(c, sizeof(float2) * (size_t)(K[2] + 1) * g.M[0] * nm);
    g.cnt = (int*)dalloc(c, sizeof(int) * (nblk + 1));
    g.cntf = (int*)dalloc(c, sizeof(int) * (nblk + 1));
    g.novf = g.cnt + nblk;
    g.bucket = (int*)dalloc(c, sizeof(int) * nblk * g.cap);
    g.ovf = (int*)dalloc(c, sizeof(int) * v.nmove);
    g.S = ks.s;
    g.qw = ks.qw;
    g.ak = ks.ak;
    if (c.alloc_failed) return set_err(&c, MDG_E_CUDA, "out of device memory for the reciprocal sum");
    // groups: two CTAs per SM where the planes are few
    const int want_n = std::max(1, (304 + g.M[0] - 1) / g.M[0]);
    g.ngrp = std::max(1, std::min(kNGrp, (K[2] + want_n) / want_n));
    g.ngrp = (K[2] + 1 + (K[2] + g.ngrp) / g.ngrp - 1) / ((K[2] + g.ngrp) / g.ngrp);  // even groups
    const int want_m = std::max(1, (304 + K[2]) / (K[2] + 1));
    g.mgrp = std::max(1, std::min(kMGrp, (nm + want_m - 1) / want_m));
    const int hy1 = g.M[1] / 2 + 1;
    g.ygrp = std::max(2, std::min(16, (hy1 + want_n - 1) / want_n));
    const int fixed = (g.M[2] / 2 + 1) * 2 * kNGrp + 2 * kNGrp * g.M[1] + ((2 * hy1 * (K[1] + 1) + 3) & ~3);
    g.yrows = std::min(kYRows, g.M[1]);
    // (the staged rows' space later holds the folded sums of 8 n)
    while (g.yrows > 32 && (fixed + g.yrows * (g.M[2] + 4)) * (int)sizeof(float) > 110 * 1024) g.yrows /= 2;
    c.nu.smem_zy = (fixed + std::max(g.yrows * (g.M[2] + 4), 4 * kNGrp * hy1)) * (int)sizeof(float);
    c.nu.smem_x = (kMGrp * (g.M[0] + 2 * (g.M[0] / 2 + 1) + nl) + (g.M[0] / 2 + 1) * ((K[0] + 1) | 1)) * (int)sizeof(float2);
    c.nu.smem_yz = ((K[2] + 1) * (2 * (K[1] + 1) + nm + 2 * g.ygrp + g.M[2] / 2 + 1) + (K[1] + 1) * g.ygrp) * (int)sizeof(float2);
    MDG_CUDA(allow_max_smem(k_nu_zy));
    MDG_CUDA(allow_max_smem(k_nu_x));
    MDG_CUDA(allow_max_smem(k_nu_yz));
    if (std::max(c.nu.smem_zy, std::max(c.nu.smem_x, c.nu.smem_yz)) > 227 * 1024)
        return set_err(&c, MDG_E_UNSUPPORTED, "k range too large for the shared-memory tables of the reciprocal sum");
    c.nu.ready = true;
    return MDG_OK;
}

void recip_nu(Ctx& c) {
    static const NuPoly P = window_poly(kBetaSpread), PF = window_poly(kBetaForce);
    const NuView& g = c.nu.g;
    const int nm = 2 * g.K[1] + 1, nmove = c.v.nmove;
    const dim3 blocks(g.nblk + 1, g.split);  // the last: atoms without a place in their bucket
    double* acc = c.v.acc + 2 * c.v.nijt;
    k_nu_spread<<<blocks, 64, 0, c.stream>>>(g, c.d_tc_atoms, P);
    k_nu_zy<<<dim3(g.M[0], (g.K[2] + g.ngrp) / g.ngrp), 256, c.nu.smem_zy, c.stream>>>(g);
    k_nu_x<<<dim3(g.K[2] + 1, (nm + g.mgrp - 1) / g.mgrp), 256, c.nu.smem_x, c.stream>>>(g, acc + ACC_UEWA, acc + ACC_EWQLL);
    k_nu_yz<<<dim3(g.M[0], (g.M[1] / 2 + 1 + g.ygrp - 1) / g.ygrp), 256, c.nu.smem_yz, c.stream>>>(g);
    k_nu_force<<<blocks, 32 * kFW, 0, c.stream>>>(g, c.d_tc_atoms, PF, nmove, c.d_frc);
}

}  // namespace mdg
