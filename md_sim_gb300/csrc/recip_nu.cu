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
// With b = 20 for spreading and 21.5 for the forces the window and its aliases leave a relative error of about
// 3e-7 in the reciprocal forces (4e-8 in S(k)); everything between the fixed-point positions and C(k) is
// FP32, C(k) and the energies are FP64 as in the direct form.  The Fourier sums are in nu_fourier.cuh.
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
// tensor-core passes take 310 (143 + 11 + 5 + 156); forces of the whole evaluation 6.2e-7 off FP64 (tensor
// cores 1.1e-6), reciprocal energy 2e-7 (1.9e-6).  Spread and
// force are bound by shared-memory wavefronts (79 and 82 % of the L1 pipe), the Fourier sums by them
// and by the few CTAs.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "nu_fourier.cuh"

namespace mdg {

namespace {

constexpr int kW = 8;       // window width in grid points
constexpr int kDeg = 9;     // degree of the window's polynomial on each unit interval (error 7e-8)
constexpr int kStage = 10;  // atoms a warp prepares at a time (3 lanes each)
constexpr int kPX = 260, kPY = 17;  // pitches of a block's points: 4 x (of one parity) times 8 y hit 32 banks
constexpr int kTile = 15 * kPX;     // x, y from 3 cells below the block, z from 4 (quads aligned to 4)

// weight of point k (0..7) for an atom at fraction t of its cell: sum_i c[k][i] s^i, s = 2t - 1
struct NuPoly {
    float c[kW][kDeg + 1];
};

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

int recip_nu_points(int K) { return std::max(16, 4 * K + 8); }  // 2.1 to 2.5 (2K + 1), a multiple of 4

int recip_nu_setup(Ctx& c) {
    if (c.ks.nk == 0 || c.v.nmove == 0) return MDG_OK;
    static const WindowTable spread(kBetaSpread), force(kBetaForce);
    return nu_setup<float>(c, c.nu, recip_nu_points, [](int h, int k, int M) { return (h ? force : spread).inverse(k, M); });
}

void recip_nu(Ctx& c) {
    static const NuPoly P = window_poly(kBetaSpread), PF = window_poly(kBetaForce);
    const NuView& g = c.nu.g;
    const dim3 blocks(g.nblk + 1, g.split);  // the last: atoms without a place in their bucket
    k_nu_spread<<<blocks, 64, 0, c.stream>>>(g, c.d_tc_atoms, P);
    nu_fourier(c, c.nu);
    k_nu_force<<<blocks, 32 * kFW, 0, c.stream>>>(g, c.d_tc_atoms, PF, c.v.nmove, c.d_frc);
}

}  // namespace mdg
