// recip_nu64.cu - reciprocal-space Ewald sum of the FP64 form by gridding (force_fouri,
// src/forcem.f90:827-937), for systems where the products of every atom with every k vector (recip.cu) take
// longer: the method and the Fourier sums of recip_nu.cu with everything in FP64 and a window of 16
// points per direction.  With beta = 39 and grids of at least 4.5 K points the window and its aliases leave
// 2e-14 of a term's amplitude in S(k) and 3e-14 in its gradient, at the rounding of the phase
// recurrences of the direct sums.
//
//   k_nu64_bin     grid coordinates and charges into the buckets of blocks of 8 x 8 x 8 cells
//   k_nu64_spread  one CTA per block (more where blocks hold many atoms): the block's 23 x 23 x 23 points in
//                  shared memory.  Warp w owns the x planes with X % 8 == w, so that an atom's 16 planes
//                  are 2 per warp and no two warps add to one point; a lane takes one z, half a
//                  warp a row.
//   k_nu_zy, k_nu_x, k_nu_yz   (nu_fourier.cuh)
//   k_nu64_force   the block's points of the potential in shared memory, a warp per atom
//
// FP64 operations bound spread and force: 1 and 2.4 per point and atom, 4,096 points.
// 98,304 atoms, 29,038 k vectors (M = 112): spread 0.98 ms, zy 0.17, x 0.07, yz 0.11, force 1.98 = 3.3 ms where
// the direct sums take 44; a force call 46.1 -> 5.4 ms.  6,144 atoms, 4,338 k in a slab: 0.39 ms for 0.49.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "nu_fourier.cuh"

namespace mdg {

namespace {

constexpr int kW = 16;            // window width in grid points
constexpr double kBeta = 39.0;    // below pi w (1 - K / M), where the first alias would see the window's pass band
constexpr int kHC = 8;            // coefficients of the even and of the odd half of a weight's polynomial
constexpr int kT = 23;            // points of a block per direction: 7 below its 8 cells, 8 above
constexpr int kTile = kT * kT * kT;
constexpr int kNT = 256, kWarps = kNT / 32;
constexpr int kSA = 32, kFA = 16;  // atoms prepared at a time by spread and force (two CTAs per SM)

// Weight of point k < 8 at fraction t of the cell, s = 2 t - 1: E_k(s^2) + s O_k(s^2), of point 15 - k:
// E_k - s O_k; derivatives by t: s F_k(s^2) + G_k(s^2), and (of 15 - k) s F_k - G_k.
struct NuPoly64 {
    double e[kW / 2][kHC], o[kW / 2][kHC], f[kW / 2][kHC], g[kW / 2][kHC];
};
__constant__ NuPoly64 c_poly;

__device__ __forceinline__ double horner(const double* c, double r) {
    double a = c[kHC - 1];
#pragma unroll
    for (int i = kHC - 2; i >= 0; --i) a = fma(a, r, c[i]);
    return a;
}

// cell (0..M-1) and fraction of a grid coordinate in [0, M)
__device__ __forceinline__ int cell64(double u, int M, double& t) {
    const int c = max(0, min(M - 1, (int)u));
    t = u - (double)c;
    return c;
}

// cell and block of an atom's record (coordinates r0.x, r0.y, r1.x)
__device__ __forceinline__ int block_of(const NuViewT<double>& g, int cx, int cy, int cz) {
    return ((cx >> 3) * g.n8[1] + (cy >> 3)) * g.n8[2] + (cz >> 3);
}

__global__ void k_nu64_bin(View v, NuViewT<double> g, double2* __restrict__ rec) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= v.nmove) return;
    double u[3] = {v.x[j] * g.scale[0], v.y[j] * g.scale[1], v.z[j] * g.scale[2]};
    int c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double M = g.M[d];
        u[d] -= M * floor(u[d] / M);
        if (u[d] >= M) u[d] -= M;  // a tiny negative coordinate rounds up to M
        c[d] = max(0, min(g.M[d] - 1, (int)u[d]));
    }
    const int b = block_of(g, c[0], c[1], c[2]), k = atomicAdd(&g.cnt[b], 1);
    size_t slot = (size_t)b * g.cap + k;
    int* ids = g.bucket;
    if (k >= g.cap) {
        const int o = atomicAdd(g.novf, 1);
        slot = (size_t)g.nblk * g.cap + o;
        ids = g.ovf - (size_t)g.nblk * g.cap;
    }
    rec[2 * slot] = make_double2(u[0], u[1]);
    rec[2 * slot + 1] = make_double2(u[2], v.q[j]);
    ids[slot] = j;
}

// Weights (GRAD: and derivatives) of n atoms and their cells: 24 tasks each, a direction and a pair of points.
// Without GRAD the x weights carry the charge.
template <bool GRAD>
__device__ __forceinline__ void prepare(const NuViewT<double>& g, const double2* __restrict__ rec, int n, double (*wts)[3][kW],
                                        double (*dwts)[3][kW], int (*cell)[4], double* charge) {
    for (int e = threadIdx.x; e < 24 * n; e += kNT) {
        const int a = e / 24, d = (e % 24) >> 3, k = e & 7;
        const double2 r0 = rec[2 * a], r1 = rec[2 * a + 1];
        double t;
        const int c = cell64(d == 0 ? r0.x : d == 1 ? r0.y : r1.x, g.M[d], t);
        const double s = 2.0 * t - 1.0, r = s * s;
        double ev = horner(c_poly.e[k], r), od = s * horner(c_poly.o[k], r);
        if (!GRAD && d == 0) {
            ev *= r1.y;
            od *= r1.y;
        }
        wts[a][d][k] = ev + od;
        wts[a][d][kW - 1 - k] = ev - od;
        if (GRAD) {
            const double f = s * horner(c_poly.f[k], r), gg = horner(c_poly.g[k], r);
            dwts[a][d][k] = f + gg;
            dwts[a][d][kW - 1 - k] = f - gg;
            if (e % 24 == 0) charge[a] = r1.y;
        }
        if (k == 0) cell[a][d] = c;
    }
}

__global__ void __launch_bounds__(kNT) k_nu64_spread(NuViewT<double> g, const double2* __restrict__ rec) {
    extern __shared__ __align__(16) double tile[];  // [x][y][z]
    __shared__ double wts[kSA][3][kW];
    __shared__ int cell[kSA][4];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nblk = g.nblk;
    if (blockIdx.x == nblk) {
        // atoms whose block's bucket was full: straight to the grid
        const int n = *g.novf;
        for (int i = blockIdx.y; i < n; i += gridDim.y) {
            __syncthreads();
            prepare<false>(g, rec + 2 * ((size_t)nblk * g.cap + i), 1, wts, nullptr, cell, nullptr);
            __syncthreads();
            const int kx = t >> 4, ky = t & 15;
            const int x = wrap(cell[0][0] - 7 + kx, g.M[0]), y = wrap(cell[0][1] - 7 + ky, g.M[1]);
            const double c = wts[0][0][kx] * wts[0][1][ky];
            for (int k = 0; k < kW; ++k)
                atomicAdd(&g.grid[((size_t)x * g.M[1] + y) * g.M[2] + wrap(cell[0][2] - 7 + k, g.M[2])], c * wts[0][2][k]);
        }
        return;
    }
    const int n = min(g.cnt[blockIdx.x], g.cap);
    const int i0 = (int)((long)n * blockIdx.y / gridDim.y), i1 = (int)((long)n * (blockIdx.y + 1) / gridDim.y);
    if (i0 >= i1) return;
    for (int e = t; e < kTile; e += kNT) tile[e] = 0.0;
    const int z = lane & 15, h = lane >> 4;
    for (int b0 = i0; b0 < i1; b0 += kSA) {
        const int nb = min(kSA, i1 - b0);
        __syncthreads();
        prepare<false>(g, rec + 2 * ((size_t)blockIdx.x * g.cap + b0), nb, wts, nullptr, cell, nullptr);
        __syncthreads();
        for (int a = 0; a < nb; ++a) {
            // this warp's planes: X = k + fx with X % 8 == warp, k < 16
            const int fx = cell[a][0] & 7, fy = cell[a][1] & 7, fz = cell[a][2] & 7, k0 = (warp - fx) & 7;
            const double wz = wts[a][2][z];
            // lane (h, z): the product of x plane k0 + 8 h and y = z
            const double c = wts[a][0][k0 + 8 * h] * wts[a][1][z];
            double* p = tile + ((k0 + fx) * kT + fy + h) * kT + fz + z;
#pragma unroll
            for (int b = 0; b < 2; ++b, p += 8 * kT * kT) {
                double s[8];
#pragma unroll
                for (int y = 0; y < 8; ++y) s[y] = p[2 * y * kT];
#pragma unroll
                for (int y = 0; y < 8; ++y)
                    p[2 * y * kT] = fma(__shfl_sync(0xffffffffu, c, 16 * b + 2 * y + h), wz, s[y]);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    const int bz = blockIdx.x % g.n8[2], by = (blockIdx.x / g.n8[2]) % g.n8[1], bx = blockIdx.x / (g.n8[2] * g.n8[1]);
    for (int e = t; e < kTile; e += kNT) {
        const double s = tile[e];
        if (s == 0.0) continue;
        const int X = e / (kT * kT), Y = (e / kT) % kT, Z = e % kT;
        const int gx = wrap(8 * bx - 7 + X, g.M[0]), gy = wrap(8 * by - 7 + Y, g.M[1]), gz = wrap(8 * bz - 7 + Z, g.M[2]);
        atomicAdd(&g.grid[((size_t)gx * g.M[1] + gy) * g.M[2] + gz], s);
    }
}

// Sums of three values over the warp: lane 0 gets a, lane 16 b, every lane c.
__device__ __forceinline__ double2 warp_sum3(double a, double b, double c) {
    const bool up = threadIdx.x & 16;
    double s = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return make_double2(s, warp_sum(c));
}

__global__ void __launch_bounds__(kNT) k_nu64_force(View v, NuViewT<double> g, const double2* __restrict__ rec) {
    extern __shared__ __align__(16) double tile[];
    __shared__ double wts[kFA][3][kW], dwts[kFA][3][kW], charge[kFA];
    __shared__ int cell[kFA][4];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nblk = g.nblk;
    // (atomics: the real-space loops may be running)
    auto add = [&](int id, double q, double2 s) {
        if (lane == 0) {
            atomicAdd(&v.fx[id], -q * g.scale[0] * s.x);
            atomicAdd(&v.fz[id], -q * g.scale[2] * s.y);
        }
        if (lane == 16) atomicAdd(&v.fy[id], -q * g.scale[1] * s.x);
    };
    const int z = lane & 15, h = lane >> 4;
    if (blockIdx.x == nblk) {
        // atoms whose block's bucket was full: one at a time, from the grid, by the first warp
        const int n = g.cntf[nblk];
        for (int i = blockIdx.y; i < n; i += gridDim.y) {
            __syncthreads();
            prepare<true>(g, rec + 2 * ((size_t)nblk * g.cap + i), 1, wts, dwts, cell, charge);
            __syncthreads();
            if (warp) continue;
            double ex = 0.0, ey = 0.0, ez = 0.0;
            const int gz = wrap(cell[0][2] - 7 + z, g.M[2]);
            for (int e = h; e < kW * kW; e += 2) {
                const int kx = e >> 4, ky = e & 15;
                const double p = g.pot[((size_t)wrap(cell[0][0] - 7 + kx, g.M[0]) * g.M[1] + wrap(cell[0][1] - 7 + ky, g.M[1])) *
                                           g.M[2] + gz];
                ex += p * dwts[0][0][kx] * wts[0][1][ky];
                ey += p * wts[0][0][kx] * dwts[0][1][ky];
                ez += p * wts[0][0][kx] * wts[0][1][ky];
            }
            add(g.ovf[i], charge[0], warp_sum3(ex * wts[0][2][z], ey * wts[0][2][z], ez * dwts[0][2][z]));
        }
        return;
    }
    const int n = min(g.cntf[blockIdx.x], g.cap);
    const int i0 = (int)((long)n * blockIdx.y / gridDim.y), i1 = (int)((long)n * (blockIdx.y + 1) / gridDim.y);
    if (i0 >= i1) return;
    const int bz = blockIdx.x % g.n8[2], by = (blockIdx.x / g.n8[2]) % g.n8[1], bx = blockIdx.x / (g.n8[2] * g.n8[1]);
#pragma unroll 8
    for (int e = t; e < kTile; e += kNT) {
        const int X = e / (kT * kT), Y = (e / kT) % kT, Z = e % kT;
        const int gx = wrap(8 * bx - 7 + X, g.M[0]), gy = wrap(8 * by - 7 + Y, g.M[1]), gz = wrap(8 * bz - 7 + Z, g.M[2]);
        tile[e] = __ldg(&g.pot[((size_t)gx * g.M[1] + gy) * g.M[2] + gz]);
    }
    for (int b0 = i0; b0 < i1; b0 += kFA) {
        const int nb = min(kFA, i1 - b0);
        __syncthreads();
        prepare<true>(g, rec + 2 * ((size_t)blockIdx.x * g.cap + b0), nb, wts, dwts, cell, charge);
        __syncthreads();
        for (int a = warp; a < nb; a += kWarps) {
            const int fx = cell[a][0] & 7, fy = cell[a][1] & 7, fz = cell[a][2] & 7;
            double wy[8], dy[8];
#pragma unroll
            for (int y = 0; y < 8; ++y) {
                wy[y] = wts[a][1][2 * y + h];
                dy[y] = dwts[a][1][2 * y + h];
            }
            const double* p = tile + (fx * kT + fy + h) * kT + fz + z;
            double sx = 0.0, sy = 0.0, s0 = 0.0;
#pragma unroll 4
            for (int k = 0; k < kW; ++k, p += kT * kT) {
                double u = 0.0, w = 0.0;
#pragma unroll
                for (int y = 0; y < 8; ++y) {
                    const double f = p[2 * y * kT];
                    u = fma(f, wy[y], u);
                    w = fma(f, dy[y], w);
                }
                const double wx = wts[a][0][k];
                sx = fma(dwts[a][0][k], u, sx);
                sy = fma(wx, w, sy);
                s0 = fma(wx, u, s0);
            }
            const double wz = wts[a][2][z];
            add(g.bucket[(size_t)blockIdx.x * g.cap + b0 + a], charge[a], warp_sum3(sx * wz, sy * wz, s0 * dwts[a][2][z]));
        }
    }
}

// ---- host: window, its transform and polynomials -----------------------------------------------
long double bessel_i0(long double x) {
    long double s = 1, t = 1;
    for (int k = 1; k < 400 && t > 1e-25L * s; ++k) {
        t *= (x / 2 / k) * (x / 2 / k);
        s += t;
    }
    return s;
}

// I0(beta sqrt(1 - (t/8)^2)) / I0(beta) on |t| < 8
long double window(long double t) {
    const long double a = 1 - (t / 8) * (t / 8);
    return bessel_i0(kBeta * std::sqrt(std::max(a, 0.0L))) / bessel_i0(kBeta);
}

// 1 / its transform at frequency k of M: w sinh(r) / (I0(beta) r), r^2 = beta^2 - (pi w k / M)^2
double inverse_transform(int k, int M) {
    const long double a = 3.14159265358979323846L * kW * k / M, r = std::sqrt(kBeta * kBeta - a * a);
    return (double)(bessel_i0(kBeta) * r / (kW * std::sinh(r)));
}

// Interpolants at the 16 Chebyshev points of each unit interval (within 1e-18), split by parity.
NuPoly64 window_poly() {
    NuPoly64 P;
    constexpr int n = 2 * kHC;
    const long double pi = 3.14159265358979323846L;
    for (int k = 0; k < kW / 2; ++k) {
        long double cheb[n] = {0}, f[n];
        for (int i = 0; i < n; ++i) {
            const long double s = std::cos(pi * (i + 0.5L) / n);
            f[i] = window((s + 1) / 2 + 7 - k);  // the atom is that far above point k
        }
        for (int j = 0; j < n; ++j) {
            for (int i = 0; i < n; ++i) cheb[j] += f[i] * std::cos(pi * j * (i + 0.5L) / n);
            cheb[j] *= (j ? 2.0L : 1.0L) / n;
        }
        long double c[n + 1] = {0}, a[n] = {1}, b[n] = {0, 1};  // T_0, T_1 in powers of s
        for (int i = 0; i < n; ++i) c[i] = cheb[0] * a[i] + cheb[1] * b[i];
        for (int j = 2; j < n; ++j) {
            long double d[n];
            for (int i = 0; i < n; ++i) d[i] = (i ? 2 * b[i - 1] : 0.0L) - a[i];
            for (int i = 0; i < n; ++i) {
                c[i] += cheb[j] * d[i];
                a[i] = b[i];
                b[i] = d[i];
            }
        }
        for (int i = 0; i < kHC; ++i) {
            P.e[k][i] = (double)c[2 * i];
            P.o[k][i] = (double)c[2 * i + 1];
            // d/dt = 2 d/ds
            P.f[k][i] = (double)(2 * (2 * i + 2) * c[2 * i + 2]);
            P.g[k][i] = (double)(2 * (2 * i + 1) * c[2 * i + 1]);
        }
    }
    return P;
}

constexpr int kSmem = kTile * (int)sizeof(double);

}  // namespace

// Atoms times k vectors from which the grid is faster: below, its six kernels and the points of mostly empty
// blocks cost more than the products.  Whole force calls, direct | grid: 1,000 waters (3.2e6) 325 | 343 us, 1,331
// (6.1e6) 435 | 399, 1,728 (1.1e7) 550 | 476; slabs of 700 (3.0e6) 313 | 343, 1,000 (6.4e6) 435 | 376 and 2,048
// waters (2.6e7) 821 | 615.
constexpr double kGridWork64 = 5.0e6;

// Takes the gridded sum where the rule asks for it and its tables and arrays have room; the direct sums
// (recip.cu) otherwise.
int recip_nu64_setup(Ctx& c) {
    const View& v = c.v;
    if (c.ks.nk == 0 || (double)v.nmove * c.ks.nk < kGridWork64) return MDG_OK;
    NuPlanT<double>& plan = c.nu64;
    // what is forgiven below is what this function asks for
    if (c.alloc_failed) return set_err(&c, MDG_E_CUDA, "out of device memory for the reciprocal sum");
    const size_t mark = c.owned.size();
    const int rc = nu_setup<double>(
        c, plan, [](int K) { return std::max(24, (9 * K / 2 + 4 + 7) / 8 * 8); },
        [](int, int k, int M) { return inverse_transform(k, M); });
    if (rc == MDG_OK) plan.rec = (double2*)dalloc(c, 2 * sizeof(double2) * ((size_t)plan.g.nblk * plan.g.cap + v.nmove));
    if (rc != MDG_OK || c.alloc_failed) {
        drop_owned(c, mark);
        plan = NuPlanT<double>();
        c.err.clear();
        return MDG_OK;
    }
    static const NuPoly64 P = window_poly();
    MDG_CUDA(cudaMemcpyToSymbol(c_poly, &P, sizeof(P)));
    MDG_CUDA(allow_max_smem(k_nu64_spread));
    MDG_CUDA(allow_max_smem(k_nu64_force));
    return MDG_OK;
}

void recip_nu64(Ctx& c) {
    const View& v = c.v;
    const NuViewT<double>& g = c.nu64.g;
    const dim3 blocks(g.nblk + 1, g.split);  // the last: atoms without a place in their bucket
    k_nu64_bin<<<(v.nmove + 127) / 128, 128, 0, c.stream>>>(v, g, c.nu64.rec);
    k_nu64_spread<<<blocks, kNT, kSmem, c.stream>>>(g, c.nu64.rec);
    nu_fourier(c, c.nu64);
    k_nu64_force<<<blocks, kNT, kSmem, c.stream>>>(v, g, c.nu64.rec);
}

}  // namespace mdg
