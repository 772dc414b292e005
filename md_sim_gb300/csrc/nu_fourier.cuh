// nu_fourier.cuh - the separable Fourier sums of the gridded reciprocal sums (recip_nu.cu in FP32,
// recip_nu64.cu in FP64) and what their plans share: k set map, twiddles, groups, shared-memory sizes.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "ctx.h"

namespace mdg {

constexpr int kSplit = 64;  // atoms of a block that one more CTA is given for

template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (BYTES == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename T>
__device__ __forceinline__ typename NuVec<T>::V2 v2(T a, T b) {
    typename NuVec<T>::V2 r;
    r.x = a;
    r.y = b;
    return r;
}
template <typename T>
__device__ __forceinline__ typename NuVec<T>::V4 v4(T a, T b, T c, T d) {
    typename NuVec<T>::V4 r;
    r.x = a;
    r.y = b;
    r.z = c;
    r.w = d;
    return r;
}

__device__ __forceinline__ int wrap(int g, int M) { return g < 0 ? g + M : g >= M ? g - M : g; }

// Twiddle tables of a direction: tw[p * (K + 1) + k] and twt[k * (M/2 + 1) + p], both
// (cos, sin)(2 pi k p / M) for p = 0..M/2, k = 0..K.
constexpr int kNGrp = 8;    // most n of one k_nu_zy CTA
constexpr int kMGrp = 8;    // most m of one k_nu_x CTA
constexpr int kYRows = 128; // most y rows staged at a time in k_nu_zy

__device__ __forceinline__ int odd(int n) { return n | 1; }

// A folded pair of terms: (a + b, a - b), or (a, 0) for a term that is its own partner.
template <typename T>
__device__ __forceinline__ typename NuVec<T>::V4 fold(typename NuVec<T>::V2 a, typename NuVec<T>::V2 b, bool own) {
    return own ? v4<T>(a.x, a.y, T(0), T(0)) : v4<T>(a.x + b.x, a.y + b.y, a.x - b.x, a.y - b.y);
}

// Two folded Fourier sums with one set of twiddles: u = sum e cos, v = sum o sin (complex each);
// u + i v is the sum at the twiddles' frequency (or point), u - i v the one at its negative.
template <typename T>
struct Sum2 {
    typedef typename NuVec<T>::V2 V2;
    typedef typename NuVec<T>::V4 V4;
    V2 u[2], v[2];
    __device__ __forceinline__ void run(const V4* __restrict__ a, const V4* __restrict__ b,
                                        const V2* __restrict__ w, int wstride, int n) {
        u[0] = u[1] = v[0] = v[1] = v2<T>(0, 0);
#pragma unroll 4
        for (int p = 0; p < n; ++p) {
            const V2 c = w[p * wstride];
            const V4 x = a[p], y = b[p];
            u[0].x = fma(x.x, c.x, u[0].x);
            u[0].y = fma(x.y, c.x, u[0].y);
            v[0].x = fma(x.z, c.y, v[0].x);
            v[0].y = fma(x.w, c.y, v[0].y);
            u[1].x = fma(y.x, c.x, u[1].x);
            u[1].y = fma(y.y, c.x, u[1].y);
            v[1].x = fma(y.z, c.y, v[1].x);
            v[1].y = fma(y.w, c.y, v[1].y);
        }
    }
    __device__ __forceinline__ V2 plus(int k) const { return v2<T>(u[k].x - v[k].y, u[k].y + v[k].x); }
    __device__ __forceinline__ V2 minus(int k) const { return v2<T>(u[k].x + v[k].y, u[k].y - v[k].x); }
};

// Sum over z then y of one x plane: H[n][x][m] for n = n0..n0 + nn - 1 (nn <= 8), m = -KM..KM.
// Staged rows are Mz and 16 bytes apart (copied by 16 bytes; in FP32 8 of them on different banks).
template <typename T>
__global__ void __launch_bounds__(256) k_nu_zy(NuViewT<T> g) {
    typedef typename NuVec<T>::V2 V2;
    typedef typename NuVec<T>::V4 V4;
    extern __shared__ __align__(16) unsigned char sm[];
    const int My = g.M[1], Mz = g.M[2], hz = Mz / 2, hy = My / 2, KM = g.K[1];
    const int x = blockIdx.x, n0 = blockIdx.y * g.ngrp, nn = min(g.ngrp, g.K[2] + 1 - n0);
    constexpr int qn = 16 / sizeof(T);  // numbers per copy
    const int t = threadIdx.x, pitch = Mz + qn, rb = min(My, g.yrows);
    // z twiddles (hz + 1) x 8 cos | sin, A[n][y], y twiddles [y][m], then the staged rows
    T* cs = reinterpret_cast<T*>(sm);
    V2* A = reinterpret_cast<V2*>(cs + (hz + 1) * 2 * kNGrp);
    V2* ty = A + kNGrp * My;
    T* rows = reinterpret_cast<T*>(ty) + ((2 * (hy + 1) * (KM + 1) + 3) & ~3);
    const int q4 = Mz / qn;
    auto stage = [&](int y0, int ny) {
        const T* src = g.grid + ((size_t)x * My + y0) * Mz;
        for (int e = t; e < ny * q4; e += 256) cp_async<16>(rows + (e / q4) * pitch + qn * (e % q4), src + qn * e);
    };
    stage(0, rb);
    for (int e = t; e < (hy + 1) * (KM + 1); e += 256) cp_async<sizeof(V2)>(ty + e, g.tw[1] + e);
    for (int e = t; e < (hz + 1) * kNGrp; e += 256) {
        const int p = e / kNGrp, k = e % kNGrp;
        const V2 w = k < nn ? __ldg(&g.tw[2][p * (g.K[2] + 1) + n0 + k]) : v2<T>(T(0), T(0));
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
        // two threads per row, each four n: neighbours in FP32 (fewer bank conflicts), in FP64 in warps of
        // their own, since a group of four n or fewer would leave every other lane of the FP64 pipe idle
        const int y = sizeof(T) == 4 ? t >> 1 : t & 127, nb = (sizeof(T) == 4 ? t & 1 : t >> 7) * 4;
        if (y < ny && nb < nn) {
            const T* r = rows + y * pitch;
            T re[4] = {0, 0, 0, 0}, im[4] = {0, 0, 0, 0};
            auto add = [&](int p, T e, T o) {
                const V4 c = *reinterpret_cast<const V4*>(cs + p * 2 * kNGrp + nb);
                const V4 s = *reinterpret_cast<const V4*>(cs + p * 2 * kNGrp + kNGrp + nb);
                re[0] = fma(e, c.x, re[0]);
                re[1] = fma(e, c.y, re[1]);
                re[2] = fma(e, c.z, re[2]);
                re[3] = fma(e, c.w, re[3]);
                im[0] = fma(o, s.x, im[0]);
                im[1] = fma(o, s.y, im[1]);
                im[2] = fma(o, s.z, im[2]);
                im[3] = fma(o, s.w, im[3]);
            };
            add(0, r[0], T(0));
#pragma unroll 4
            for (int p = 1; p < hz; ++p) {
                const T a = r[p], b = r[Mz - p];
                add(p, a + b, a - b);
            }
            add(hz, r[hz], T(0));
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (nb + k < nn) A[(nb + k) * My + y0 + y] = v2<T>(re[k], im[k]);
        }
    }
    __syncthreads();
    // fold y and My - y (over the staged rows): sum and difference side by side
    V4* F = reinterpret_cast<V4*>(rows);
    for (int e = t; e < nn * (hy + 1); e += 256) {
        const int k = e / (hy + 1), y = e % (hy + 1);
        F[k * (hy + 1) + y] = fold<T>(A[k * My + y], A[k * My + (y ? My - y : 0)], y == 0 || y == hy);
    }
    __syncthreads();
    // over y, for m and -m at once, two n per thread
    const int nm = 2 * KM + 1, half = (nn + 1) / 2;
    for (int e = t; e < (KM + 1) * half; e += 256) {
        const int m = e % (KM + 1), k0 = e / (KM + 1), k1 = min(k0 + half, nn - 1);
        Sum2<T> s;
        s.run(F + k0 * (hy + 1), F + k1 * (hy + 1), ty + m, KM + 1, hy + 1);
        V2* o = g.H + ((size_t)(n0 + k0) * g.M[0] + x) * nm + KM;
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
template <typename T>
__global__ void __launch_bounds__(256) k_nu_x(NuViewT<T> g, double* __restrict__ acc_uewa, double* __restrict__ acc_ll) {
    typedef typename NuVec<T>::V2 V2;
    typedef typename NuVec<T>::V4 V4;
    extern __shared__ __align__(16) unsigned char sm[];
    const int Mx = g.M[0], hx = Mx / 2, KL = g.K[0], nm = 2 * g.K[1] + 1, nl = 2 * KL + 1, tp = odd(KL + 1);
    const int n = blockIdx.x, m0 = blockIdx.y * g.mgrp, mm = min(g.mgrp, nm - m0);
    const int t = threadIdx.x;
    // columns [m][x]; folded columns [m][x <= hx], later [m][l]; C(k) [m][l + KL]; twiddles [x][l]
    V2* Hs = reinterpret_cast<V2*>(sm);
    V4* F = reinterpret_cast<V4*>(Hs + kMGrp * Mx);
    V2* Cs = reinterpret_cast<V2*>(F + kMGrp * (hx + 1));
    V2* tx = Cs + kMGrp * nl;
    V2* Hn = g.H + (size_t)n * Mx * nm + m0;
    for (int e = t; e < mm * Mx; e += 256) {
        const int x = e / mm, m = e % mm;
        cp_async<sizeof(V2)>(Hs + m * Mx + x, Hn + (size_t)x * nm + m);
    }
    for (int e = t; e < (hx + 1) * (KL + 1); e += 256) cp_async<sizeof(V2)>(tx + (e / (KL + 1)) * tp + e % (KL + 1), g.tw[0] + e);
    {
        const size_t n4 = (size_t)Mx * g.M[1] * g.M[2] / 4, nthr = (size_t)gridDim.x * gridDim.y * 256;
        for (size_t e = (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * 256 + t; e < n4; e += nthr)
            reinterpret_cast<V4*>(g.grid)[e] = v4<T>(T(0), T(0), T(0), T(0));
        for (size_t e = (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * 256 + t; e < (size_t)g.nblk + 1; e += nthr) {
            g.cntf[e] = g.cnt[e];
            g.cnt[e] = 0;
        }
    }
    cp_async_wait();
    __syncthreads();
    for (int e = t; e < mm * (hx + 1); e += 256) {
        const int m = e / (hx + 1), x = e % (hx + 1);
        F[e] = fold<T>(Hs[m * Mx + x], Hs[m * Mx + (x ? Mx - x : 0)], x == 0 || x == hx);
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
        Sum2<T> s2;
        s2.run(F + ma * (hx + 1), F + mb * (hx + 1), tx + l, tp, hx + 1);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int m = i ? mb : ma, am = abs(m0 + m - g.K[1]);
            const double dec = g.dec[0][l] * g.dec[1][am] * g.dec[2][n];
            const double dec2 = g.dec[0][KL + 1 + l] * g.dec[1][g.K[1] + 1 + am] * g.dec[2][g.K[2] + 1 + n];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if ((h && l == 0) || (i && ma + half >= mm)) break;
                V2 c = v2<T>(T(0), T(0));
                if (km[i][h] >= 0) {
                    const bool cj = km[i][h] & 1;
                    const V2 v = h ? s2.minus(i) : s2.plus(i);
                    double2 s = make_double2((double)v.x * dec, (double)v.y * dec);
                    if (cj) s.y = -s.y;
                    g.S[km[i][h] >> 1] = s;
                    const double2 st = make_double2(s.x + q[i][h].x, s.y + q[i][h].y);
                    const double ak = a[i][h];
                    ll += ak * (s.x * s.x + s.y * s.y);
                    ew += ak * (st.x * st.x + st.y * st.y);
                    c = v2<T>((T)(ak * st.x * dec2), (T)((cj ? ak : -ak) * st.y * dec2));
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
        F[e] = fold<T>(Cs[m * nl + KL + l], Cs[m * nl + KL - l], l == 0);
    }
    __syncthreads();
    for (int e = t; e < (hx + 1) * half; e += 256) {
        const int x = e % (hx + 1), ma = e / (hx + 1), mb = min(ma + half, mm - 1);
        Sum2<T> s;
        s.run(F + ma * (KL + 1), F + mb * (KL + 1), tx + x * tp, 1, KL + 1);
        // staged in Hs so that the stores below run along m
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            V2* o = Hs + (i ? mb : ma) * Mx;
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
template <typename T>
__global__ void __launch_bounds__(256) k_nu_yz(NuViewT<T> g) {
    typedef typename NuVec<T>::V2 V2;
    typedef typename NuVec<T>::V4 V4;
    extern __shared__ __align__(16) unsigned char sm[];
    const int My = g.M[1], Mz = g.M[2], hy = My / 2, hz = Mz / 2, KM = g.K[1], KN = g.K[2], nm = 2 * KM + 1;
    const int x = blockIdx.x, y0 = blockIdx.y * g.ygrp, ny = min(g.ygrp, hy + 1 - y0);
    const int t = threadIdx.x;
    V4* F = reinterpret_cast<V4*>(sm);     // folded [n][m]
    V2* Hs = reinterpret_cast<V2*>(F + (size_t)(KN + 1) * (KM + 1));  // [n][m + KM]
    V2* B = Hs + (size_t)(KN + 1) * nm;        // [y pair][2][n]
    V2* ty = B + 2 * g.ygrp * (KN + 1);        // y twiddles [m][y pair]
    V2* tz = ty + (KM + 1) * g.ygrp;           // z twiddles [n][z]
    for (int e = t; e < (KN + 1) * nm; e += 256) {
        const int n = e / nm, m = e % nm;
        cp_async<sizeof(V2)>(Hs + e, g.H + ((size_t)n * g.M[0] + x) * nm + m);
    }
    for (int e = t; e < (KM + 1) * ny; e += 256) cp_async<sizeof(V2)>(ty + e, g.twt[1] + (e / ny) * (hy + 1) + y0 + e % ny);
    for (int e = t; e < (KN + 1) * (hz + 1); e += 256) cp_async<sizeof(V2)>(tz + e, g.twt[2] + e);
    cp_async_wait();
    __syncthreads();
    for (int e = t; e < (KN + 1) * (KM + 1); e += 256) {
        const V2* h = Hs + (e / (KM + 1)) * nm + KM;
        const int m = e % (KM + 1);
        F[e] = fold<T>(h[m], h[-m], m == 0);
    }
    __syncthreads();
    const int half = (KN + 2) / 2;
    for (int e = t; e < half * ny; e += 256) {
        const int yi = e % ny, na = e / ny, nb = min(na + half, KN);
        Sum2<T> s;
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
        const V2* b[4];
        T u[4], v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            b[k] = B + min(r0 + k, nrow - 1) * (KN + 1);
            u[k] = b[k][0].x;
            v[k] = T(0);
        }
#pragma unroll 4
        for (int n = 1; n <= KN; ++n) {
            const V2 w = tz[n * (hz + 1) + z];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const V2 h = b[k][n];
                u[k] = fma(h.x, w.x, u[k]);
                v[k] = fma(h.y, w.y, v[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int r = r0 + k;
            if (r >= nrow) break;
            const int yp = y0 + (r >> 1), y = (r & 1) ? My - yp : yp;
            if ((r & 1) && (yp == 0 || yp == hy)) continue;
            T* o = g.pot + ((size_t)x * My + y) * Mz;
            o[z] = u[k] - v[k];
            if (z > 0 && z < hz) o[Mz - z] = u[k] + v[k];
        }
    }
}

// What both plans share: sizes, the map from (n, m, l) to the k set, twiddles, arrays, groups.  rule(K): grid
// points of a direction; inverse(h, k, M): 1 / transform of the spreading (h = 0) and the force window.
template <typename T, typename Rule, typename Inverse>
int nu_setup(Ctx& c, NuPlanT<T>& plan, Rule rule, Inverse inverse) {
    typedef typename NuVec<T>::V2 V2;
    View& v = c.v;
    KSet& ks = c.ks;
    NuViewT<T>& g = plan.g;
    const int K[3] = {ks.klmax, ks.kmmax, ks.knmax};
    const double pip[3] = {ks.pipix, ks.pipiy, ks.pipiz}, len[3] = {v.lx, v.ly, v.lz};
    size_t npts = 1, nblk = 1;
    double cell = 1.0;
    for (int d = 0; d < 3; ++d) {
        g.K[d] = K[d];
        g.M[d] = rule(K[d]);
        g.n8[d] = (g.M[d] + 7) / 8;
        g.scale[d] = (T)(g.M[d] * pip[d] / (2.0 * 3.14159265358979323846));
        npts *= g.M[d];
        nblk *= g.n8[d];
        cell *= 8.0 * len[d] / g.M[d];
    }
    // bucket room: three times the mean, or three times a dense liquid's 0.11 atoms / A^3
    const double want = 3.0 * std::max((double)v.nmove / (double)nblk, 0.11 * cell) + 16.0;
    g.cap = (int)std::min<double>(want, v.nmove);
    g.nblk = (int)nblk;
    // CTAs per block: for kSplit atoms each, for 912 in all, and where most of the box is empty for 340 over the blocks
    // that a liquid would fill (with no more than 4,096 in all, most of which have nothing to do).  Slabs of 4,000 and 1,400 waters in boxes 4.5 and 9 edges tall (mixed, a force call):
    // by the box's mean density 118 and 83 us, this 98 and 81 (912 over the filled blocks 104 and 97).
    const double dense = std::max((double)v.nmove / (double)nblk, 0.1 * cell), full = std::max(v.nmove / dense, 1.0);
    g.split = std::max({(int)(dense / kSplit) + 1, (int)(912 / nblk), std::min((int)(340.0 / full), (int)(4096 / nblk))});
    g.split = std::min(g.split, 64);
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
        std::vector<V2> a((size_t)(h + 1) * k1), b(a.size());
        std::vector<double> dec(2 * k1);
        for (int p = 0; p <= h; ++p)
            for (int k = 0; k < k1; ++k) {
                const double w = 2.0 * 3.14159265358979323846 * (double)((long)p * k % g.M[d]) / g.M[d];
                a[(size_t)p * k1 + k] = b[(size_t)k * (h + 1) + p] = V2{(T)std::cos(w), (T)std::sin(w)};
            }
        for (int k = 0; k < k1; ++k) {
            dec[k] = inverse(0, k, g.M[d]);
            dec[k1 + k] = inverse(1, k, g.M[d]);
        }
        g.tw[d] = (V2*)put(a.data(), sizeof(V2) * a.size());
        g.twt[d] = (V2*)put(b.data(), sizeof(V2) * b.size());
        g.dec[d] = (double*)put(dec.data(), sizeof(double) * dec.size());
    }
    g.grid = (T*)dalloc(c, sizeof(T) * npts);
    g.pot = (T*)dalloc(c, sizeof(T) * npts);
    g.H = (V2*)dalloc(c, sizeof(V2) * (size_t)(K[2] + 1) * g.M[0] * nm);
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
    while (g.yrows > 32 && (fixed + g.yrows * (g.M[2] + 4)) * (int)sizeof(T) > 110 * 1024) g.yrows /= 2;
    plan.smem_zy = (fixed + std::max(g.yrows * (g.M[2] + 4), 4 * kNGrp * hy1)) * (int)sizeof(T);
    plan.smem_x = (kMGrp * (g.M[0] + 2 * (g.M[0] / 2 + 1) + nl) + (g.M[0] / 2 + 1) * ((K[0] + 1) | 1)) * (int)sizeof(V2);
    plan.smem_yz = ((K[2] + 1) * (2 * (K[1] + 1) + nm + 2 * g.ygrp + g.M[2] / 2 + 1) + (K[1] + 1) * g.ygrp) * (int)sizeof(V2);
    MDG_CUDA(allow_max_smem(k_nu_zy<T>));
    MDG_CUDA(allow_max_smem(k_nu_x<T>));
    MDG_CUDA(allow_max_smem(k_nu_yz<T>));
    if (std::max(plan.smem_zy, std::max(plan.smem_x, plan.smem_yz)) > 227 * 1024)
        return set_err(&c, MDG_E_UNSUPPORTED, "k range too large for the shared-memory tables of the reciprocal sum");
    plan.ready = true;
    return MDG_OK;
}


// The three sums between the atoms' charges on the grid and the potential on it.
template <typename T>
void nu_fourier(Ctx& c, const NuPlanT<T>& plan) {
    const NuViewT<T>& g = plan.g;
    const int nm = 2 * g.K[1] + 1;
    double* acc = c.v.acc + 2 * c.v.nijt;
    k_nu_zy<T><<<dim3(g.M[0], (g.K[2] + g.ngrp) / g.ngrp), 256, plan.smem_zy, c.stream>>>(g);
    k_nu_x<T><<<dim3(g.K[2] + 1, (nm + g.mgrp - 1) / g.mgrp), 256, plan.smem_x, c.stream>>>(g, acc + ACC_UEWA, acc + ACC_EWQLL);
    k_nu_yz<T><<<dim3(g.M[0], (g.M[1] / 2 + 1 + g.ygrp - 1) / g.ygrp), 256, plan.smem_yz, c.stream>>>(g);
}

}  // namespace mdg
