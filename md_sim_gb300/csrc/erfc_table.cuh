// erfc_table.cuh - the Ewald real-space functions of a site pair from a table in (alpha r)^2.
//
// With y = (alpha r)^2 and the erfc of Abramowitz-Stegun 7.1.26 that the reference uses
// (src/forcem.f90:334-340), a pair of charges needs
//   G(y) = erfc(x) / x                                    energy / (alpha q q'),
//   H(y) = (2/sqrt(pi) x exp(-y) + erfc(x)) / x^3         force  / (alpha^3 q q' d),   x = sqrt(y).
// Evaluated directly they take a reciprocal square root, a division, an exponential and the
// polynomial: about 55 FP64 operations, and FP64 operations are what bounds the loops that use them
// (1.6 lanes per clock per SM).  Each octave of y is cut into 128 intervals with degree-6 Chebyshev
// interpolants of both about the interval's centre: one row of 128 bytes per interval, 12 FMAs and one
// subtraction.  Against 64-bit-mantissa arithmetic the rows are within 3e-16 of both functions (5e-16 from
// y = 8 on), the direct form, which rounds at every step, within 3e-15 (6e-15).  Outside
// 2^-4 <= y < 2^4 (r from 0.8 to 12.5 A at alpha = 0.32) and for NaN the direct form runs.
#pragma once

#include <cmath>
#include <vector>

#include "common.cuh"

namespace mdg {

constexpr int kEtLo = -4, kEtHi = 4;               // octaves of y
constexpr int kEtRows = (kEtHi - kEtLo) * 128;      // 128 KB
constexpr int kEtDeg = 6;

// Direct form: (G, H) at y.
static __device__ __noinline__ double2 ewald_direct(double y, double spii) {
    const double xi = rsqrt(y), x = y * xi;
    const double t = 1.0 / (1.0 + kP * x);
    const double e = exp(-y);
    const double f = ((((kA5 * t + kA4) * t + kA3) * t + kA2) * t + kA1) * t * e;
    return make_double2(f * xi, (spii * x * e + f) * (xi * (xi * xi)));
}

// Row of y and its offset from the row's centre; false where the table does not reach.
__device__ __forceinline__ bool ewald_row(double y, const double2* tab, const double2*& row, double& u) {
    const int hi = __double2hiint(y);
    const unsigned k = (unsigned)((hi >> 13) - ((1023 + kEtLo) << 7));
    u = y - __hiloint2double((hi & ~0x1fff) | 0x1000, 0);
    row = tab + 8 * (size_t)(k < (unsigned)kEtRows ? k : 0u);
    return k < (unsigned)kEtRows;
}

__device__ __forceinline__ double2 ewald_gh(double y, const double2* __restrict__ tab, double spii) {
    const double2* r;
    double u;
    if (!ewald_row(y, tab, r, u)) return ewald_direct(y, spii);
    const double2 a = r[0], b = r[1], c = r[2], d = r[3], e = r[4], f = r[5], g = r[6];
    // the row: g0 g1 .. g6, h0 .. h6
    return make_double2(((((((d.x * u + c.y) * u + c.x) * u + b.y) * u + b.x) * u + a.y) * u + a.x),
                        ((((((g.y * u + g.x) * u + f.y) * u + f.x) * u + e.y) * u + e.x) * u + d.y));
}

__device__ __forceinline__ double ewald_g(double y, const double2* __restrict__ tab, double spii) {
    const double2* r;
    double u;
    if (!ewald_row(y, tab, r, u)) return ewald_direct(y, spii).x;
    const double2 a = r[0], b = r[1], c = r[2], d = r[3];
    return ((((((d.x * u + c.y) * u + c.x) * u + b.y) * u + b.x) * u + a.y) * u + a.x);
}

// Rows of 16 doubles (14 used).  spii: the reference's 2/sqrt(pi).
inline std::vector<double> ewald_table(double spii) {
    std::vector<double> t((size_t)kEtRows * 16, 0.0);
    constexpr int n = kEtDeg + 1;
    for (int k = 0; k < kEtRows; ++k) {
        const long double w = std::ldexp(1.0L / 128, kEtLo + k / 128), h = w / 2;
        const long double y0 = std::ldexp(1.0L, kEtLo + k / 128) + w * (k % 128) + h;
        long double u[n], f[2][n];
        for (int i = 0; i < n; ++i) {
            u[i] = h * std::cos(3.14159265358979323846L * (i + 0.5L) / n);
            const long double y = y0 + u[i], x = std::sqrt(y), e = std::exp(-y), s = 1 / (1 + kP * x);
            const long double p = ((((kA5 * s + kA4) * s + kA3) * s + kA2) * s + kA1) * s * e;
            f[0][i] = p / x;
            f[1][i] = (spii * x * e + p) / (x * y);
        }
        for (int d = 0; d < 2; ++d) {
            for (int j = 1; j < n; ++j)  // Newton's divided differences
                for (int i = n - 1; i >= j; --i) f[d][i] = (f[d][i] - f[d][i - 1]) / (u[i] - u[i - j]);
            long double c[n] = {f[d][n - 1]};  // to powers of u
            for (int j = n - 2, m = 0; j >= 0; --j) {
                ++m;
                for (int i = m; i > 0; --i) c[i] = c[i - 1] - u[j] * (i < m ? c[i] : 0.0L);
                c[0] = f[d][j] - u[j] * c[0];
            }
            for (int i = 0; i < n; ++i) t[16 * (size_t)k + 7 * d + i] = (double)c[i];
        }
    }
    return t;
}

}  // namespace mdg
