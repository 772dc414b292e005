// integrate.cu - the MD step around the force phases, on the device (resident mode).
//
//   k_pred   move_predict, src/move.f90:48-217: 5-value Gear predictor for ions, centres of mass,
//            angular velocities and quaternions; quaternion normalisation, rotation matrix, site
//            rebuild and the H offsets rsx (:148-162); the block that finishes last computes the
//            kinetic energies, the Nose-like thermostat predictor, htot and sft/sfr.
//   k_corr   move_correct, src/move.f90:220-383, for ions and rigid molecules; its last block adds
//            uconf and press of force_sum (src/forcem.f90:1055,1079,1081) and the thermostat
//            corrector.
//
// Systems of more than 80 molecules per SM: one thread per ion or molecule in blocks of four warps, where
// FP64 operations bound them.  Smaller ones (k_pred_small, k_corr_small): what bounds these is the chain of
// dependent instructions of one molecule (a warp issued one instruction per 14 clocks), so a block of five
// warps takes 16 molecules and a thread one component of one of them (3 of the centre, 3 of the angular
// velocity, 4 of the quaternion) through the Gear arithmetic, the forces of one site, the placing and
// packing of one atom: 2,048 waters between walls k_pred 16.4 -> 8.1 us, k_corr 17.3 -> 9.8 us against two
// lanes per molecule with 14 molecules per warp; 20 resident steps 1.99 -> 1.73 ms.
// Kinetic sums go through reductions into a small accumulator array that the last block reads and
// clears.  Gear coefficients are the reference's single-precision literals.
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "lr_tail.cuh"
#include "merge.cuh"
#include "pack.cuh"

namespace mdg {

namespace {

constexpr int kSM = 152;

// unit served by this thread in sweep `r` of the grid-stride loop over the first `nb` blocks
template <int NT>
__device__ __forceinline__ int unit_of(int r, int nb) {
    return (r * nb + blockIdx.x) * NT + threadIdx.x;
}

constexpr double Gf01 = F32D(0.348611111), Gf11 = 1.0, Gf21 = F32D(0.916666667), Gf31 = F32D(0.333333333),
                 Gf41 = F32D(0.041666667);
constexpr double Gf02 = F32D(0.158300000), Gf12 = F32D(0.757000000), Gf22 = 1.0, Gf32 = 0.5,
                 Gf42 = F32D(0.083333333);

__device__ __forceinline__ void gpred(double& a0, double& a1, double& a2, double& a3, double a4) {
    a0 = a0 + a1 + a2 + a3 + a4;
    a1 = a1 + 2 * a2 + 3 * a3 + 4 * a4;
    a2 = a2 + 3 * a3 + 6 * a4;
    a3 = a3 + 4 * a4;
}

struct Dyn {
    unsigned* done;  // [2] blocks finished (k_pred, k_corr), reset by the last block
    double* xd;     // [4][3][nion]
    double* c;      // [5][3][nrig]
    double* q;      // [4][5][nrig]
    double* w;      // [5][3][nrig]
    double* a;      // [9][nrig]
    double* th;     // thermostat + scalars
    double* isum;   // kinetic partial sums
    const double* ft;  // 3 x nflex
    const double* fc;  // 3 x nrig
    const double* tq;  // 3 x nrig
    mdg_rigid body;
    int nion;
};

__device__ __forceinline__ double pred_ion(const View& v, const Dyn& D, int k, double* xn) {
    const int n = D.nion;
    const int i = v.nriga + k;
    double* X[3] = {v.x, v.y, v.z};
    double s2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double* x1 = D.xd + (0 * 3 + d) * n;
        double* x2 = D.xd + (1 * 3 + d) * n;
        double* x3 = D.xd + (2 * 3 + d) * n;
        double* x4 = D.xd + (3 * 3 + d) * n;
        double a0 = X[d][i], a1 = x1[k], a2 = x2[k], a3 = x3[k];
        gpred(a0, a1, a2, a3, x4[k]);
        X[d][i] = a0;
        xn[d] = a0;
        x1[k] = a1;
        x2[k] = a2;
        x3[k] = a3;
        s2 += a1 * a1;
    }
    return v.mi[i] * s2;
}

// True in every thread of the block that finished last; each block's atomics are visible before
// it counts itself done.
__device__ __forceinline__ bool last_block(unsigned* done, int nblk) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1u) == nblk - 1;
    __syncthreads();
    return last;
}

// rotation matrix of the normalised predicted quaternion (src/move.f90:128-146)
__device__ __forceinline__ void quat_rot(const double* qq, double* qn, double* a) {
    const double cr = 1.0 / sqrt(qq[0] * qq[0] + qq[1] * qq[1] + qq[2] * qq[2] + qq[3] * qq[3]);
    const double q1 = qq[0] * cr, q2 = qq[1] * cr, q3 = qq[2] * cr, q4 = qq[3] * cr;
    qn[0] = q1;
    qn[1] = q2;
    qn[2] = q3;
    qn[3] = q4;
    a[0] = -q1 * q1 + q2 * q2 - q3 * q3 + q4 * q4;
    a[1] = 2.0 * (q3 * q4 - q1 * q2);
    a[2] = 2.0 * (q2 * q3 + q1 * q4);
    a[3] = -2.0 * (q1 * q2 + q3 * q4);
    a[4] = q1 * q1 - q2 * q2 - q3 * q3 + q4 * q4;
    a[5] = 2.0 * (q2 * q4 - q1 * q3);
    a[6] = 2.0 * (q2 * q3 - q1 * q4);
    a[7] = -2.0 * (q1 * q3 + q4 * q2);
    a[8] = -q1 * q1 - q2 * q2 + q3 * q3 + q4 * q4;
}

// lab-frame position of site j (src/move.f90:148-162)
__device__ __forceinline__ void site_pos(const double* cx, const double* a, const mdg_rigid& b, int j, double& x,
                                         double& y, double& z) {
    x = cx[0] + a[0] * b.xbody[j] + a[3] * b.ybody[j] + a[6] * b.zbody[j];
    y = cx[1] + a[1] * b.xbody[j] + a[4] * b.ybody[j] + a[7] * b.zbody[j];
    z = cx[2] + a[2] * b.xbody[j] + a[5] * b.ybody[j] + a[8] * b.zbody[j];
}

__device__ __forceinline__ void load_cw(const Dyn& D, int nr, int i, double (&C)[5][3], double (&W)[5][3]) {
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            C[k][d] = D.c[(k * 3 + d) * nr + i];
            W[k][d] = D.w[(k * 3 + d) * nr + i];
        }
}

__device__ __forceinline__ void load_q(const Dyn& D, int nr, int i, double (&Q)[5][4]) {
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) Q[k][cc] = D.q[(cc * 5 + k) * nr + i];
}

// predictor of the centre and angular velocity; stores their first four derivatives
__device__ __forceinline__ void pred_cw(const Dyn& D, int nr, int i, double (&C)[5][3], double (&W)[5][3], double* sc,
                                        double* sw, double* cx) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        gpred(C[0][d], C[1][d], C[2][d], C[3][d], C[4][d]);
        sc[d] += C[1][d] * C[1][d];
        cx[d] = C[0][d];
        gpred(W[0][d], W[1][d], W[2][d], W[3][d], W[4][d]);
        sw[d] += W[0][d] * W[0][d];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
#pragma unroll
        for (int k = 0; k < 4; ++k) D.c[(k * 3 + d) * nr + i] = C[k][d];
#pragma unroll
        for (int k = 0; k < 4; ++k) D.w[(k * 3 + d) * nr + i] = W[k][d];
    }
}

// predictor of the orientation; stores the quaternion derivatives and the rotation matrix
__device__ __forceinline__ void pred_q(const Dyn& D, int nr, int i, double (&Q)[5][4], double* a) {
    double qq[4], qn[4];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        gpred(Q[0][cc], Q[1][cc], Q[2][cc], Q[3][cc], Q[4][cc]);
        qq[cc] = Q[0][cc];
    }
    quat_rot(qq, qn, a);
#pragma unroll
    for (int cc = 0; cc < 4; ++cc)
#pragma unroll
        for (int k = 1; k < 4; ++k) D.q[(cc * 5 + k) * nr + i] = Q[k][cc];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) D.q[(cc * 5) * nr + i] = qn[cc];
#pragma unroll
    for (int k = 0; k < 9; ++k) D.a[k * nr + i] = a[k];
}

// All of a molecule's state is loaded before anything is stored: the arrays may alias as far as
// the compiler knows, and loads issued back to back overlap their latency instead of queueing
// behind the stores (the per-molecule work is short; memory latency, not FP64, bounds it).
__device__ __forceinline__ void pred_rigid(const View& v, const Dyn& D, int i, double* sc, double* sw, double* cn,
                                           double* sx, double* sy, double* sz) {
    const int nr = v.nrig;
    double C[5][3], W[5][3], Q[5][4], a[9];
    load_cw(D, nr, i, C, W);
    load_q(D, nr, i, Q);
    pred_cw(D, nr, i, C, W, sc, sw, cn);
    pred_q(D, nr, i, Q, a);
    const int ix = 3 * i;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        site_pos(cn, a, D.body, j, sx[j], sy[j], sz[j]);
        v.x[ix + j] = sx[j];
        v.y[ix + j] = sy[j];
        v.z[ix + j] = sz[j];
    }
#pragma unroll
    for (int j = 1; j < 3; ++j) {
        v.rsx[ix + j] = sx[j] - sx[0];
        v.rsy[ix + j] = sy[j] - sy[0];
        v.rsz[ix + j] = sz[j] - sz[0];
    }
}

// thermostat predictor and kinetic energies from the summed isum[0..6] (one thread).  Runs in the
// tail of a kernel, where every dependent round trip to L2 is about a microsecond: all loads are
// issued first, into registers, then the arithmetic, then the stores.
struct ThermoIn {
    double is[7], s[5], rs[5], uc;
};

__device__ __forceinline__ ThermoIn thermo_pred_load(const Dyn& D) {
    ThermoIn t;
#pragma unroll
    for (int k = 0; k < 7; ++k) t.is[k] = __ldcg(&D.isum[k]);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        t.s[k] = __ldcg(&D.th[TH_S + k]);
        t.rs[k] = __ldcg(&D.th[TH_RS + k]);
    }
    t.uc = __ldcg(&D.th[TH_UCONF]);
    return t;
}

__device__ void thermo_pred(const View& v, const Dyn& D, ThermoIn t) {
    double* th = D.th;
    const mdg_rigid& b = D.body;
    double* is = t.is;
    double* s = t.s;
    double* rs = t.rs;
    const double uc = t.uc;
    const double kp = is[0] + b.mw * (is[1] + is[2] + is[3]);
    const double kw = b.inxx * is[4] + b.inyy * is[5] + b.inzz * is[6];
    if (b.temper == -1.0) {
        s[0] = s[1] = rs[0] = rs[1] = 0.0;
    } else {
        gpred(s[0], s[1], s[2], s[3], s[4]);
        gpred(rs[0], rs[1], rs[2], rs[3], rs[4]);
    }
    const long nfree = v.nliqa - v.nriga;
    const double tstar = F32D(8.31441) * b.temper / 1000.0;
    double qmass = (double)(float)(3 * (nfree + v.nrig)) * tstar * F32D(2e3);
    double rmass = (double)(float)(3 * v.nrig) * tstar * F32D(1e3);
    qmass = qmass / 10.0;
    rmass = rmass / 10.0;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        th[TH_S + k] = s[k];
        th[TH_RS + k] = rs[k];
    }
    th[TH_KP] = kp;
    th[TH_KW] = kw;
    th[TH_KE] = kp + kw;
    th[TH_HTOT] = 0.5 * (kp + kw + qmass * s[0] * s[0] + rmass * rs[0] * rs[0]) + uc;
    th[TH_SFT] = (kp - (double)(float)(3 * (nfree + v.nrig) - 2) * tstar) / qmass;
    th[TH_SFR] = (kw - (double)(float)(3 * v.nrig + 1) * tstar) / rmass;
#pragma unroll
    for (int k = 0; k < 7; ++k) D.isum[k] = 0.0;  // ready for the next step
}

// Sums that the rest of the step accumulates into, zeroed by the predictor (block 0) so that the
// step graph needs no memset nodes.
struct Clear {
    double* p[2];
    int n[2];
};

// The records of the force evaluation that follows (pack.cuh), written by the predictor of a
// resident mixed-precision step from the positions it has just computed: blocks below npred
// predict and pack their molecules and flexible atoms, the blocks after them pack the wall atoms.
struct PackArgs {
    Pk pk;
    int dip;    // slab dipole term
    int npred;  // blocks of the predictor proper
};

// A packing predictor has no tail: block 0 clears the energy sums first (all but the displacement
// maximum, which the blocks raise as they go), and the close of the packing and the thermostat
// predictor run in k_step_close on the list's stream, off the path of the reciprocal sum.
//
// First block of a predictor: the sums that the step adds to.
template <bool PACK>
__device__ __forceinline__ void pred_clear(const View& v, const Clear& z, const PackArgs& P) {
    for (int j = 0; j < 2; ++j)
        for (int k = threadIdx.x; k < z.n[j]; k += blockDim.x) z.p[j][k] = 0.0;
    if constexpr (PACK) {
        const int na = 2 * v.nijt + ACC_NSLOT, kmax = 2 * v.nijt + ACC_MAXD;
        for (int k = threadIdx.x; k < na; k += blockDim.x)
            if (k != kmax) v.acc[k] = 0.0;
        if (P.pk.cmax && threadIdx.x == 0) *P.pk.cmax = 0.f;
    }
}

// ion u with its record; its share of kp, the dipole and the displacement maximum
template <bool PACK>
__device__ __forceinline__ void pred_ion_pack(const View& v, const Dyn& D, const PackArgs& P, int u, double& kp, double& mz,
                                              double& md) {
    double xn[3];
    kp += pred_ion(v, D, u, xn);
    if constexpr (PACK) {
        const int at = v.nriga + u;
        const double a = v.ox[u] - xn[0], b = v.oy[u] - xn[1], c = v.oz[u] - xn[2];
        md = fmax(md, a * a + b * b + c * c);
        mz += pack_atom(v, P.pk, at, xn[0], xn[1], xn[2], v.rsx[at], v.rsy[at], v.rsz[at], true);
    }
}

template <bool PACK>
__device__ __forceinline__ void pred_end(const View& v, const Dyn& D, const PackArgs& P, double mz, double md, double* red,
                                         int bid, int nblk) {
    if constexpr (PACK) {
        pack_block(v, P.pk, mz, md, red, bid);
    } else if (last_block(&D.done[0], nblk) && threadIdx.x == 0) {
        thermo_pred(v, D, thermo_pred_load(D));
        D.done[0] = 0u;
    }
}

template <int NT, bool PACK>
__global__ void __launch_bounds__(NT) k_pred(View v, Dyn D, Clear z, PackArgs P) {
    __shared__ double red[8];
    double kp = 0.0, sc[3] = {0, 0, 0}, sw[3] = {0, 0, 0};
    double mz = 0.0, md = 0.0;
    const int nu = D.nion + v.nrig;
    const int npred = PACK ? P.npred : gridDim.x;
    if (blockIdx.x == 0) pred_clear<PACK>(v, z, P);
    if (blockIdx.x < npred) {
        for (int r = 0;; ++r) {
            const int u = unit_of<NT>(r, npred);
            if (u >= nu) break;
            if (u < D.nion) {
                pred_ion_pack<PACK>(v, D, P, u, kp, mz, md);
                continue;
            }
            const int i = u - D.nion, ix = 3 * i;
            double cn[3], px[3], py[3], pz[3];
            pred_rigid(v, D, i, sc, sw, cn, px, py, pz);
            if constexpr (PACK) {
                // site 0's offset is the stored one (force_sum leaves rsx(1:3) stale), the others
                // the offsets just computed, as the packing kernel would read them back
                const double a = v.ocx[i] - cn[0], b = v.ocy[i] - cn[1], c = v.ocz[i] - cn[2];
                md = fmax(md, a * a + b * b + c * c);
                mz += pack_atom(v, P.pk, ix, px[0], py[0], pz[0], v.rsx[ix], v.rsy[ix], v.rsz[ix], true);
#pragma unroll
                for (int j = 1; j < 3; ++j)
                    mz += pack_atom(v, P.pk, ix + j, px[j], py[j], pz[j], px[j] - px[0], py[j] - py[0],
                                    pz[j] - pz[0], true);
            }
        }
    } else if constexpr (PACK) {
        const int nw = gridDim.x - npred;
        for (int a = v.nmove + (blockIdx.x - npred) * NT + threadIdx.x; a < v.ntota; a += nw * NT)
            pack_atom(v, P.pk, a, v.x[a], v.y[a], v.z[a], 0.0, 0.0, 0.0, false);
    }
    if (blockIdx.x < npred) {
        double t[8] = {kp, sc[0], sc[1], sc[2], sw[0], sw[1], sw[2], 0.0};
        const double sum = warp_sums(t);
        const int lane = threadIdx.x & 31;
        if ((lane & 3) == 0 && lane < 28) atomicAdd(&D.isum[lane >> 2], sum);
    }
    pred_end<PACK>(v, D, P, mz, md, red, blockIdx.x, gridDim.x);
}

// ---- small systems -----------------------------------------------------------------------------
constexpr int kMol = 16, kComp = 10, kST = kMol * kComp;  // molecules, components, threads of a block
constexpr int kFlex = 32;                                 // ions or surface atoms of a block that takes those

// Component k of molecule i: its derivatives are st apart from the returned pointer on.
__device__ __forceinline__ double* component(const Dyn& D, int nr, int i, int k, int& st) {
    st = k < 6 ? 3 * nr : nr;
    return (k < 3 ? D.c + (size_t)k * nr : k < 6 ? D.w + (size_t)(k - 3) * nr : D.q + (size_t)(k - 6) * 5 * nr) + i;
}

// Sum over the 16 lanes of a component.
__device__ __forceinline__ double sum16(double x) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Blocks below nrb: 16 molecules each; below nrb + nfb: ions; then (PACK) wall atoms.
template <bool PACK>
__device__ __forceinline__ void pred_small(const View& v, const Dyn& D, const Clear& z, const PackArgs& P, int nrb, int nfb,
                                           int bid, int nblk) {
    __shared__ double red[8], s_c[3][kMol], s_q[4][kMol], s_a[9][kMol];
    double mz = 0.0, md = 0.0;
    const int t = threadIdx.x;
    if (bid == 0) pred_clear<PACK>(v, z, P);
    if (bid < nrb) {
        const int m = t & (kMol - 1), k = t / kMol, nr = v.nrig, i = bid * kMol + m;
        const bool act = i < nr;
        int st;
        double* b = component(D, nr, act ? i : 0, k, st);
        double a0 = b[0], a1 = b[st], a2 = b[2 * st], a3 = b[3 * (size_t)st];
        gpred(a0, a1, a2, a3, b[4 * (size_t)st]);
        if (k < 3) s_c[k][m] = a0;
        if (k >= 6) s_q[k - 6][m] = a0;
        __syncthreads();
        if (act) {
            if (k < 6) b[0] = a0;
            b[st] = a1;
            b[2 * st] = a2;
            b[3 * (size_t)st] = a3;
        }
        if (t >= kST - 32) {  // the warp with the last two quaternion components: no kinetic sums there
            if (t < kST - kMol) {
                double qq[4], qn[4], a[9];
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) qq[cc] = s_q[cc][m];
                quat_rot(qq, qn, a);
#pragma unroll
                for (int e = 0; e < 9; ++e) s_a[e][m] = a[e];
                if (act)
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) D.q[(size_t)(cc * 5) * nr + i] = qn[cc];
            }
        } else {
            const double x = k < 3 ? a1 : a0;  // d/dt of the centre, angular velocity
            const double s = sum16(act && k < 6 ? x * x : 0.0);
            if (m == 0 && k < 6) atomicAdd(&D.isum[1 + k], s);
        }
        __syncthreads();
        if (act && k < 9) D.a[(size_t)k * nr + i] = s_a[k][m];
        if (act && k < 3) {
            double cn[3], a[9], p0[3], p[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) cn[d] = s_c[d][m];
#pragma unroll
            for (int e = 0; e < 9; ++e) a[e] = s_a[e][m];
            const int ix = 3 * i;
            site_pos(cn, a, D.body, 0, p0[0], p0[1], p0[2]);
            site_pos(cn, a, D.body, k, p[0], p[1], p[2]);
            v.x[ix + k] = p[0];
            v.y[ix + k] = p[1];
            v.z[ix + k] = p[2];
            double rx = 0.0, ry = 0.0, rz = 0.0;
            if (k > 0) {
                v.rsx[ix + k] = rx = p[0] - p0[0];
                v.rsy[ix + k] = ry = p[1] - p0[1];
                v.rsz[ix + k] = rz = p[2] - p0[2];
            }
            if constexpr (PACK) {
                if (k == 0) {
                    // site 0's offset is the stored one (force_sum leaves rsx(1:3) stale)
                    rx = v.rsx[ix];
                    ry = v.rsy[ix];
                    rz = v.rsz[ix];
                    const double dx = v.ocx[i] - cn[0], dy = v.ocy[i] - cn[1], dz = v.ocz[i] - cn[2];
                    md = dx * dx + dy * dy + dz * dz;
                }
                mz = pack_atom(v, P.pk, ix + k, p[0], p[1], p[2], rx, ry, rz, true);
            }
        }
    } else if (bid < nrb + nfb) {
        const int u = (bid - nrb) * kFlex + t;
        double kp = 0.0;
        if (t < kFlex && u < D.nion) pred_ion_pack<PACK>(v, D, P, u, kp, mz, md);
        if (t < kFlex) {
            kp = warp_sum(kp);
            if (t == 0) atomicAdd(&D.isum[0], kp);
        }
    } else if constexpr (PACK) {
        const int b0 = nrb + nfb, nw = nblk - b0;
        for (int a = v.nmove + (bid - b0) * kST + t; a < v.ntota; a += nw * kST)
            pack_atom(v, P.pk, a, v.x[a], v.y[a], v.z[a], 0.0, 0.0, 0.0, false);
    }
    pred_end<PACK>(v, D, P, mz, md, red, bid, nblk);
}

template <bool PACK>
__global__ void __launch_bounds__(kST) k_pred_small(View v, Dyn D, Clear z, PackArgs P, int nrb, int nfb) {
    pred_small<PACK>(v, D, z, P, nrb, nfb, blockIdx.x, gridDim.x);
}

// After a packing predictor (one block of two warps): the close of its packing (slab dipole from
// the nparts block shares, list rebuild decision) on one warp and the thermostat predictor on the
// other.
__device__ __forceinline__ void step_close(const View& v, const Dyn& D, const Pk& pk, int dip, int nparts) {
    if (threadIdx.x < 32) {
        pack_close_warp(v, pk, dip, 0, 0, nparts, false);
    } else if (threadIdx.x == 32) {
        thermo_pred(v, D, thermo_pred_load(D));
    }
}

__global__ void __launch_bounds__(64) k_step_close(View v, Dyn D, Pk pk, int dip, int nparts) {
    step_close(v, D, pk, dip, nparts);
}

__device__ __forceinline__ void corr_ion(const View& v, const Dyn& D, int k) {
    const int n = D.nion;
    const double s0i = D.th[TH_S];
    const int nflex = v.nmove - v.nriga;
    {
        const int i = v.nriga + k;
        double* X[3] = {v.x, v.y, v.z};
        for (int d = 0; d < 3; ++d) {
            double* x1 = D.xd + (0 * 3 + d) * n;
            double* x2 = D.xd + (1 * 3 + d) * n;
            double* x3 = D.xd + (2 * 3 + d) * n;
            double* x4 = D.xd + (3 * 3 + d) * n;
            const double cort = 0.5 * D.ft[d * nflex + k] * v.mii[i] - x1[k] * s0i - x2[k];
            X[d][i] = X[d][i] + Gf02 * cort;
            x1[k] = x1[k] + Gf12 * cort;
            x2[k] = x2[k] + Gf22 * cort;
            x3[k] = x3[k] + Gf32 * cort;
            x4[k] = x4[k] + Gf42 * cort;
        }
    }
}

// corrector of the orientation (Q and the predicted angular velocity w0); stores its derivatives
__device__ __forceinline__ void corr_q(const Dyn& D, int nr, int i, double (&Q)[5][4], const double* w0) {
    const double q1 = Q[0][0], q2 = Q[0][1], q3 = Q[0][2], q4 = Q[0][3];
    const double wx = w0[0], wy = w0[1], wz = w0[2];
    double cq[4];
    cq[0] = 0.5 * (-q3 * wx - q4 * wy + q2 * wz);
    cq[1] = 0.5 * (q4 * wx - q3 * wy - q1 * wz);
    cq[2] = 0.5 * (q1 * wx + q2 * wy + q4 * wz);
    cq[3] = 0.5 * (-q2 * wx + q1 * wy - q3 * wz);
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        const double co = cq[cc] - Q[1][cc];
        Q[0][cc] = Q[0][cc] + Gf01 * co;
        Q[1][cc] = Q[1][cc] + Gf11 * co;
        Q[2][cc] = Q[2][cc] + Gf21 * co;
        Q[3][cc] = Q[3][cc] + Gf31 * co;
        Q[4][cc] = Q[4][cc] + Gf41 * co;
    }
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) D.q[(cc * 5 + k) * nr + i] = Q[k][cc];
}

// corrector of the centre (force fc) and the angular velocity (torque tq through the rotation
// matrix a); stores their derivatives
__device__ __forceinline__ void corr_cw(const Dyn& D, int nr, int i, double (&C)[5][3], double (&W)[5][3],
                                        const double* a, const double* fc, const double* tq, double s0i,
                                        double rs0i) {
    const mdg_rigid& b = D.body;
    const double rcorr = 0.5 / b.mw;
    const double inxxi = 1.0 / b.inxx, inyyi = 1.0 / b.inyy, inzzi = 1.0 / b.inzz;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const double co = rcorr * fc[d] - C[1][d] * s0i - C[2][d];
        C[0][d] = C[0][d] + Gf02 * co;
        C[1][d] = C[1][d] + Gf12 * co;
        C[2][d] = C[2][d] + Gf22 * co;
        C[3][d] = C[3][d] + Gf32 * co;
        C[4][d] = C[4][d] + Gf42 * co;
    }
    const double wx = W[0][0], wy = W[0][1], wz = W[0][2];
    const double tx = tq[0], ty = tq[1], tz = tq[2];
    double c1 = a[0] * tx + a[1] * ty + a[2] * tz;
    c1 = ((c1 * 1.0 + wy * wz * (b.inyy - b.inzz)) * inxxi) - W[1][0] - rs0i * wx;
    double c2 = a[3] * tx + a[4] * ty + a[5] * tz;
    c2 = ((c2 * 1.0 + wz * wx * (b.inzz - b.inxx)) * inyyi) - W[1][1] - rs0i * wy;
    double c3 = a[6] * tx + a[7] * ty + a[8] * tz;
    c3 = ((c3 * 1.0 + wx * wy * (b.inxx - b.inyy)) * inzzi) - W[1][2] - rs0i * wz;
    const double cw[3] = {c1, c2, c3};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        W[0][d] += Gf01 * cw[d];
        W[1][d] += Gf11 * cw[d];
        W[2][d] += Gf21 * cw[d];
        W[3][d] += Gf31 * cw[d];
        W[4][d] += Gf41 * cw[d];
    }
#pragma unroll
    for (int k = 0; k < 5; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            D.c[(k * 3 + d) * nr + i] = C[k][d];
            D.w[(k * 3 + d) * nr + i] = W[k][d];
        }
}

__device__ __forceinline__ void corr_rigid(const View& v, const Dyn& D, int i) {
    const int nr = v.nrig;
    const double s0i = D.th[TH_S], rs0i = D.th[TH_RS];
    // loads first (see pred_rigid)
    double C[5][3], W[5][3], Q[5][4], a[9], fc[3], tq[3];
    load_cw(D, nr, i, C, W);
    load_q(D, nr, i, Q);
#pragma unroll
    for (int k = 0; k < 9; ++k) a[k] = D.a[k * nr + i];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        fc[d] = D.fc[d * nr + i];
        tq[d] = D.tq[d * nr + i];
    }
    const double w0[3] = {W[0][0], W[0][1], W[0][2]};
    corr_q(D, nr, i, Q, w0);
    corr_cw(D, nr, i, C, W, a, fc, tq, s0i, rs0i);
}

constexpr int kTailAcc = 512;  // energy sums staged in shared memory by the corrector's tail

// The corrector's tail, in the block that finished last, as two independent parts on two warps:
// uconf = sum(elj) + sum(eqq) + uewa + urf (src/forcem.f90:1055,1079) and the wall pressure (the
// energy sums loaded by one warp at once into shared memory, then summed by its lane 0 in the
// reference's order), and the thermostat corrector with the step counters.
__device__ void corr_energy(const View& v, const Dyn& D, int slab, double* sh) {
    const int l = threadIdx.x & 31;
    const int na = 2 * v.nijt + ACC_NSLOT;
    const bool staged = na <= kTailAcc;
    if (staged)
        for (int k = l; k < na; k += 32) sh[k] = __ldcg(&v.acc[k]);
    __syncwarp();
    if (l != 0) return;
    double* th = D.th;
    const double* a = staged ? sh : v.acc;
    const double* sl = a + 2 * v.nijt;
    double slj = 0.0, sqq = 0.0;
    for (int k = 0; k < v.nijt; ++k) {
        slj += a[k];
        sqq += a[v.nijt + k];
    }
    double urf = 0.0;
    if (slab) {
        const double crf = -2.0 * F32D(3.1415926535898) * v.lzi * v.lxi * v.lyi;
        urf = -crf * v.facq * sl[ACC_DIPZ] * sl[ACC_DIPZ];
    }
    th[TH_UCONF] = slj + sqq + 0.5 * sl[ACC_UEWA] + urf;
    th[TH_PRESS] = (sl[ACC_FWS + 8] - sl[ACC_FWS + 6]) / (2.0 * v.lx * v.ly) * 1000.0 /
                   (F32D(6.022045e23) * F32D(1e-30)) * F32D(1e-5);
}

// the thermostat corrector and the step counters (one thread; all loads first)
__device__ void corr_thermo(const View& v, const Dyn& D) {
    double* th = D.th;
    double s[5], rs[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        s[k] = __ldcg(&th[TH_S + k]);
        rs[k] = __ldcg(&th[TH_RS + k]);
    }
    const double sft = __ldcg(&th[TH_SFT]), sfr = __ldcg(&th[TH_SFR]), ke = __ldcg(&th[TH_KE]);
    const double steps = __ldcg(&th[TH_STEPS]), nreb = __ldcg(&th[TH_REBUILDS]);
    const int reb = __ldcg(&v.status[ST_REBUILD]);
    if (D.body.temper != -1.0) {
        double rc = sft - s[1];
        s[0] = s[0] + Gf01 * rc;
        s[1] = sft;
        s[2] = s[2] + Gf21 * rc;
        s[3] = s[3] + Gf31 * rc;
        s[4] = s[4] + Gf41 * rc;
        rc = sfr - rs[1];
        rs[0] = rs[0] + Gf01 * rc;
        rs[1] = sfr;
        rs[2] = rs[2] + Gf21 * rc;
        rs[3] = rs[3] + Gf31 * rc;
        rs[4] = rs[4] + Gf41 * rc;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            th[TH_S + k] = s[k];
            th[TH_RS + k] = rs[k];
        }
    }
    const long nfree = v.nliqa - v.nriga;
    th[TH_TEMPNOW] = ke * 1000.0 / (3.0 * F32D(8.31441) * (double)(float)(nfree + 2 * v.nrig));
    th[TH_STEPS] = steps + 1.0;
    if (reb) th[TH_REBUILDS] = nreb + 1.0;
}

// The block that finished last adds uconf/press and corrects the thermostat.
__device__ __forceinline__ void corr_end(const View& v, const Dyn& D, int slab, double* sh, int nblk) {
    if (!last_block(&D.done[1], nblk)) return;
    if (threadIdx.x < 32) {
        if (threadIdx.x == 0) D.done[1] = 0u;
        corr_energy(v, D, slab, sh);
    } else if (threadIdx.x == 32) {
        corr_thermo(v, D);
    }
}

// The correctors read the thermostat values of the predictor.  MERGE: the mixed force form's final merge and
// force_sum (merge.cuh) run here, each unit's just before its corrector, instead of in a kernel
// of their own; units past the molecules and ions are the surface atoms, whose forces SHAKE's
// Verlet step reads next.
template <int NT, bool MERGE>
__global__ void __launch_bounds__(NT) k_corr(View v, Dyn D, int slab, MergeArgs A) {
    const int nsurf = MERGE ? v.nmove - v.nliqa : 0;
    const int nu = D.nion + v.nrig + nsurf;
    MergeArgs M;
    if constexpr (MERGE) M = merge_begin(v, A);
    double sx = 0.0, sy = 0.0, sz = 0.0;
    for (int r = 0;; ++r) {
        const int u = unit_of<NT>(r, gridDim.x);
        if (u >= nu) break;
        if (u < D.nion) {
            if constexpr (MERGE) merge_flex(v, M, u, sx, sy, sz);
            corr_ion(v, D, u);
        } else if (u < D.nion + v.nrig) {
            const int i = u - D.nion;
            if constexpr (MERGE) merge_rigid(v, M, i, sx, sy, sz);
            corr_rigid(v, D, i);
        } else if constexpr (MERGE) {
            merge_flex(v, M, u - v.nrig, sx, sy, sz);  // surface atom: flexible index nion + s
        }
    }
    if constexpr (MERGE) {
        double t[4] = {sx, sy, sz, 0.0};
        const double sum = warp_sums(t);
        const int lane = threadIdx.x & 31;
        if ((lane & 7) == 0 && lane < 24) atomicAdd(&v.acc[2 * v.nijt + ACC_FWS0 + (lane >> 3)], sum);
    }
    __shared__ double sh_acc[kTailAcc];
    corr_end(v, D, slab, sh_acc, gridDim.x);
}

// The same for small systems: blocks below nrb 16 molecules each, the others ions and surface atoms.
template <bool MERGE>
__device__ __forceinline__ void corr_small(const View& v, const Dyn& D, int slab, const MergeArgs& A, int nrb, int bid, int nblk) {
    __shared__ double s_w[3][kMol], s_q[4][kMol], s_f[3][3][kMol], s_t[3][3][kMol];
    const int t = threadIdx.x;
    MergeArgs M;
    if constexpr (MERGE) M = merge_begin(v, A);
    if (bid < nrb) {
        const int m = t & (kMol - 1), k = t / kMol, nr = v.nrig;
        const bool act = bid * kMol + m < nr;
        const int i = act ? bid * kMol + m : 0;
        const mdg_rigid& body = D.body;
        int st;
        double* b = component(D, nr, i, k, st);
        double a0 = b[0], a1 = b[st], a2 = b[2 * st], a3 = b[3 * (size_t)st], a4 = b[4 * (size_t)st];
        const double s0i = D.th[TH_S], rs0i = D.th[TH_RS];
        double rot[3] = {0, 0, 0};
        if (k >= 3 && k < 6)
#pragma unroll
            for (int e = 0; e < 3; ++e) rot[e] = D.a[(size_t)(3 * (k - 3) + e) * nr + i];
        if (k >= 3 && k < 6) s_w[k - 3][m] = a0;
        if (k >= 6) s_q[k - 6][m] = a0;
        if constexpr (MERGE) {
            if (act && k < 3) {  // site k
                const int j = 3 * i + k;
                double fx, fy, fz;
                merged_force(v, M, j, fx, fy, fz);
                const double rx = v.x[j] - v.cx[i], ry = v.y[j] - v.cy[i], rz = v.z[j] - v.cz[i];
                s_f[k][0][m] = fx;
                s_f[k][1][m] = fy;
                s_f[k][2][m] = fz;
                s_t[k][0][m] = ry * fz - rz * fy;
                s_t[k][1][m] = rz * fx - rx * fz;
                s_t[k][2][m] = rx * fy - ry * fx;
                if (i == nr - 1) {
                    v.rsx[k] = rx;
                    v.rsy[k] = ry;
                    v.rsz[k] = rz;
                }
            }
        }
        __syncthreads();
        double fsum = 0.0;
        if (act && k < 3) {
            double fc;
            if constexpr (MERGE) {
                fc = s_f[0][k][m] + s_f[1][k][m] + s_f[2][k][m];
                fsum = fc;
                M.fc[(size_t)k * nr + i] = fc;
            } else {
                fc = D.fc[(size_t)k * nr + i];
            }
            const double co = (0.5 / body.mw) * fc - a1 * s0i - a2;
            a0 = a0 + Gf02 * co;
            a1 = a1 + Gf12 * co;
            a2 = a2 + Gf22 * co;
            a3 = a3 + Gf32 * co;
            a4 = a4 + Gf42 * co;
        } else if (act) {
            const double wx = s_w[0][m], wy = s_w[1][m], wz = s_w[2][m];
            double co;
            if (k < 6) {
                double tq[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    if constexpr (MERGE) tq[d] = s_t[0][d][m] + s_t[1][d][m] + s_t[2][d][m];
                    else tq[d] = D.tq[(size_t)d * nr + i];
                }
                if constexpr (MERGE) M.tq[(size_t)(k - 3) * nr + i] = k == 3 ? tq[0] : k == 4 ? tq[1] : tq[2];
                const double dI = k == 3 ? body.inyy - body.inzz : k == 4 ? body.inzz - body.inxx : body.inxx - body.inyy;
                const double ww = k == 3 ? wy * wz : k == 4 ? wz * wx : wx * wy;
                const double inv = 1.0 / (k == 3 ? body.inxx : k == 4 ? body.inyy : body.inzz);
                const double c = rot[0] * tq[0] + rot[1] * tq[1] + rot[2] * tq[2];
                co = (c + ww * dI) * inv - a1 - rs0i * a0;
            } else {
                const double q1 = s_q[0][m], q2 = s_q[1][m], q3 = s_q[2][m], q4 = s_q[3][m];
                double cq;
                if (k == 6) cq = 0.5 * (-q3 * wx - q4 * wy + q2 * wz);
                else if (k == 7) cq = 0.5 * (q4 * wx - q3 * wy - q1 * wz);
                else if (k == 8) cq = 0.5 * (q1 * wx + q2 * wy + q4 * wz);
                else cq = 0.5 * (-q2 * wx + q1 * wy - q3 * wz);
                co = cq - a1;
            }
            a0 = a0 + Gf01 * co;
            a1 = a1 + Gf11 * co;
            a2 = a2 + Gf21 * co;
            a3 = a3 + Gf31 * co;
            a4 = a4 + Gf41 * co;
        }
        if (act) {
            b[0] = a0;
            b[st] = a1;
            b[2 * st] = a2;
            b[3 * (size_t)st] = a3;
            b[4 * (size_t)st] = a4;
        }
        if constexpr (MERGE) {
            if (t < 2 * 32) {
                fsum = sum16(fsum);
                if (m == 0 && k < 3) atomicAdd(&v.acc[2 * v.nijt + ACC_FWS0 + k], fsum);
            }
        }
    } else {
        const int nflex = D.nion + (MERGE ? v.nmove - v.nliqa : 0), u = (bid - nrb) * kFlex + t;
        if (t < kFlex) {
            double sx = 0.0, sy = 0.0, sz = 0.0;
            if constexpr (MERGE) {
                if (u < nflex) merge_flex(v, M, u, sx, sy, sz);
            }
            if (u < D.nion) corr_ion(v, D, u);
            if constexpr (MERGE) {
                sx = warp_sum(sx);
                sy = warp_sum(sy);
                sz = warp_sum(sz);
                if (t == 0) {
                    atomicAdd(&v.acc[2 * v.nijt + ACC_FWS0 + 0], sx);
                    atomicAdd(&v.acc[2 * v.nijt + ACC_FWS0 + 1], sy);
                    atomicAdd(&v.acc[2 * v.nijt + ACC_FWS0 + 2], sz);
                }
            }
        }
    }
    __shared__ double sh_acc[kTailAcc];
    corr_end(v, D, slab, sh_acc, nblk);
}

template <bool MERGE>
__global__ void __launch_bounds__(kST) k_corr_small(View v, Dyn D, int slab, MergeArgs A, int nrb) {
    corr_small<MERGE>(v, D, slab, A, nrb, blockIdx.x, gridDim.x);
}

// ---- the replicas of a batch, one launch per kernel --------------------------------------------
// The forms for small systems, the close of the packing and the wall tail of several systems at once:
// 16 replicas of 2,250 waters made 128 graph nodes a step with a launch per replica and kernel, 68 so.
// 20 steps 15.6 -> 14.8 ms.
struct alignas(16) IntRep {
    View v;
    Dyn D;
    PackArgs P;
    MergeArgs A;
    const double* lr;
    int slab, nrb, nfb, nparts, nrb_c;
};

struct RepOf {
    int r, bid, nblk;
};

// This block's system (its descriptor copied to shared memory) and the block within it.
__device__ __forceinline__ RepOf load_rep(const IntRep* __restrict__ reps, const int* __restrict__ first, int nrep, IntRep* dst) {
    static_assert(sizeof(IntRep) % 8 == 0, "word copy");
    RepOf o;
    o.r = rep_of_block(first, nrep, blockIdx.x);
    o.bid = blockIdx.x - first[o.r];
    o.nblk = first[o.r + 1] - first[o.r];
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(reps + o.r);
    unsigned long long* d = reinterpret_cast<unsigned long long*>(dst);
    for (int k = threadIdx.x; k < (int)(sizeof(IntRep) / 8); k += blockDim.x) d[k] = src[k];
    __syncthreads();
    return o;
}

__global__ void __launch_bounds__(kST) k_pred_small_b(const IntRep* reps, const int* first, int nrep) {
    __shared__ alignas(16) unsigned char raw[sizeof(IntRep)];  // IntRep has member initialisers
    IntRep& R = *reinterpret_cast<IntRep*>(raw);
    const RepOf o = load_rep(reps, first, nrep, &R);
    pred_small<true>(R.v, R.D, Clear{}, R.P, R.nrb, R.nfb, o.bid, o.nblk);
}

__global__ void __launch_bounds__(64) k_step_close_b(const IntRep* reps) {
    const IntRep& R = reps[blockIdx.x];
    step_close(R.v, R.D, R.P.pk, R.P.dip, R.nparts);
}

__global__ void __launch_bounds__(kLrNT) k_lr_tail_b(const IntRep* reps, const int* first, int nrep) {
    __shared__ alignas(16) unsigned char raw[sizeof(IntRep)];
    IntRep& R = *reinterpret_cast<IntRep*>(raw);
    const RepOf o = load_rep(reps, first, nrep, &R);
    if (R.slab) lr_tail_block(R.v, R.lr, o.bid, o.nblk);
}

__global__ void __launch_bounds__(kST) k_corr_small_b(const IntRep* reps, const int* first, int nrep) {
    __shared__ alignas(16) unsigned char raw[sizeof(IntRep)];
    IntRep& R = *reinterpret_cast<IntRep*>(raw);
    const RepOf o = load_rep(reps, first, nrep, &R);
    corr_small<true>(R.v, R.D, R.slab, R.A, R.nrb_c, o.bid, o.nblk);
}

Dyn dyn_of(Ctx& c) {
    Dyn D;
    D.done = c.d_done;
    D.xd = c.d_xd;
    D.c = c.d_c;
    D.q = c.d_q;
    D.w = c.d_w;
    D.a = c.d_a;
    D.th = c.d_thermo;
    D.isum = c.d_isum;
    D.ft = c.d_ft;
    D.fc = c.d_fc;
    D.tq = c.d_tq;
    D.body = c.body;
    D.nion = c.v.nliqa - c.v.nriga;
    return D;
}

// Units up to which the forms for small systems are the faster ones: with more the FP64 pipe is the limit and
// their half-filled warps cost (bulk water, k_pred and k_corr, one thread per molecule | component): 1,000
// 17 and 17 | 8 and 11 us, 4,913 19 and 17 | 11 and 13, 8,000 19 and 18 | 12 and 15, 15,625 19 and 19 | 19
// and 20, 32,768 28 and 25 (24 and
// 24 since a warp's sums share their steps) | 37 and 33.
bool small(int nu) { return nu <= 80 * kSM; }
int nblk(int n) { return std::max(1, std::min((n + 127) / 128, kSM * 8)); }

}  // namespace

void predict_launch(Ctx& c, bool clear_acc, bool clear_kps, bool pack) {
    const View& v = c.v;
    Dyn D = dyn_of(c);
    const int nu = D.nion + v.nrig;
    Clear z{{v.acc, c.d_kps}, {clear_acc ? 2 * v.nijt + ACC_NSLOT : 0, clear_kps && c.d_kps ? v.nit : 0}};
    PackArgs P{};
    if (pack) {
        P.pk = c.pk;
        P.dip = c.variant == MDG_SLAB ? 1 : 0;
    }
    const int nwall = v.ntota - v.nmove;
    if (small(nu)) {
        const int nrb = (v.nrig + kMol - 1) / kMol, nfb = (D.nion + kFlex - 1) / kFlex;
        const int nb = std::max(1, nrb + nfb), nwb = pack ? std::min((nwall + kST - 1) / kST, kSM * 8) : 0;
        c.pred_parts = nb + nwb;
        if (pack) k_pred_small<true><<<nb + nwb, kST, 0, c.stream>>>(v, D, z, P, nrb, nb - nrb);
        else k_pred_small<false><<<nb, kST, 0, c.stream>>>(v, D, z, P, nrb, nb - nrb);
    } else {
        const int nb = nblk(nu);
        P.npred = nb;
        const int nwb = pack ? std::min((nwall + 127) / 128, kSM * 8) : 0;
        c.pred_parts = nb + nwb;
        if (pack) k_pred<128, true><<<nb + nwb, 128, 0, c.stream>>>(v, D, z, P);
        else k_pred<128, false><<<nb, 128, 0, c.stream>>>(v, D, z, P);
    }
}

void step_close_launch(Ctx& c) {
    k_step_close<<<1, 64, 0, c.stream>>>(c.v, dyn_of(c), c.pk, c.variant == MDG_SLAB ? 1 : 0, c.pred_parts);
}

void correct_launch(Ctx& c, bool merge) {
    const View& v = c.v;
    Dyn D = dyn_of(c);
    const int nu = D.nion + v.nrig + (merge ? v.nmove - v.nliqa : 0);
    const int slab = c.variant == MDG_SLAB ? 1 : 0;
    const MergeArgs A = merge ? merge_args(c, c.d_frc) : MergeArgs{};
    if (small(nu)) {
        const int nrb = (v.nrig + kMol - 1) / kMol, nb = std::max(1, nrb + (nu - v.nrig + kFlex - 1) / kFlex);
        if (merge) k_corr_small<true><<<nb, kST, 0, c.stream>>>(v, D, slab, A, nrb);
        else k_corr_small<false><<<nb, kST, 0, c.stream>>>(v, D, slab, A, nrb);
    } else {
        if (merge) k_corr<128, true><<<nblk(nu), 128, 0, c.stream>>>(v, D, slab, A);
        else k_corr<128, false><<<nblk(nu), 128, 0, c.stream>>>(v, D, slab, A);
    }
}

// ---- replica batches: host side ------------------------------------------------------------
bool int_batchable(const Ctx& c) { return small(c.v.nliqa - c.v.nriga + c.v.nrig); }

int int_batch_setup(IntBatch& ib, const std::vector<Ctx*>& cs, std::string& err) {
    ib.nrep = (int)cs.size();
    if (ib.nrep == 0) return MDG_OK;
    std::vector<IntRep> reps(ib.nrep);
    std::vector<int> first(3 * (ib.nrep + 1), 0);
    for (int r = 0; r < ib.nrep; ++r) {
        Ctx& c = *cs[r];
        IntRep& R = reps[r];
        R.v = c.v;
        R.D = dyn_of(c);
        R.P.pk = c.pk;
        R.P.dip = c.variant == MDG_SLAB ? 1 : 0;
        R.P.npred = 0;
        R.A = merge_args(c, c.d_frc);
        R.lr = c.d_lr;
        R.slab = R.P.dip;
        R.nrb = R.nrb_c = (c.v.nrig + kMol - 1) / kMol;
        R.nfb = (R.D.nion + kFlex - 1) / kFlex;
        R.nparts = R.nrb + R.nfb + (c.v.ntota - c.v.nmove + kST - 1) / kST;
        R.nparts = c.pred_parts = std::min(R.nparts, R.nrb + R.nfb + kSM * 8);
        const int nb[3] = {R.nparts, R.nrb + R.nfb, std::max(1, (c.v.nmove + kLrNT - 1) / kLrNT)};
        for (int k = 0; k < 3; ++k) first[k * (ib.nrep + 1) + r + 1] = first[k * (ib.nrep + 1) + r] + nb[k];
    }
    const size_t off = (sizeof(IntRep) * ib.nrep + 255) & ~size_t(255), need = off + sizeof(int) * first.size();
    if (need > ib.cap) {
        if (ib.d_buf) cudaFree(ib.d_buf);
        ib.d_buf = nullptr;
        ib.cap = 0;
        if (cudaMalloc(&ib.d_buf, need) != cudaSuccess) {
            err = "replica batch: integrator descriptor allocation failed";
            return MDG_E_CUDA;
        }
        ib.cap = need;
    }
    unsigned char* base = static_cast<unsigned char*>(ib.d_buf);
    for (int k = 0; k < 3; ++k) {
        ib.first[k] = reinterpret_cast<int*>(base + off) + k * (ib.nrep + 1);
        ib.nblk[k] = first[k * (ib.nrep + 1) + ib.nrep];
    }
    if (cudaMemcpy(base, reps.data(), sizeof(IntRep) * ib.nrep, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(base + off, first.data(), sizeof(int) * first.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
        err = "replica batch: integrator descriptor upload failed";
        return MDG_E_CUDA;
    }
    return MDG_OK;
}

static const IntRep* reps_of(const IntBatch& ib) { return static_cast<const IntRep*>(ib.d_buf); }

void int_batch_pred(const IntBatch& ib, cudaStream_t st) {
    k_pred_small_b<<<ib.nblk[0], kST, 0, st>>>(reps_of(ib), ib.first[0], ib.nrep);
}

void int_batch_close(const IntBatch& ib, cudaStream_t st) { k_step_close_b<<<ib.nrep, 64, 0, st>>>(reps_of(ib)); }

void int_batch_lr(const IntBatch& ib, cudaStream_t st) {
    k_lr_tail_b<<<ib.nblk[2], kLrNT, 0, st>>>(reps_of(ib), ib.first[2], ib.nrep);
}

void int_batch_correct(const IntBatch& ib, cudaStream_t st) {
    k_corr_small_b<<<ib.nblk[1], kST, 0, st>>>(reps_of(ib), ib.first[1], ib.nrep);
}

void int_batch_free(IntBatch& ib) {
    if (ib.d_buf) cudaFree(ib.d_buf);
    ib = IntBatch();
}

}  // namespace mdg
