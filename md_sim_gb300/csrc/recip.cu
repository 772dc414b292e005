// recip.cu - reciprocal-space Ewald sum (force_fouri_init / force_fouri,
// src/forcem.f90:657-825 and :827-937), FP64.
//
// k vectors keep the reference's order and selection: l = 0..klmax outer, m, n innermost over
// the half space, kept when  real(l^2+m^2) + real(n^2 kmax^2)/real(knmax^2) < real(kmax^2)+2.01
// in single precision (src/forcem.f90:756-759).  For a fixed (l, m) the kept n form the
// contiguous range -nmax..nmax (1..nmax when l = m = 0), so the list is a sequence of rows.
//
// The n range of a row is symmetric, so both directions work on the pairs (n, -n), n >= 0 ("entries"
// of a row, 0..nmax), and the number of FP64 operations, which is what bounds them (an FP64 FMA
// retires 1.6 lanes per clock per SM on this part), is that of the real sums of a pair:
//
//   k_sfac       S(k) = sum_j q_j e^{i k.r_j} over moving atoms.  With a = q e^{i(l tx + m ty)} and
//                e^{i n tz} = c + i s the four real sums of a.re c, a.im s, a.re s, a.im c give both
//                S(n) and S(-n): 4 FMAs per (atom, entry), 2 per (atom, k), where a complex product
//                and sum per (atom, k) takes 6.  Work item = (row, up to kChunk entries), items
//                sorted by length; phase factors of a tile of atoms are built in shared memory by
//                the same recurrences as the reference (el(l) = el(l-1)*el(1)); partial sums over
//                atom splits meet in FP64 atomics.
//   k_kenergy    uewa, ewqLL and C(k) = Ak conj(S(k) + Sw(k)) (Sw: static walls), stored per entry as
//                P = C(n) + C(-n), M = C(n) - C(-n) and both times n
//   k_kforce     f_j += sum_k Ak Im(conj(S) q_j e^{ik.r_j}) k; one thread per atom with its phase
//                tables in shared memory: per entry T += P c + i M s and T' += nM c + i nP s, 8 FMAs
//                (4 per k), then Im(a T), Im(a T') once per row; P and M are warp broadcasts.  The
//                rows are dealt to as many grid rows as give every SM work when atoms are few.
// 2,048-water slab (6,144 atoms, 4,338 k): k_sfac 586 -> 204 us, k_kforce 1,778 -> 290 us against the
// form with complex products, items of 8 n, 256-thread blocks and one thread per atom over all rows;
// 32,768 waters (29,038 k) 112 -> 44 ms, of which k_kforce 27 ms, its FMAs at the 0.5 TFMA/s that a loop of
// independent FP64 FMAs reaches on this part.  From 5e6 (atom, k) on contexts take the gridded sum of
// recip_nu64.cu instead; mdg_recip_forces_noalloc always runs these.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "ctx.h"

namespace mdg {

namespace {

constexpr int kChunk = 13;    // most entries per work item in k_sfac (4 sums each, in registers)
constexpr int kSfacNT = 128;
constexpr int kForceNT = 64;
constexpr int kSfacTile = 32;   // most atoms per phase table of k_sfac (fewer where one atom's factors are many)
constexpr int kMaxSplit = 64;   // most grid rows of k_kforce

// Entries of a row: n = 0..nmax, whose (n, -n) are the row's k vectors ((0, 0, n > 0) for the first).
__host__ __device__ __forceinline__ int row_entries(int n_first, int nlen) {
    return (n_first > 0 ? n_first + nlen - 1 : -n_first) + 1;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 conjd(double2 a) { return make_double2(a.x, -a.y); }

struct KDims {
    int KL, KM, KN;        // table extents (positive powers 0..K)
    double px, py, pz;     // 2 pi / L
};

// Phase table of one atom and direction, e^{i k a} for k = 0..K at t[k * stride], by recurrence.
__device__ void phase_table(double a, int K, double2* t, int stride) {
    double s, c;
    sincos(a, &s, &c);
    const double2 e1 = make_double2(c, s);
    double2 e = make_double2(1.0, 0.0);
    t[0] = e;
    for (int k = 1; k <= K; ++k) {
        e = k == 1 ? e1 : cmul(e, e1);
        t[(size_t)k * stride] = e;
    }
}

// rows: (l, m, n_first, k_first); witem_n: first entry | entries << 16 of each work item
__global__ void __launch_bounds__(kSfacNT) k_sfac(View v, KDims d, int nrow, const int4* __restrict__ rows,
                                                  const int* __restrict__ witem_row, const int* __restrict__ witem_n,
                                                  int nwork, int tile, int atoms_per_split, double2* S, int nk_total) {
    extern __shared__ double2 sm[];
    // per atom: q e^{i l tx} (l = 0..KL), e^{i m ty} (m = 0..KM), e^{i n tz} (n = 0..KN)
    const int per = d.KL + 1 + d.KM + 1 + d.KN + 1;
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    int l = 0, m = 0, n0 = 0, nn = 0, kc = 0;  // kc: the k index of n = 0 (of n, if that row had it)
    bool half = false;                         // the row of l = m = 0 has no n <= 0
    if (w < nwork) {
        const int4 rw = rows[CK(witem_row[w], nrow, 201)];
        l = rw.x;
        m = rw.y;
        n0 = witem_n[w] & 0xffff;
        nn = witem_n[w] >> 16;
        kc = rw.w - rw.z;
        half = rw.z > 0;
    }
    const int nw = __reduce_max_sync(0xffffffffu, nn);  // items are sorted: a warp's lengths are alike
    const int ma = abs(m);
    const double sgm = m < 0 ? -1.0 : 1.0;
    double x1[kChunk], x2[kChunk], x3[kChunk], x4[kChunk];
#pragma unroll
    for (int c = 0; c < kChunk; ++c) x1[c] = x2[c] = x3[c] = x4[c] = 0.0;
    const int a_begin = blockIdx.y * atoms_per_split;
    const int a_end = min(v.nmove, a_begin + atoms_per_split);
    for (int t0 = a_begin; t0 < a_end; t0 += tile) {
        const int nt = min(tile, a_end - t0);
        __syncthreads();
        for (int s = threadIdx.x; s < nt * 3; s += blockDim.x) {
            const int a = s % nt, which = s / nt;
            const int at = CK(t0 + a, v.nmove, 202);
            double2* base = sm + (size_t)CK(a, tile, 203) * per;
            if (which == 0) {
                phase_table(d.px * v.x[at], d.KL, base, 1);
                const double q = v.q[at];
                for (int k = 0; k <= d.KL; ++k) base[k] = make_double2(q * base[k].x, q * base[k].y);
            } else if (which == 1) {
                phase_table(d.py * v.y[at], d.KM, base + d.KL + 1, 1);
            } else {
                phase_table(d.pz * v.z[at], d.KN, base + d.KL + 1 + d.KM + 1, 1);
            }
        }
        __syncthreads();
        for (int a = 0; a < nt; ++a) {
            const double2* base = sm + (size_t)a * per;
            const double2 el = base[CK(l, d.KL + 1, 204)];
            double2 em = base[d.KL + 1 + CK(ma, d.KM + 1, 209)];
            em.y *= sgm;
            const double2* en = base + d.KL + 1 + d.KM + 1 + n0;
            const double2 e = cmul(el, em);
#pragma unroll
            for (int c = 0; c < kChunk; ++c) {
                if (c < nw) {
                    const double2 p = en[c < nn ? c : 0];
                    x1[c] = fma(e.x, p.x, x1[c]);
                    x2[c] = fma(e.y, p.y, x2[c]);
                    x3[c] = fma(e.x, p.y, x3[c]);
                    x4[c] = fma(e.y, p.x, x4[c]);
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < kChunk; ++c) {
        if (c < nn) {
            const int n = n0 + c;
            if (n > 0) {
                atomicAdd(&S[CK(kc + n, nk_total, 205)].x, x1[c] - x2[c]);
                atomicAdd(&S[CK(kc + n, nk_total, 205)].y, x3[c] + x4[c]);
            }
            if (!half) {
                atomicAdd(&S[CK(kc - n, nk_total, 205)].x, n > 0 ? x1[c] + x2[c] : x1[c]);
                atomicAdd(&S[CK(kc - n, nk_total, 205)].y, n > 0 ? x4[c] - x3[c] : x4[c]);
            }
        }
    }
}

// One warp per row: energies, and the row's entries of the pair table C4 (two double4 per entry:
// P.re, P.im, M.re, M.im and the same times n).  qw may be null (no static walls).
__global__ void k_kenergy(View v, int nrow, const int4* __restrict__ rows, const int* __restrict__ nlen,
                          const int* __restrict__ ent, const double* __restrict__ ak, const double2* __restrict__ S,
                          const double2* __restrict__ qw, double2* __restrict__ C4) {
    double ew = 0.0, ll = 0.0;
    const int lane = threadIdx.x & 31;
    auto coef = [&](int k) {
        const double2 s = S[k];
        const double2 q = qw ? qw[k] : make_double2(0.0, 0.0);
        const double2 st = make_double2(s.x + q.x, s.y + q.y);
        const double a = ak[k];
        ll += a * (s.x * s.x + s.y * s.y);
        ew += a * (st.x * st.x + st.y * st.y);
        return make_double2(a * st.x, -a * st.y);
    };
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrow; r += (gridDim.x * blockDim.x) >> 5) {
        const int4 rw = rows[r];
        const int ne = row_entries(rw.z, nlen[r]), kc = rw.w - rw.z;
        for (int n = lane; n < ne; n += 32) {
            double2 cp = make_double2(0.0, 0.0), cm = cp;
            if (n > 0 || rw.z <= 0) cp = coef(kc + n);
            if (n > 0 && rw.z <= 0) cm = coef(kc - n);
            const double2 P = make_double2(cp.x + cm.x, cp.y + cm.y);
            const double2 M = n > 0 ? make_double2(cp.x - cm.x, cp.y - cm.y) : make_double2(0.0, 0.0);
            double2* o = C4 + 4 * (size_t)(ent[r] + n);
            o[0] = P;
            o[1] = M;
            o[2] = make_double2((double)n * P.x, (double)n * P.y);
            o[3] = make_double2((double)n * M.x, (double)n * M.y);
        }
    }
    block_atomic_sum<256>(ew, &v.acc[2 * v.nijt + ACC_UEWA]);
    block_atomic_sum<256>(ll, &v.acc[2 * v.nijt + ACC_EWQLL]);
}

__global__ void __launch_bounds__(kForceNT) k_kforce(View v, KDims d, int nrow, const int4* __restrict__ rows,
                                                     const int* __restrict__ nlen, const int* __restrict__ ent,
                                                     const double2* __restrict__ C4) {
    extern __shared__ double2 sm[];
    // this thread's e^{i m ty} and e^{i n tz}, kForceNT apart (no bank conflicts)
    double2* em = sm + threadIdx.x;
    double2* en = em + (size_t)(d.KM + 1) * kForceNT;
    const int j = blockIdx.x * kForceNT + threadIdx.x;
    const bool active = j < v.nmove;
    const int jj = active ? j : 0;
    phase_table(d.py * v.y[jj], d.KM, em, kForceNT);
    phase_table(d.pz * v.z[jj], d.KN, en, kForceNT);
    double s, c;
    sincos(d.px * v.x[jj], &s, &c);
    const double2 el1 = make_double2(c, s);
    const double q = v.q[jj];
    double2 el = make_double2(q, 0.0);
    int lcur = 0;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    for (int r = blockIdx.y; r < nrow; r += gridDim.y) {
        const int4 rw = rows[r];
        while (lcur < rw.x) {
            el = cmul(el, el1);
            ++lcur;
        }
        double2 emm = em[(size_t)CK(abs(rw.y), d.KM + 1, 211) * kForceNT];
        if (rw.y < 0) emm.y = -emm.y;
        const double2 elm = cmul(el, emm);
        const int ne = row_entries(rw.z, nlen[r]);
        const double2* Ck = C4 + 4 * (size_t)ent[r];
        // each sum in two chains, so that consecutive FMAs do not wait for one another
        const double2 P0 = __ldg(Ck);  // n = 0: e = 1, M = 0
        double tr0 = P0.x, tr1 = 0.0, ti0 = P0.y, ti1 = 0.0, ur0 = 0.0, ur1 = 0.0, ui0 = 0.0, ui1 = 0.0;
#pragma unroll 2
        for (int n = 1; n < ne; ++n) {
            const double2 e = en[(size_t)CK(n, d.KN + 1, 212) * kForceNT];
            const double2 P = __ldg(Ck + 4 * n), M = __ldg(Ck + 4 * n + 1), nP = __ldg(Ck + 4 * n + 2),
                          nM = __ldg(Ck + 4 * n + 3);
            tr0 = fma(P.x, e.x, tr0);
            tr1 = fma(M.y, e.y, tr1);
            ti0 = fma(P.y, e.x, ti0);
            ti1 = fma(M.x, e.y, ti1);
            ur0 = fma(nM.x, e.x, ur0);
            ur1 = fma(nP.y, e.y, ur1);
            ui0 = fma(nM.y, e.x, ui0);
            ui1 = fma(nP.x, e.y, ui1);
        }
        const double st = elm.x * (ti0 + ti1) + elm.y * (tr0 - tr1);
        const double stn = elm.x * (ui0 + ui1) + elm.y * (ur0 - ur1);
        fx += st * (double)rw.x;
        fy += st * (double)rw.y;
        fz += stn;
    }
    if (!active) return;
    fx *= d.px;
    fy *= d.py;
    fz *= d.pz;
    atomicAdd(&v.fx[j], fx);  // other grid rows add to it too, and the real-space loops may be running
    atomicAdd(&v.fy[j], fy);
    atomicAdd(&v.fz[j], fz);
}

// Widom insertion: P and M of every entry (two double2), from S and the walls' sums as they stand.
__global__ void k_pot_table(int nrow, const int4* __restrict__ rows, const int* __restrict__ nlen,
                            const int* __restrict__ ent, const double* __restrict__ ak, const double2* __restrict__ S,
                            const double2* __restrict__ qw, double2* __restrict__ PM) {
    const int lane = threadIdx.x & 31;
    auto coef = [&](int k) {
        const double a = ak[k];
        return make_double2(a * (S[k].x + qw[k].x), -a * (S[k].y + qw[k].y));
    };
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrow; r += (gridDim.x * blockDim.x) >> 5) {
        const int4 rw = rows[r];
        const int ne = row_entries(rw.z, nlen[r]), kc = rw.w - rw.z;
        for (int n = lane; n < ne; n += 32) {
            double2 cp = make_double2(0.0, 0.0), cm = cp;
            if (n > 0 || rw.z <= 0) cp = coef(kc + n);
            if (n > 0 && rw.z <= 0) cm = coef(kc - n);
            double2* o = PM + 2 * (size_t)(ent[r] + n);
            o[0] = make_double2(cp.x + cm.x, cp.y + cm.y);
            o[1] = make_double2(cp.x - cm.x, cp.y - cm.y);
        }
    }
}

// phi(r) = sum_k Re(C(k) e^{ik.r}) at the points (x, y, z)[0, *np): k_kforce's sums without the forces, 4
// FMAs per entry.  A point costs the FMAs of nk / 2 entries whatever molecule it belongs to, so the
// points of all insertions share the blocks.
__global__ void __launch_bounds__(kForceNT) k_pot(KDims d, int nrow, const int4* __restrict__ rows,
                                                  const int* __restrict__ nlen, const int* __restrict__ ent,
                                                  const double2* __restrict__ PM, const double* __restrict__ xyz,
                                                  size_t stride, const int* __restrict__ np, double* __restrict__ phi) {
    extern __shared__ double2 sm[];
    const int n_pts = *np;
    if (blockIdx.x * kForceNT >= n_pts) return;
    double2* em = sm + threadIdx.x;
    double2* en = em + (size_t)(d.KM + 1) * kForceNT;
    const int p = min(blockIdx.x * kForceNT + (int)threadIdx.x, n_pts - 1);
    phase_table(d.py * xyz[stride + p], d.KM, em, kForceNT);
    phase_table(d.pz * xyz[2 * stride + p], d.KN, en, kForceNT);
    double s, c;
    sincos(d.px * xyz[p], &s, &c);
    const double2 el1 = make_double2(c, s);
    double2 el = make_double2(1.0, 0.0);
    int lcur = 0;
    double sum = 0.0;
    for (int r = blockIdx.y; r < nrow; r += gridDim.y) {
        const int4 rw = rows[r];
        while (lcur < rw.x) {
            el = cmul(el, el1);
            ++lcur;
        }
        double2 emm = em[(size_t)CK(abs(rw.y), d.KM + 1, 213) * kForceNT];
        if (rw.y < 0) emm.y = -emm.y;
        const double2 elm = cmul(el, emm);
        const int ne = row_entries(rw.z, nlen[r]);
        const double2* Ck = PM + 2 * (size_t)ent[r];
        const double2 P0 = __ldg(Ck);
        double tr0 = P0.x, tr1 = 0.0, ti0 = P0.y, ti1 = 0.0;
#pragma unroll 4
        for (int n = 1; n < ne; ++n) {
            const double2 e = en[(size_t)CK(n, d.KN + 1, 214) * kForceNT];
            const double2 P = __ldg(Ck + 2 * n), M = __ldg(Ck + 2 * n + 1);
            tr0 = fma(P.x, e.x, tr0);
            tr1 = fma(M.y, e.y, tr1);
            ti0 = fma(P.y, e.x, ti0);
            ti1 = fma(M.x, e.y, ti1);
        }
        sum += elm.x * (tr0 - tr1) - elm.y * (ti0 + ti1);
    }
    if (blockIdx.x * kForceNT + (int)threadIdx.x >= n_pts) return;
    if (gridDim.y > 1) atomicAdd(&phi[p], sum);
    else phi[p] = sum;
}

// Work items of k_sfac for the rows (n_first, nlen): (row, first entry | entries << 16), each row cut
// into equal items of at most kChunk entries, sorted by length so that the lanes of a warp run alike.
// Returns the number of entries of all rows; ent[r] is row r's first.
int sfac_items(const int4* rows, const int* nlen, int nrow, int* ent, int* wr, int* wn, int& nwork) {
    int ne = 0;
    nwork = 0;
    for (int r = 0; r < nrow; ++r) {
        ent[r] = ne;
        ne += row_entries(rows[r].z, nlen[r]);
    }
    for (int len = kChunk; len >= 1; --len)
        for (int r = 0; r < nrow; ++r) {
            const int e = row_entries(rows[r].z, nlen[r]), parts = (e + kChunk - 1) / kChunk;
            for (int p = 0; p < parts; ++p) {
                const int a = e * p / parts, b = e * (p + 1) / parts;
                if (b - a != len) continue;
                wr[nwork] = r;
                wn[nwork++] = a | len << 16;
            }
        }
    return ne;
}

// Launch shapes: atom splits of k_sfac and grid rows of k_kforce that give every SM a few blocks
// (both kernels keep the FP64 pipe busy with four warps per SM), at least 4 atoms and 4 rows each.
struct KGrid {
    dim3 sfac, force;
    int tile, atoms_per_split, smem_sfac, smem_force;
};
constexpr int kTableRoom = 200 * 1024;  // shared memory for phase tables
// Whether the phase tables fit: 8 atoms of k_sfac, and (the limit set by a block of 128 atoms) k_kforce's.
bool tables_fit(const KDims& d) {
    const int per = (d.KL + 1 + d.KM + 1 + d.KN + 1) * (int)sizeof(double2) + (int)sizeof(double);
    return 128 * (d.KM + 1 + d.KN + 1) * (int)sizeof(double2) <= kTableRoom && 8 * per <= kTableRoom;
}
KGrid k_grid(const KDims& d, int natom, int nrow, int nwork) {
    KGrid g;
    const int kb = std::max(1, (nwork + kSfacNT - 1) / kSfacNT), fb = std::max(1, (natom + kForceNT - 1) / kForceNT);
    int splits = std::max(1, std::min((152 * 16 + kb - 1) / kb, (natom + 3) / 4));
    g.atoms_per_split = (natom + splits - 1) / splits;
    splits = (natom + g.atoms_per_split - 1) / g.atoms_per_split;
    g.sfac = dim3(kb, splits);
    g.force = dim3(fb, std::max(1, std::min({(152 * 16 + fb - 1) / fb, kMaxSplit, nrow / 4})));
    const int per = (d.KL + 1 + d.KM + 1 + d.KN + 1) * (int)sizeof(double2);
    g.tile = std::min(kSfacTile, kTableRoom / per);  // (at least 8: tables_fit)
    g.smem_sfac = g.tile * per;
    g.smem_force = kForceNT * (d.KM + 1 + d.KN + 1) * (int)sizeof(double2);
    return g;
}

}  // namespace

// Host side: k set in reference order, rows, Ak, static wall structure factors, work items.
int recip_setup(Ctx& c, int64_t kmax, const double* x0, const double* y0, const double* z0) {
    View& v = c.v;
    KSet& ks = c.ks;
    typedef std::complex<double> cd;
    const double pi_r = (double)3.1415926535898f;
    const double PH_e = (double)1.6021892e-19f, PH_Na = (double)6.022045e23f,
                 PH_eps0 = (double)8.85418782e-12f, PH_A2m = (double)1.0e-10f;
    ks.pipix = 2.0 * pi_r / v.lx;
    ks.pipiy = 2.0 * pi_r / v.ly;
    ks.pipiz = 2.0 * pi_r / v.lz;
    const double alf4i = -1.0 / (4.0 * v.alfa * v.alfa);
    const double fac = 2.0 * PH_e * PH_e * PH_Na / (PH_eps0 * PH_A2m * 1000.0 * v.lx * v.ly * v.lz);
    const double lmin = std::min(v.lx, std::min(v.ly, v.lz));
    const double rk = (double)(float)kmax;
    const int KL = (int)std::lround(rk * v.lx / lmin), KM = (int)std::lround(rk * v.ly / lmin),
              KN = (int)std::lround(rk * v.lz / lmin);
    ks.klmax = KL;
    ks.kmmax = KM;
    ks.knmax = KN;
    std::vector<int4> rows;
    std::vector<int> nlen;
    std::vector<int3> kvec;
    std::vector<double> ak;
    const float lim = (float)(kmax * kmax) + 2.01f;
    int kmmin = 0, knmin = 1;
    for (int kl = 0; kl <= KL; ++kl) {
        const double rl = ks.pipix * (double)(float)kl;
        for (int km = kmmin; km <= KM; ++km) {
            const double rm = ks.pipiy * (double)(float)km;
            int first = 0, cnt = 0;
            for (int kn = knmin; kn <= KN; ++kn) {
                volatile float a = (float)(kl * kl + km * km);
                volatile float b = (float)((int64_t)kn * kn * kmax * kmax) / (float)((int64_t)KN * KN);
                volatile float ksq = a + b;
                if (!(ksq < lim)) continue;
                const double rn = ks.pipiz * (double)(float)kn;
                const double rksq = rl * rl + rm * rm + rn * rn;
                if (cnt == 0) first = kn;
                ++cnt;
                kvec.push_back(make_int3(kl, km, kn));
                ak.push_back(fac * std::exp(rksq * alf4i) / rksq);
            }
            if (cnt > 0) {
                rows.push_back(make_int4(kl, km, first, (int)kvec.size() - cnt));
                nlen.push_back(cnt);
            }
            knmin = -KN;
        }
        kmmin = -KM;
    }
    ks.nk = (int)kvec.size();
    ks.nrow = (int)rows.size();
    // static wall structure factor, two halves summed separately as Qsumw1/Qsumw2
    std::vector<cd> q1(ks.nk, cd(0, 0)), q2(ks.nk, cd(0, 0));
    {
        std::vector<cd> el(KL + 1), em(2 * KM + 1), en(2 * KN + 1);
        const int nw = v.nwall;
        for (int w = 0; w < nw; ++w) {
            const int i = v.nmove + w;
            el[0] = em[KM] = en[KN] = cd(1, 0);
            const double tx = ks.pipix * x0[i], ty = ks.pipiy * y0[i], tz = ks.pipiz * z0[i];
            if (KL >= 1) el[1] = cd(std::cos(tx), std::sin(tx));
            if (KM >= 1) em[KM + 1] = cd(std::cos(ty), std::sin(ty));
            if (KN >= 1) en[KN + 1] = cd(std::cos(tz), std::sin(tz));
            for (int l = 2; l <= KL; ++l) el[l] = el[l - 1] * el[1];
            for (int m = 2; m <= KM; ++m) em[KM + m] = em[KM + m - 1] * em[KM + 1];
            for (int m = 1; m <= KM; ++m) em[KM - m] = std::conj(em[KM + m]);
            for (int n = 2; n <= KN; ++n) en[KN + n] = en[KN + n - 1] * en[KN + 1];
            for (int n = 1; n <= KN; ++n) en[KN - n] = std::conj(en[KN + n]);
            const double qw = c.h_qs_wall[w];
            std::vector<cd>& dst = (w < nw / 2) ? q1 : q2;
            for (int r = 0; r < ks.nrow; ++r) {
                const int4 rw = rows[r];
                const cd elm = qw * el[rw.x] * em[KM + rw.y];
                for (int t = 0; t < nlen[r]; ++t) dst[rw.w + t] += elm * en[KN + rw.z + t];
            }
        }
    }
    std::vector<double2> qw(ks.nk);
    c.ewqWW = 0.0;
    for (int k = 0; k < ks.nk; ++k) {
        const cd s = q1[k] + q2[k];
        qw[k] = make_double2(s.real(), s.imag());
        c.ewqWW += (ak[k] * s * std::conj(s)).real();
    }
    c.ewqWW *= 0.5;
    std::vector<int> ent(std::max(ks.nrow, 1)), wr(ks.nk + 1), wn(ks.nk + 1);
    const int nent = sfac_items(rows.data(), nlen.data(), ks.nrow, ent.data(), wr.data(), wn.data(), ks.nwork);
    const int nk1 = std::max(ks.nk, 1), nr1 = std::max(ks.nrow, 1), nw1 = std::max(ks.nwork, 1);
    ks.row = (int4*)dalloc(c, sizeof(int4) * nr1);
    ks.row_nlen = (int*)dalloc(c, sizeof(int) * nr1);
    ks.ak = (double*)dalloc(c, sizeof(double) * nk1);
    ks.qw = (double2*)dalloc(c, sizeof(double2) * nk1);
    ks.s = (double2*)dalloc(c, sizeof(double2) * nk1);
    ks.c4 = (double2*)dalloc(c, 4 * sizeof(double2) * std::max(nent, 1));
    ks.ent = (int*)dalloc(c, sizeof(int) * nr1);
    ks.kvec = (int3*)dalloc(c, sizeof(int3) * nk1);
    ks.witem_row = (int*)dalloc(c, sizeof(int) * nw1);
    ks.witem_n = (int*)dalloc(c, sizeof(int) * nw1);
    ks.h_row = rows;
    ks.h_nlen = nlen;
    if (ks.nk > 0) {
        MDG_CUDA(cudaMemcpy(ks.row, rows.data(), sizeof(int4) * ks.nrow, cudaMemcpyHostToDevice));
        MDG_CUDA(cudaMemcpy(ks.row_nlen, nlen.data(), sizeof(int) * ks.nrow, cudaMemcpyHostToDevice));
        MDG_CUDA(cudaMemcpy(ks.ent, ent.data(), sizeof(int) * ks.nrow, cudaMemcpyHostToDevice));
        MDG_CUDA(cudaMemcpy(ks.ak, ak.data(), sizeof(double) * ks.nk, cudaMemcpyHostToDevice));
        MDG_CUDA(cudaMemcpy(ks.qw, qw.data(), sizeof(double2) * ks.nk, cudaMemcpyHostToDevice));
        MDG_CUDA(cudaMemcpy(ks.kvec, kvec.data(), sizeof(int3) * ks.nk, cudaMemcpyHostToDevice));
        MDG_CUDA(cudaMemcpy(ks.witem_row, wr.data(), sizeof(int) * ks.nwork, cudaMemcpyHostToDevice));
        MDG_CUDA(cudaMemcpy(ks.witem_n, wn.data(), sizeof(int) * ks.nwork, cudaMemcpyHostToDevice));
    }
    MDG_CUDA(allow_max_smem(k_sfac));
    MDG_CUDA(allow_max_smem(k_kforce));
    MDG_CUDA(allow_max_smem(k_pot));
    ks.nent = nent;
    if (!tables_fit(KDims{KL, KM, KN, ks.pipix, ks.pipiy, ks.pipiz}))
        return set_err(&c, MDG_E_UNSUPPORTED, "kmax too large for the shared-memory phase tables");
    return MDG_OK;
}

void recip_fp64(Ctx& c) {
    const View& v = c.v;
    KSet& ks = c.ks;
    if (ks.nk == 0 || v.nmove == 0) return;
    if (c.nu64.ready) {
        recip_nu64(c);
        return;
    }
    KDims d{ks.klmax, ks.kmmax, ks.knmax, ks.pipix, ks.pipiy, ks.pipiz};
    const KGrid g = k_grid(d, v.nmove, ks.nrow, ks.nwork);
    cudaMemsetAsync(ks.s, 0, sizeof(double2) * ks.nk, c.stream);
    k_sfac<<<g.sfac, kSfacNT, g.smem_sfac, c.stream>>>(v, d, ks.nrow, ks.row, ks.witem_row, ks.witem_n, ks.nwork,
                                                       g.tile, g.atoms_per_split, ks.s, ks.nk);
    k_kenergy<<<std::min((ks.nrow + 7) / 8, 256), 256, 0, c.stream>>>(v, ks.nrow, ks.row, ks.row_nlen, ks.ent, ks.ak,
                                                                     ks.s, ks.qw, ks.c4);
    k_kforce<<<g.force, kForceNT, g.smem_force, c.stream>>>(v, d, ks.nrow, ks.row, ks.row_nlen, ks.ent, ks.c4);
}

void recip_pot_table(Ctx& c, double2* pm, cudaStream_t st) {
    const KSet& ks = c.ks;
    if (ks.nk == 0) return;
    k_pot_table<<<std::min((ks.nrow + 7) / 8, 256), 256, 0, st>>>(ks.nrow, ks.row, ks.row_nlen, ks.ent, ks.ak, ks.s, ks.qw,
                                                                  pm);
}

// np: number of points on the device, at most `most`, of which `likely` are expected.
void recip_potential(Ctx& c, const double2* pm, const double* xyz, size_t stride, const int* np, int most, int likely,
                     double* phi, cudaStream_t st) {
    const KSet& ks = c.ks;
    cudaMemsetAsync(phi, 0, sizeof(double) * most, st);
    if (ks.nk == 0) return;
    const KDims d{ks.klmax, ks.kmmax, ks.knmax, ks.pipix, ks.pipiy, ks.pipiz};
    const int want = (152 * 8 * kForceNT + likely - 1) / likely;
    const dim3 grid((most + kForceNT - 1) / kForceNT, std::max(1, std::min(std::min(want, kMaxSplit), ks.nrow)));
    k_pot<<<grid, kForceNT, sizeof(double2) * kForceNT * (size_t)(d.KM + 1 + d.KN + 1), st>>>(
        d, ks.nrow, ks.row, ks.row_nlen, ks.ent, pm, xyz, stride, np, phi);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free reciprocal sum (mdg_recip_forces_noalloc).
//
// Some callers cannot allocate device memory while they run: a host that has sized its device
// memory once at start-up and forbids later driver allocations, a framework whose caching
// allocator owns all device memory (a cudaMalloc behind its back fragments the pool and
// synchronises the device).  For them the
// structure-factor sum runs here with all of its scratch in one static device array that the
// library carries (every GPU that loads the library holds it until the process exits).  The caller
// passes device arrays in and out; nothing is allocated by this path.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr int kNaMaxK = MDG_NOALLOC_MAX_K;
constexpr int kNaMaxRows = MDG_NOALLOC_MAX_ROWS;
// a row of 2 nmax + 1 k vectors has nmax + 1 entries; the first row, with n > 0 only, at most 100
// (the phase tables' limit on knmax)
constexpr int kNaMaxEnt = (kNaMaxK + kNaMaxRows) / 2 + 128;
constexpr int kNaMaxWork = kNaMaxK / kChunk + kNaMaxRows;

// byte offsets of the regions inside the scratch array
constexpr size_t kNaS = 0;                                              // double2 [MAX_K]  S(k)
constexpr size_t kNaC = kNaS + sizeof(double2) * kNaMaxK;               // 4 x double2 [MAX_ENT]  C(k) by entry
constexpr size_t kNaAk = kNaC + 4 * sizeof(double2) * kNaMaxEnt;        // double  [MAX_K]
constexpr size_t kNaRows = kNaAk + sizeof(double) * kNaMaxK;            // int4    [MAX_ROWS]
constexpr size_t kNaNlen = kNaRows + sizeof(int4) * kNaMaxRows;         // int     [MAX_ROWS]
constexpr size_t kNaEnt = kNaNlen + sizeof(int) * kNaMaxRows;           // int     [MAX_ROWS]
constexpr size_t kNaWr = kNaEnt + sizeof(int) * kNaMaxRows;             // int     [MAX_WORK]
constexpr size_t kNaWn = kNaWr + sizeof(int) * kNaMaxWork;              // int     [MAX_WORK]
constexpr size_t kNaAcc = (kNaWn + sizeof(int) * kNaMaxWork + 255) / 256 * 256;  // double [64]
constexpr size_t kNaStatus = kNaAcc + sizeof(double) * 64;              // int [ST_NWORDS]
constexpr size_t kNaBytes = (kNaStatus + sizeof(int) * ST_NWORDS + 255) / 256 * 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

__global__ void k_noalloc_energy(const double* acc, double* uewa) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && uewa) *uewa = 0.5 * acc[ACC_UEWA];
}

std::mutex g_na_mutex;
constexpr int kNaMaxDev = 64;
unsigned char* g_na_ptr[kNaMaxDev] = {nullptr};
// host-side k tables, reused by every call (calls are serialised by g_na_mutex)
int4 g_na_rows[kNaMaxRows];
int g_na_nlen[kNaMaxRows], g_na_ent[kNaMaxRows];
double g_na_ak[kNaMaxK];
int g_na_wr[kNaMaxWork], g_na_wn[kNaMaxWork];
thread_local char g_na_err[256] = "";

int na_fail(int code, const char* msg) {
    std::snprintf(g_na_err, sizeof g_na_err, "%s", msg);
    return code;
}

}  // namespace

const char* recip_noalloc_error() { return g_na_err; }

int recip_forces_noalloc(const double* x, const double* y, const double* z, const double* q, int64_t n,
                         double lx, double ly, double lz, double alpha, int64_t kmax, double* fx, double* fy,
                         double* fz, double* uewa, cudaStream_t st) {
    if (!x || !y || !z || !q || !fx || !fy || !fz || n < 1 || n >= (1LL << 31) || kmax < 1 || alpha <= 0.0 ||
        lx <= 0.0 || ly <= 0.0 || lz <= 0.0)
        return na_fail(MDG_E_ARG, "mdg_recip_forces_noalloc: bad argument");
    std::lock_guard<std::mutex> lock(g_na_mutex);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNaMaxDev)
        return na_fail(MDG_E_CUDA, "mdg_recip_forces_noalloc: no current CUDA device");
    if (!g_na_ptr[dev]) {
        // once per device, with that device current: the device address of the static scratch
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) return na_fail(MDG_E_CUDA, "mdg_recip_forces_noalloc: cudaGetSymbolAddress failed");
        g_na_ptr[dev] = static_cast<unsigned char*>(p);
    }
    unsigned char* base = g_na_ptr[dev];
    // k set in the reference's order and selection (src/forcem.f90:743-776)
    const double pi_r = (double)3.1415926535898f;
    const double PH_e = (double)1.6021892e-19f, PH_Na = (double)6.022045e23f, PH_eps0 = (double)8.85418782e-12f,
                 PH_A2m = (double)1.0e-10f;
    const double pipix = 2.0 * pi_r / lx, pipiy = 2.0 * pi_r / ly, pipiz = 2.0 * pi_r / lz;
    const double alf4i = -1.0 / (4.0 * alpha * alpha);
    const double fac = 2.0 * PH_e * PH_e * PH_Na / (PH_eps0 * PH_A2m * 1000.0 * lx * ly * lz);
    const double lmin = std::min(lx, std::min(ly, lz));
    const double rk = (double)(float)kmax;
    const int KL = (int)std::lround(rk * lx / lmin), KM = (int)std::lround(rk * ly / lmin),
              KN = (int)std::lround(rk * lz / lmin);
    const float lim = (float)(kmax * kmax) + 2.01f;
    int nk = 0, nrow = 0, nwork = 0;
    int kmmin = 0, knmin = 1;
    for (int kl = 0; kl <= KL; ++kl) {
        const double rl = pipix * (double)(float)kl;
        for (int km = kmmin; km <= KM; ++km) {
            const double rm = pipiy * (double)(float)km;
            int first = 0, cnt = 0;
            for (int kn = knmin; kn <= KN; ++kn) {
                volatile float a = (float)(kl * kl + km * km);
                volatile float b = (float)((int64_t)kn * kn * kmax * kmax) / (float)((int64_t)KN * KN);
                volatile float ksq = a + b;
                if (!(ksq < lim)) continue;
                if (nk >= kNaMaxK) return na_fail(MDG_E_UNSUPPORTED, "mdg_recip_forces_noalloc: more than MDG_NOALLOC_MAX_K k vectors");
                const double rn = pipiz * (double)(float)kn;
                const double rksq = rl * rl + rm * rm + rn * rn;
                if (cnt == 0) first = kn;
                ++cnt;
                g_na_ak[nk++] = fac * std::exp(rksq * alf4i) / rksq;
            }
            if (cnt > 0) {
                if (nrow >= kNaMaxRows) return na_fail(MDG_E_UNSUPPORTED, "mdg_recip_forces_noalloc: too many k rows");
                g_na_rows[nrow] = make_int4(kl, km, first, nk - cnt);
                g_na_nlen[nrow] = cnt;
                ++nrow;
            }
            knmin = -KN;
        }
        kmmin = -KM;
    }
    if (nk == 0) return na_fail(MDG_E_ARG, "mdg_recip_forces_noalloc: empty k set");
    const KDims d{KL, KM, KN, pipix, pipiy, pipiz};
    if (!tables_fit(d))
        return na_fail(MDG_E_UNSUPPORTED, "mdg_recip_forces_noalloc: kmax too large for the phase tables");
    if (sfac_items(g_na_rows, g_na_nlen, nrow, g_na_ent, g_na_wr, g_na_wn, nwork) > kNaMaxEnt)
        return na_fail(MDG_E_UNSUPPORTED, "mdg_recip_forces_noalloc: too many k rows");
    auto ck = [](cudaError_t e) { return e == cudaSuccess; };
    if (!ck(allow_max_smem(k_sfac)) ||
        !ck(allow_max_smem(k_kforce)))
        return na_fail(MDG_E_CUDA, "mdg_recip_forces_noalloc: cudaFuncSetAttribute failed");
    double2* S = reinterpret_cast<double2*>(base + kNaS);
    double2* C = reinterpret_cast<double2*>(base + kNaC);
    double* Ak = reinterpret_cast<double*>(base + kNaAk);
    int4* rows = reinterpret_cast<int4*>(base + kNaRows);
    int* nlen = reinterpret_cast<int*>(base + kNaNlen);
    int* ent = reinterpret_cast<int*>(base + kNaEnt);
    int* wr = reinterpret_cast<int*>(base + kNaWr);
    int* wn = reinterpret_cast<int*>(base + kNaWn);
    double* acc = reinterpret_cast<double*>(base + kNaAcc);
    int* status = reinterpret_cast<int*>(base + kNaStatus);
    // the array keeps the previous call's contents: clear what the sums start from
    bool ok = ck(cudaMemcpyAsync(Ak, g_na_ak, sizeof(double) * nk, cudaMemcpyHostToDevice, st)) &&
              ck(cudaMemcpyAsync(rows, g_na_rows, sizeof(int4) * nrow, cudaMemcpyHostToDevice, st)) &&
              ck(cudaMemcpyAsync(nlen, g_na_nlen, sizeof(int) * nrow, cudaMemcpyHostToDevice, st)) &&
              ck(cudaMemcpyAsync(ent, g_na_ent, sizeof(int) * nrow, cudaMemcpyHostToDevice, st)) &&
              ck(cudaMemcpyAsync(wr, g_na_wr, sizeof(int) * nwork, cudaMemcpyHostToDevice, st)) &&
              ck(cudaMemcpyAsync(wn, g_na_wn, sizeof(int) * nwork, cudaMemcpyHostToDevice, st)) &&
              ck(cudaMemsetAsync(S, 0, sizeof(double2) * nk, st)) &&
              ck(cudaMemsetAsync(acc, 0, sizeof(double) * 64, st)) &&
              ck(cudaMemsetAsync(status, 0, sizeof(int) * ST_NWORDS, st)) &&
              ck(cudaMemsetAsync(fx, 0, sizeof(double) * n, st)) && ck(cudaMemsetAsync(fy, 0, sizeof(double) * n, st)) &&
              ck(cudaMemsetAsync(fz, 0, sizeof(double) * n, st));
    if (!ok) return na_fail(MDG_E_CUDA, "mdg_recip_forces_noalloc: copy of the k tables failed");
    View v{};
    v.nmove = (int)n;
    v.ntota = (int)n;
    v.nijt = 0;
    v.x = const_cast<double*>(x);
    v.y = const_cast<double*>(y);
    v.z = const_cast<double*>(z);
    v.q = q;
    v.fx = fx;
    v.fy = fy;
    v.fz = fz;
    v.acc = acc;
    v.status = status;
    const KGrid g = k_grid(d, (int)n, nrow, nwork);
    k_sfac<<<g.sfac, kSfacNT, g.smem_sfac, st>>>(v, d, nrow, rows, wr, wn, nwork, g.tile, g.atoms_per_split, S, nk);
    k_kenergy<<<std::min((nrow + 7) / 8, 256), 256, 0, st>>>(v, nrow, rows, nlen, ent, Ak, S, nullptr, C);
    k_kforce<<<g.force, kForceNT, g.smem_force, st>>>(v, d, nrow, rows, nlen, ent, C);
    k_noalloc_energy<<<1, 32, 0, st>>>(acc, uewa);
    if (cudaGetLastError() != cudaSuccess) return na_fail(MDG_E_CUDA, "mdg_recip_forces_noalloc: launch failed");
    return MDG_OK;
}

}  // namespace mdg
