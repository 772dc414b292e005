// pair.cu - real-space forces of force_real (src/forcem.f90:233-552).
//
//   k_pair_fp64   head-head pairs with the molecular cutoff, LJ/Buckingham on the heads,
//                 Ewald erfc on every site pair (src/forcem.f90:288-403)
//   k_wall_fp64   head-wall pairs: vdW on the head, erfc for each site of the head molecule
//                 against the frozen wall atom, wall reaction sums fws (src/forcem.f90:418-498)
//   k_surf_part   z forces of surface atoms booked to the wall they sit on (:408-413)
//   k_lr_tail     analytic wall long-range tail (:509-543, slab variant only)
//
// Layout: a unit of work is a head atom and every parts-th chunk of 32 of its list; one warp walks
// it.  The FP64 pipe bounds both loops, and an instruction there costs the same whatever the number
// of active lanes, so partners inside the cutoff go through a queue in shared memory and are
// evaluated 32 at a time (the list also holds the skin's), with the pair functions from a table
// (erfc_table.cuh).  The i-side site forces stay in registers and are reduced over the warp at the
// end (one atomic per component); j-side forces go out as FP64 atomics.  Energies are booked per
// head type pair (elj/eqq(ijt), src/forcem.f90:317,338,378) into shared memory, then once per block
// to HBM.  Blocks of four warps are dealt by the hardware as they finish: heads differ in partners
// (j > i), and with few heads the parts spread them over the SMs.
// Against one warp per list, blocks of eight, every list entry evaluated in place and the functions
// evaluated directly: head-head 212 -> 27 us at 256 waters, 259 -> 123 us in a 2,048-water slab and
// 3.7 -> 1.8 ms at 32,768; head-wall 218 -> 70 us in the slab.  FP64 operations are still what bounds
// them (about 300 per partner; a batch of 32 lanes is on average 80 % full).
#include <algorithm>

#include "common.cuh"
#include "ctx.h"
#include "erfc_table.cuh"
#include "lr_tail.cuh"

namespace mdg {

namespace {

constexpr int kWarps = 4;
constexpr int kNT = kWarps * 32;

struct EAcc {
    int ijt = -1;
    double lj = 0.0, qq = 0.0;
};

__device__ __forceinline__ void e_flush(EAcc& e, double* s_e, int nijt) {
    if (e.ijt >= 0 && (e.lj != 0.0 || e.qq != 0.0)) {
        atomicAdd(&s_e[e.ijt], e.lj);
        atomicAdd(&s_e[nijt + e.ijt], e.qq);
    }
    e.lj = e.qq = 0.0;
}

// End of the loops: lanes holding the warp's (largest) pair type reduce with shuffles, one shared
// atomic per warp; lanes left with another type flush one by one.
__device__ __forceinline__ void e_final(EAcc& e, double* s_e, int nijt) {
    const int ij0 = __reduce_max_sync(0xffffffffu, e.ijt);
    if (ij0 < 0) return;
    const bool mine = e.ijt == ij0;
    const double lj = warp_sum(mine ? e.lj : 0.0);
    const double qq = warp_sum(mine ? e.qq : 0.0);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_e[ij0], lj);
        atomicAdd(&s_e[nijt + ij0], qq);
    }
    if (!mine) e_flush(e, s_e, nijt);
}

__device__ __forceinline__ void e_add(EAcc& e, int ijt, double lj, double qq, double* s_e, int nijt) {
    if (ijt != e.ijt) {
        e_flush(e, s_e, nijt);
        e.ijt = ijt;
    }
    e.lj += lj;
    e.qq += qq;
}

// Sums of nine values over the warp: lane 4 k gets that of v[k] for k < 8, every lane that of v[8].
__device__ __forceinline__ double2 warp_sum9(const double v[9]) {
    const int lane = threadIdx.x & 31;
    double a[4], b[2];
    const bool u16 = lane & 16, u8 = lane & 8, u4 = lane & 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double keep = u16 ? v[k + 4] : v[k], send = u16 ? v[k] : v[k + 4];
        a[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double keep = u8 ? a[k + 2] : a[k], send = u8 ? a[k] : a[k + 2];
        b[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    double c = (u4 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, u4 ? b[0] : b[1], 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    return make_double2(c, warp_sum(v[8]));
}

// Sites of a unit's head molecule: offsets from the head, charges times facq alpha, forces.
struct Head {
    double rx[3], ry[3], rz[3], q[3];
    double fx[3], fy[3], fz[3];
    __device__ __forceinline__ void load(const View& v, int i, int nsi) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const bool ok = a < nsi;
            rx[a] = ok ? v.rsx[CK(i + a, v.nmove, 105)] : 0.0;
            ry[a] = ok ? v.rsy[CK(i + a, v.nmove, 105)] : 0.0;
            rz[a] = ok ? v.rsz[CK(i + a, v.nmove, 105)] : 0.0;
            q[a] = ok ? v.facq * v.alfa * v.q[CK(i + a, v.ntota, 106)] : 0.0;
            fx[a] = fy[a] = fz[a] = 0.0;
        }
    }
    // adds the warp's forces to the sites and, with ws, their negative sum to ws[0..2]; clears them
    __device__ __forceinline__ void store(const View& v, int i, int nsi, double* ws) {
        const int lane = threadIdx.x & 31;
        const double f[9] = {fx[0], fy[0], fz[0], fx[1], fy[1], fz[1], fx[2], fy[2], fz[2]};
        const double2 s = warp_sum9(f);
        const int k = lane == 1 ? 8 : (lane & 3) == 0 ? lane >> 2 : 9;
        if (k < 3 * nsi) {
            const int site = k / 3, d = k - 3 * site;
            const double val = k == 8 ? s.y : s.x;
            atomicAdd((d == 0 ? v.fx : d == 1 ? v.fy : v.fz) + CK(i + site, v.nmove, 119), val);
            if (ws) atomicAdd(ws + d, -val);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) fx[a] = fy[a] = fz[a] = 0.0;
    }
};

// A warp's partners inside the cutoff: separation and index, a ring of 64.
struct QueueMem {
    double x[64], y[64], z[64];
    int j[64];
};
struct Queue {
    QueueMem* m;
    int head = 0, n = 0;
    __device__ __forceinline__ void push(bool in, double dx, double dy, double dz, int j) {
        const unsigned b = __ballot_sync(0xffffffffu, in), lt = (1u << (threadIdx.x & 31)) - 1u;
        const int k = (head + n + __popc(b & lt)) & 63;
        if (in) {
            m->x[k] = dx;
            m->y[k] = dy;
            m->z[k] = dz;
            m->j[k] = j;
        }
        n += __popc(b);
        __syncwarp();
    }
    __device__ __forceinline__ void pop() {
        head = (head + 32) & 63;
        n = max(n - 32, 0);
        __syncwarp();
    }
};

// vdW of a head pair (src/forcem.f90:313-330): energy, and the force factor.
__device__ __forceinline__ double vdw_pair(const View& v, int ijt, double rsq, double& fij) {
    const int vk = v.vdw[ijt];
    if (vk == 1) {
        const double rsqi = 1.0 / rsq;
        const double r6 = v.sig[ijt] * (rsqi * rsqi * rsqi);
        fij = 6.0 * rsqi * v.eps[ijt] * r6 * (2.0 * r6 - 1.0);
        return v.eps[ijt] * r6 * (r6 - 1.0);
    }
    if (vk == 2) {
        const double rinv = rsqrt(rsq), rsqi = rinv * rinv;
        const double r6 = v.cc[ijt] * (rsqi * rsqi * rsqi);
        const double aux = v.aa[ijt] * exp(-(rsq * rinv) * v.rhoi[ijt]);
        fij = aux * v.rhoi[ijt] * rinv - 6.0 * rsqi * r6;
        return aux - r6;
    }
    fij = 0.0;
    return 0.0;
}

__global__ void __launch_bounds__(kNT) k_pair_fp64(View v, int parts) {
    extern __shared__ double s_e[];  // 2 * nijt
    __shared__ QueueMem s_q[kWarps];
    for (int k = threadIdx.x; k < 2 * v.nijt; k += blockDim.x) s_e[k] = 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const double alfa2 = v.alfa * v.alfa;
    EAcc e;
    for (int un = blockIdx.x * kWarps + (threadIdx.x >> 5); un < v.nheads * parts; un += gridDim.x * kWarps) {
        const int h = un / parts, part = un - h * parts;
        const int n = v.nbcnt[CK(h, v.nheads, 107)];
        if (32 * part >= n) continue;
        const int i = v.head_atom[CK(h, v.nheads, 101)];
        const int it = v.type[CK(i, v.ntota, 102)];
        const int nsi_i = v.nsi[CK(it, v.nit, 103)];
        const double xi0 = v.x[CK(i, v.ntota, 104)], yi0 = v.y[CK(i, v.ntota, 104)], zi0 = v.z[CK(i, v.ntota, 104)];
        Head H;
        H.load(v, i, nsi_i);
        const int* nb = v.nb + (size_t)CK(h, v.nheads, 120) * v.maxnb;
        Queue Q{&s_q[threadIdx.x >> 5]};
        auto evaluate = [&]() {
            if (lane >= Q.n) return;
            const int s = (Q.head + lane) & 63;
            const double xio = Q.m->x[s], yio = Q.m->y[s], zio = Q.m->z[s];
            const int j = Q.m->j[s];
            const int jt = v.type[CK(j, v.ntota, 110)];
            const int ijt = CK(v.ijt[CK(it * v.nit + jt, v.nit * v.nit, 111)], v.nijt, 112);
            const int nsi_j = v.nsi[CK(jt, v.nit, 113)];
            double fjx[3], fjy[3], fjz[3], rjx[3], rjy[3], rjz[3], qj[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const bool ok = b < nsi_j;
                rjx[b] = ok ? v.rsx[CK(j + b, v.nmove, 115)] : 0.0;
                rjy[b] = ok ? v.rsy[CK(j + b, v.nmove, 115)] : 0.0;
                rjz[b] = ok ? v.rsz[CK(j + b, v.nmove, 115)] : 0.0;
                qj[b] = ok ? v.q[CK(j + b, v.ntota, 116)] : 0.0;
                fjx[b] = fjy[b] = fjz[b] = 0.0;
            }
            double eqq = 0.0, elj = 0.0;
            // all site pairs (src/forcem.f90:306-402), the heads' own with the vdW force
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (a >= nsi_i) break;
                const double xa = xio + H.rx[a], ya = yio + H.ry[a], za = zio + H.rz[a];
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    if (b >= nsi_j) break;
                    const bool hh = a == 0 && b == 0;  // the heads' own distance
                    const double xd = hh ? xio : xa - rjx[b], yd = hh ? yio : ya - rjy[b], zd = hh ? zio : za - rjz[b];
                    const double r2 = xd * xd + yd * yd + zd * zd;
                    const double2 gh = ewald_gh(alfa2 * r2, v.etab, v.spii);
                    const double qq = H.q[a] * qj[b];
                    eqq += qq * gh.x;
                    double fs = alfa2 * qq * gh.y;
                    if (hh) {
                        double fv;
                        elj = vdw_pair(v, ijt, r2, fv);
                        fs += fv;
                    }
                    H.fx[a] += xd * fs; H.fy[a] += yd * fs; H.fz[a] += zd * fs;
                    fjx[b] -= xd * fs; fjy[b] -= yd * fs; fjz[b] -= zd * fs;
                }
            }
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                if (b >= nsi_j) break;
                atomicAdd(&v.fx[CK(j + b, v.nmove, 118)], fjx[b]);
                atomicAdd(&v.fy[CK(j + b, v.nmove, 118)], fjy[b]);
                atomicAdd(&v.fz[CK(j + b, v.nmove, 118)], fjz[b]);
            }
            e_add(e, ijt, elj, eqq, s_e, v.nijt);
        };
        for (int k0 = 32 * part;; k0 += 32 * parts) {
            const bool more = k0 < n;
            if (more) {
                const int k = k0 + lane;
                double dx = 0.0, dy = 0.0, dz = 0.0;
                int j = 0;
                bool in = k < n;
                if (in) {
                    j = nb[CK(k, v.maxnb, 108)];
                    dx = minimg(xi0 - v.x[CK(j, v.nmove, 109)], v.lx, v.lxi);
                    dy = minimg(yi0 - v.y[j], v.ly, v.lyi);
                    dz = zi0 - v.z[j];
                    if (v.bulk) dz = minimg(dz, v.lz, v.lzi);
                    in = !(dx * dx + dy * dy + dz * dz > v.rcutsq);
                }
                Q.push(in, dx, dy, dz, j);
            }
            if (Q.n >= 32 || (!more && Q.n > 0)) {
                evaluate();
                Q.pop();
            }
            if (!more) break;
        }
        H.store(v, i, nsi_i, nullptr);
    }
    e_final(e, s_e, v.nijt);
    __syncthreads();
    for (int k = threadIdx.x; k < 2 * v.nijt; k += blockDim.x)
        if (s_e[k] != 0.0) atomicAdd(&v.acc[k], s_e[k]);
}

__global__ void __launch_bounds__(kNT) k_wall_fp64(View v, int parts) {
    extern __shared__ double s_e[];  // 2 * nijt + 6 (fws x,y,z for sgn -1 / +1)
    __shared__ QueueMem s_q[kWarps];
    for (int k = threadIdx.x; k < 2 * v.nijt + 6; k += blockDim.x) s_e[k] = 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const double alfa2 = v.alfa * v.alfa;
    // energy sums per wall site type (the last two site types alternate from partner to partner)
    EAcc ew[2];
    const int wt0 = v.nit - 2;
    for (int un = blockIdx.x * kWarps + (threadIdx.x >> 5); un < v.nheads * parts; un += gridDim.x * kWarps) {
        const int h = un / parts, part = un - h * parts;
        const int n = v.wnbcnt[h];
        if (32 * part >= n) continue;
        const int i = v.head_atom[h];
        const int it = v.type[i];
        const int nsi_i = v.nsi[it];
        const bool book = (it + 1) <= v.nltype;  // `it <= nltype` on 1-based ids (src/forcem.f90:481)
        const double xi0 = v.x[i], yi0 = v.y[i], zi0 = v.z[i];
        Head H;
        H.load(v, i, nsi_i);
        int side = -1;  // the wall (0: z < 0, 3: z > 0) that H's forces come from
        const int* nb = v.wnb + (size_t)h * v.maxwnb;
        Queue Q{&s_q[threadIdx.x >> 5]};
        auto store = [&]() { H.store(v, i, nsi_i, book ? s_e + 2 * v.nijt + side : nullptr); };
        auto evaluate = [&](bool on, int s) {
            if (!on) return;
            const double xi = Q.m->x[s], yi = Q.m->y[s], zi = Q.m->z[s];
            const int j = Q.m->j[s] & 0x7fffffff;
            const int jt = v.type[j], ijt = v.ijt[it * v.nit + jt];
            const double qj = v.q[j];
            double eqq = 0.0, elj = 0.0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (a >= nsi_i) break;
                const double xd = xi + H.rx[a], yd = yi + H.ry[a], zd = zi + H.rz[a];
                const double r2 = xd * xd + yd * yd + zd * zd;
                const double2 gh = ewald_gh(alfa2 * r2, v.etab, v.spii);
                const double qq = H.q[a] * qj;
                eqq += qq * gh.x;
                double fs = alfa2 * qq * gh.y;
                if (a == 0) {
                    double fv;
                    elj = vdw_pair(v, ijt, xi * xi + yi * yi + zi * zi, fv);
                    fs += fv;
                }
                H.fx[a] += xd * fs; H.fy[a] += yd * fs; H.fz[a] += zd * fs;
            }
            if (jt <= wt0) e_add(ew[0], ijt, elj, eqq, s_e, v.nijt);
            else e_add(ew[1], ijt, elj, eqq, s_e, v.nijt);
        };
        for (int k0 = 32 * part;; k0 += 32 * parts) {
            const bool more = k0 < n;
            if (more) {
                const int k = k0 + lane;
                double dx = 0.0, dy = 0.0, dz = 0.0;
                int j = 0;
                bool in = k < n;
                if (in) {
                    j = nb[k];
                    const double zj = v.z[j];
                    dx = minimg(xi0 - v.x[j], v.lx, v.lxi);
                    dy = minimg(yi0 - v.y[j], v.ly, v.lyi);
                    dz = zi0 - zj;
                    if (v.bulk) dz = minimg(dz, v.lz, v.lzi);
                    in = !(dx * dx + dy * dy + dz * dz > v.rcutsq);
                    if (!signbit(zj)) j |= (int)0x80000000;  // which wall rides on the index
                }
                Q.push(in, dx, dy, dz, j);
            }
            if (Q.n >= 32 || (!more && Q.n > 0)) {
                // a head between two near walls has partners of both: one after the other
                const bool on = lane < Q.n;
                const int s = (Q.head + lane) & 63;
                const bool up = Q.m->j[s] < 0;
                const unsigned sides[2] = {__ballot_sync(0xffffffffu, on && !up), __ballot_sync(0xffffffffu, on && up)};
#pragma unroll 1
                for (int w = 0; w < 2; ++w) {
                    if (!(w ? sides[1] : sides[0])) continue;
                    if (side >= 0 && side != 3 * w) store();
                    side = 3 * w;
                    evaluate(on && up == (w != 0), s);
                }
                Q.pop();
            }
            if (!more) break;
        }
        if (side >= 0) store();
    }
    e_final(ew[0], s_e, v.nijt);
    e_final(ew[1], s_e, v.nijt);
    __syncthreads();
    for (int k = threadIdx.x; k < 2 * v.nijt; k += blockDim.x)
        if (s_e[k] != 0.0) atomicAdd(&v.acc[k], s_e[k]);
    if (threadIdx.x < 6) {
        // fws layout: [x(-1),x(0),x(1), y(-1),y(0),y(1), z(-1),z(0),z(1)]
        const int comp = threadIdx.x % 3, sg = threadIdx.x / 3;  // sg 0 -> -1, 1 -> +1
        const double s = s_e[2 * v.nijt + threadIdx.x];
        if (s != 0.0) atomicAdd(&v.acc[2 * v.nijt + ACC_FWS + comp * 3 + (sg ? 2 : 0)], s);
    }
}

// fwsz(sign(z0(i))) += fz(i) for surface atoms, right after the head-head loop.
__global__ void k_surf_part(View v) {
    double lo = 0.0, hi = 0.0;
    for (int i = v.nliqa + blockIdx.x * blockDim.x + threadIdx.x; i < v.nmove; i += gridDim.x * blockDim.x) {
        if (signbit(v.z[i])) lo += v.fz[i];
        else hi += v.fz[i];
    }
    block_atomic_sum<kNT>(lo, &v.acc[2 * v.nijt + ACC_FWS + 6 + 0]);
    block_atomic_sum<kNT>(hi, &v.acc[2 * v.nijt + ACC_FWS + 6 + 2]);
}

__global__ void __launch_bounds__(kLrNT) k_lr_tail(View v, const double* lr) { lr_tail_block(v, lr, blockIdx.x, gridDim.x); }

// Parts of a head's list: enough warps for every SM where heads are few; more parts leave queues that
// end less than half full.  1, 2, 3, 4, 8 parts: 256 heads 50, 34, 38, 27, 41 us; 2,048 heads 146, 123,
// 135, 138, 146 us (walls 77, 70, 78, 73, 80).  One part from 2,049 heads on: with 1 and 2 parts 2,197 bulk heads
// 170 and 154 us but whole force calls, beside the reciprocal sum, 458 and 463; 2,744 heads 207 and 180, calls 524
// and 532; slabs of 2,600 heads 141 and 155, calls 536 and 555, of 6,000 heads 300 and 330, calls 1,081 and 1,125.
int list_parts(int nheads) { return std::max(1, std::min(4, 4096 / nheads)); }
int pair_blocks(int units) { return std::max(1, std::min((units + kWarps - 1) / kWarps, 152 * 64)); }

}  // namespace

// The table lives in a static device array: one per GPU, the same bytes for every context.
static __device__ __align__(128) double g_etab[kEtRows * 16];

int pair_setup(Ctx& c) {
    if (c.precision == MDG_MIXED) return MDG_OK;
    static const std::vector<double> table = ewald_table(c.v.spii);  // of the functions, no system's own
    void* p = nullptr;
    MDG_CUDA(cudaGetSymbolAddress(&p, g_etab));
    MDG_CUDA(cudaMemcpy(p, table.data(), sizeof(double) * table.size(), cudaMemcpyHostToDevice));
    c.v.etab = static_cast<const double2*>(p);
    // the energy sums share a block's 48 KB with the queues (7 KB); a kernel takes more only where allowed
    if (sizeof(double) * (2 * c.v.nijt + 6) > 32 * 1024) {
        MDG_CUDA(allow_max_smem(k_pair_fp64));
        MDG_CUDA(allow_max_smem(k_wall_fp64));
    }
    return MDG_OK;
}

void pair_forces_fp64(Ctx& c) {
    const View& v = c.v;
    if (v.nheads == 0) return;
    const int parts = list_parts(v.nheads);
    k_pair_fp64<<<pair_blocks(v.nheads * parts), kNT, sizeof(double) * 2 * v.nijt, c.stream>>>(v, parts);
}

void wall_forces_fp64(Ctx& c) {
    const View& v = c.v;
    if (v.nheads == 0 || v.nwall == 0) return;
    const int parts = list_parts(v.nheads);
    k_wall_fp64<<<pair_blocks(v.nheads * parts), kNT, sizeof(double) * (2 * v.nijt + 6), c.stream>>>(v, parts);
}

void surf_partition(Ctx& c) {
    const View& v = c.v;
    if (v.nmove <= v.nliqa) return;
    k_surf_part<<<std::min((v.nmove - v.nliqa + kNT - 1) / kNT, 64), kNT, 0, c.stream>>>(v);
}

void lr_tail(Ctx& c) {
    const View& v = c.v;
    if (c.variant != MDG_SLAB || v.nmove == 0) return;
    k_lr_tail<<<std::min((v.nmove + kLrNT - 1) / kLrNT, 152 * 8), kLrNT, 0, c.stream>>>(v, c.d_lr);
}

}  // namespace mdg
