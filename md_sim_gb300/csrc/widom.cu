// widom.cu - Widom test-particle insertion of a rigid 3-site water (chempot, src/forcem.f90:1226-1507).
//
// The host draws the positions and orientations with the reference's congruential generator
// (src/rndmod.f90:26-35) in the reference's order, assuming every position is accepted, and
// records the generator state after each position and after its orientations, a chunk of positions while the
// device evaluates the one before; the device makes the orientations from the states they start at.
// (2,000 positions: 4.9 ms a call when they were drawn with fmod, up front and on one buffer, 1.46 ms now,
// about 1 ms of it the drawing of 40,000 orientations.)  What an insertion needs:
//   - all sites against the O of the probe: overlap test (2.35 A to a water O, 2 A to others,
//     src/forcem.f90:1303-1313), vdW + Ewald erfc of the O (src/forcem.f90:1315-1334) and the
//     neighbour list within rcut (every site that is not of the H type), kept in shared memory;
//   - per orientation, the Ewald erfc terms of the probe's sites against the neighbours' sites
//     (src/forcem.f90:1378-1423), the reciprocal term 0.5 Ak Re(sum_s q_s e^{ik r_s} conj(Qsum))
//     (src/forcem.f90:1428-1474), the optional slab term and the O's wall tail (:1481-1494);
//     exp(-beta u) summed over the orientations.
// The host keeps the positions up to the first overlap (the reference leaves the insertion loop
// there, src/forcem.f90:1342) unless MDG_WIDOM_SKIP_OVERLAP is set, and accumulates pave/inave.
//
// FP64 contexts (FP64 operations bound it, so the kernels are cut to have few of them):
//   k_widom_atoms  the sites that are not of the H type, in the box, in FP32
//   k_widom_real   a CTA per position.  A scan in FP32 picks the sites that may be inside the cutoff
//                  (margin far above FP32 rounding), these are tested in FP64; a site certainly too
//                  near ends the position.  Terms of the O are summed once, those of the two H over
//                  (orientation, neighbour) pairs dealt evenly to the threads, with the pair
//                  function from a table (erfc_table.cuh).  Accepted positions append their points (the
//                  O, two H per orientation) to one list.
//   k_pot          (recip.cu) sum_k Ak Re(e^{ik r} conj(Qsum)) at all points of all positions: the O's once
//                  per position, 2 FMAs per k and point where the product of the phase factors of
//                  three sites per orientation takes about 37 operations per k
//   k_widom_sum    energies and exponentials, a warp per position
// 2,000 positions in a 2,048-water slab (4,338 k, 7,744 sites): 4.64 ms in one kernel per position before,
// now 0.31 ms (k_pot), 0.23 ms (k_widom_real) and 0.015 ms for the other three.
// Mixed contexts: k_widom, one CTA per position, the orientation loop in FP32 (block sums, the O's scan,
// the wall tail and the exponential stay FP64).
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "ctx.h"
#include "erfc_table.cuh"

namespace mdg {

namespace {

constexpr int kWT = 256;        // threads per insertion
constexpr int kWNb = 1024;      // neighbour capacity per insertion
constexpr int kMaxRot = 20;
constexpr int kIns = 512;       // positions drawn, copied and evaluated at a time
constexpr int kDraw = 4 + kMaxRot;  // doubles per position: O and orientations, generator states

// The reference's generator (src/rndmod.f90:26-35): seed <- mod(8192 seed, 67099547).
constexpr double kRndMod = 67099547.0, kRndScale = 1.4903230270690e-8;

// Its states one after the other, drawn ahead 1,024 at a time: from an integer state (what any integer seed
// gives) eight interleaved chains of integer arithmetic, each eight steps a turn, with the same values
// as fmod one by one, whose latency was most of a call (40 ns a number, 4.3 ms of a call with 2,000 positions).
class Generator {
public:
    explicit Generator(double seed) : last_(seed) {}
    double state() {
        if (k_ == kAhead) fill();
        return buf_[k_++];
    }
    double number() { return state() * kRndScale; }

private:
    static constexpr int kAhead = 1024;
    void fill() {
        constexpr uint64_t M = 67099547;
        const double first = std::fmod(8192.0 * last_, kRndMod);
        if (first >= 0.0 && first == std::floor(first)) {
            uint64_t x[8] = {(uint64_t)first}, a = 8192;  // products stay below 2^52
            for (int i = 1; i < 8; ++i) {
                x[i] = x[i - 1] * 8192 % M;
                a = a * 8192 % M;
            }
            for (int k = 0; k < kAhead; k += 8)
                for (int i = 0; i < 8; ++i) {
                    buf_[k + i] = (double)x[i];
                    x[i] = x[i] * a % M;
                }
        } else {
            buf_[0] = first;
            for (int k = 1; k < kAhead; ++k) buf_[k] = std::fmod(8192.0 * buf_[k - 1], kRndMod);
        }
        last_ = buf_[kAhead - 1];
        k_ = 0;
    }
    double last_, buf_[kAhead];
    int k_ = kAhead;
};

struct WArgs {
    const double4* pos;   // O position per insertion, w: its orientations
    const double* rot;    // [ins][kMaxRot][6]: H1 x y z, H2 x y z (the reference's rins(2,:), rins(3,:))
    double2* res;         // (sum exp(-beta u), status: 0 accepted, 1 overlap, 2 neighbour overflow)
    const int3* kvec;     // k set in the reference's order
    const double* lr;     // [9][nit] wall tail tables
    int nk, KL, KM, KN;
    double pipix, pipiy, pipiz;
    double beta, rinsmin, rwinsmin, crf;
    double q0, q1;        // probe charges (O, H)
    // mixed form: FP32 operands of the orientation loop
    const float2* qsf;    // Qsum = S + S_wall in FP32
    const float* akf;     // Ak in FP32
    const float4* rsf;    // per site: rs offset (moving sites) and charge, FP32
};

__device__ __forceinline__ float ewald_ef(float rr, float alfa) {
    const float ar = alfa * rr;
    const float t = __fdividef(1.0f, 1.0f + (float)kP * ar);
    const float e2 = __expf(-ar * ar);
    return (((((float)kA5 * t + (float)kA4) * t + (float)kA3) * t + (float)kA2) * t + (float)kA1) * t * e2;
}

// FP32 operands of one call: Qsum per k, and per site its offset rs (as force_sum left it, like
// the reference's module array) and charge.
__global__ void k_widom_prep(View v, const double2* __restrict__ sk, const double2* __restrict__ qw, float2* qsf,
                             int nk, float4* rsf) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nk; k += gridDim.x * blockDim.x)
        qsf[k] = make_float2((float)(sk[k].x + qw[k].x), (float)(sk[k].y + qw[k].y));
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < v.ntota; a += gridDim.x * blockDim.x) {
        const bool mv = a < v.nmove;
        rsf[a] = make_float4(mv ? (float)v.rsx[a] : 0.f, mv ? (float)v.rsy[a] : 0.f, mv ? (float)v.rsz[a] : 0.f,
                             (float)v.q[a]);
    }
}

__device__ __forceinline__ double ewald_e(double rij, double alfa) {
    const double alfar = alfa * rij;
    const double t = 1.0 / (1.0 + kP * alfar);
    const double exp2a = exp(-alfar * alfar);
    return ((((kA5 * t + kA4) * t + kA3) * t + kA2) * t + kA1) * t * exp2a;
}

__device__ double block_sum_d(double x, double* red) {
    x = warp_sum(x);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = x;
    __syncthreads();
    double s = 0.0;
    for (int k = 0; k < kWT / 32; ++k) s += red[k];
    return s;
}

// Orientations (src/forcem.f90:1345-1377) from the generator's state at the first of their four numbers.
__global__ void k_widom_rot(const double4* __restrict__ pos, const double* __restrict__ states, double* __restrict__ rot,
                            int nins) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, ins = t / kMaxRot;
    if (ins >= nins) return;
    const double4 o = pos[ins];
    if (t - ins * kMaxRot >= (int)o.w) return;
    double sd = states[t], h1[3];
    for (int d = 0; d < 3; ++d) {
        h1[d] = sd * kRndScale - 0.5;
        sd = fmod(8192.0 * sd, kRndMod);
    }
    double ri = 1.0 / sqrt(h1[0] * h1[0] + h1[1] * h1[1] + h1[2] * h1[2]);
    for (int d = 0; d < 3; ++d) h1[d] *= ri;
    ri = 1.0 / sqrt(h1[0] * h1[0] + h1[1] * h1[1]);
    const double h2[3] = {-h1[1] * ri, h1[0] * ri, 0.0};
    const double mr[3] = {h2[1] * h1[2] - h2[2] * h1[1], h2[2] * h1[0] - h2[0] * h1[2], h2[0] * h1[1] - h2[1] * h1[0]};
    const double alph = 2.0 * (double)3.1415926535898f * (sd * kRndScale);
    double sina, cosa;
    sincos(alph, &sina, &cosa);
    const double aco = (double)-0.333333f, asi = (double)0.942809f, oo[3] = {o.x, o.y, o.z};
    for (int d = 0; d < 3; ++d) {
        rot[6 * (size_t)t + d] = oo[d] + aco * h1[d] + asi * (cosa * h2[d] + sina * mr[d]);
        rot[6 * (size_t)t + 3 + d] = oo[d] + h1[d];
    }
}

// The O's wall tail (src/forcem.f90:1481-1494).
__device__ double wall_tail(const View& v, const double* lr, double oz) {
    const int nit = v.nit;
    double u = 0.0;
    for (int j = -1; j <= 1; j += 2) {
        const double dw = v.lwh - (double)j * oz;
        if (dw < v.rcut) {
            u += lr[8 * nit];
        } else {
            u += lr[7 * nit];
            const double dw3 = dw * dw * dw;
            u += (lr[2 * nit] / (9.0 * (dw3 * dw3 * dw3)) - lr[3 * nit] / (3.0 * dw3));
            const double tt = lr[6 * nit];
            const double exp2a = lr[4 * nit] * exp(-dw / tt);
            u += (tt * (2.0 * tt + dw) * exp2a - lr[5 * nit] / (3.0 * dw3));
        }
    }
    return u;
}

constexpr int kRT = 128;           // threads per position of k_widom_real
constexpr int kCand = 2048;        // sites picked by its FP32 scan (more are tested where they are found)
constexpr int kPts = 1 + 2 * kMaxRot;

// FP64 form's scratch of one call.
struct W64 {
    float4* atoms;   // x, y (in the box), z, index
    int* cnt;        // sites in atoms, points
    int* off;        // first point of each accepted position
    double* u;       // [ins][kMaxRot] real-space energies
    double* xyz;     // points: x, y, z, stride apart
    double* phi;     // reciprocal potential at the points
    size_t stride;
    float lx, lxi, ly, lyi, near2, far2;  // below near2: certainly an overlap; above far2: certainly outside
};

__global__ void k_widom_atoms(View v, W64 s) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= v.ntota || v.type[a] == 1) return;
    const int k = atomicAdd(&s.cnt[0], 1);
    s.atoms[k] = make_float4((float)minimg(v.x[a], v.lx, v.lxi), (float)minimg(v.y[a], v.ly, v.lyi), (float)v.z[a],
                             __int_as_float(a));
}

__global__ void __launch_bounds__(kRT) k_widom_real(View v, WArgs w, W64 s) {
    __shared__ int cand[kCand], nb_j[kWNb];          // water neighbours from the front, others from the back
    __shared__ double nb_d[3 * kWNb];
    __shared__ double so[kMaxRot][6], su[kMaxRot];   // H offsets from the O, sums per orientation
    __shared__ double red[kRT / 32];
    __shared__ int s_nc, s_nw, s_no, s_flag, s_off;
    const int ins = blockIdx.x, t = threadIdx.x, lane = t & 31;
    const double4 o = w.pos[ins];
    const int nr = (int)o.w;
    if (t == 0) s_nc = s_nw = s_no = s_flag = 0;
    if (t < kMaxRot) su[t] = 0.0;
    __syncthreads();
    const double alfa2 = v.alfa * v.alfa, fq = v.facq * v.alfa;
    double ux = 0.0;
    // a site in FP64: overlap test, the O's terms with it (and, of a water, with its other sites), the list
    auto visit = [&](int j) {
        const int jt = v.type[j];
        const double zio = o.z - v.z[j];
        if (fabs(zio) > v.rcut) return;
        const double xio = minimg(o.x - v.x[j], v.lx, v.lxi);
        const double yio = minimg(o.y - v.y[j], v.ly, v.lyi);
        const double rsq = xio * xio + yio * yio + zio * zio;
        if (rsq > v.rcutsq) return;
        if (rsq < w.rwinsmin && (jt == 0 || rsq < w.rinsmin)) {
            atomicOr(&s_flag, 1);
            return;
        }
        const int ijt = v.ijt[jt];  // it = 1 (the water O type)
        const int vk = v.vdw[ijt];
        if (vk == 1) {
            const double rsqi = 1.0 / rsq;
            const double r6 = v.sig[ijt] * (rsqi * rsqi * rsqi);
            ux += v.eps[ijt] * r6 * (r6 - 1.0);
        } else if (vk == 2) {
            const double rsqi = 1.0 / rsq;
            const double r6 = v.cc[ijt] * (rsqi * rsqi * rsqi);
            ux += v.aa[ijt] * exp(-sqrt(rsq) * v.rhoi[ijt]) - r6;
        }
        double e = v.q[j] * ewald_g(alfa2 * rsq, v.etab, v.spii);
        if (jt == 0)
            for (int jx = j + 1; jx < j + v.nsi[0]; ++jx) {
                const double xd = xio - v.rsx[jx], yd = yio - v.rsy[jx], zd = zio - v.rsz[jx];
                e += v.q[jx] * ewald_g(alfa2 * (xd * xd + yd * yd + zd * zd), v.etab, v.spii);
            }
        ux += fq * w.q0 * e;
        const int k = jt == 0 ? atomicAdd(&s_nw, 1) : kWNb - 1 - atomicAdd(&s_no, 1);
        if (k >= 0 && k < kWNb) {
            nb_j[k] = j;
            nb_d[3 * k + 0] = xio;
            nb_d[3 * k + 1] = yio;
            nb_d[3 * k + 2] = zio;
        }
    };
    {
        const float ox = (float)minimg(o.x, v.lx, v.lxi), oy = (float)minimg(o.y, v.ly, v.lyi), oz = (float)o.z;
        const int na = s.cnt[0];
#pragma unroll 4
        for (int k = t; k < na; k += kRT) {
            const float4 a = s.atoms[k];
            float dx = ox - a.x, dy = oy - a.y;
            const float dz = oz - a.z;
            dx -= s.lx * rintf(dx * s.lxi);
            dy -= s.ly * rintf(dy * s.lyi);
            const float r2 = dx * dx + dy * dy + dz * dz;
            if (r2 > s.far2) continue;
            if (r2 < s.near2) s_flag = 1;
            const int c = atomicAdd(&s_nc, 1);
            if (c < kCand) cand[c] = __float_as_int(a.w);
            else visit(__float_as_int(a.w));
        }
    }
    __syncthreads();
    if (!(s_flag & 1))
        for (int c = t; c < min(s_nc, kCand); c += kRT) visit(cand[c]);
    __syncthreads();
    const int nw = s_nw, no = s_no;
    if ((s_flag & 1) || nw + no > kWNb) {
        if (t == 0) w.res[ins] = make_double2(0.0, (s_flag & 1) ? 1.0 : 2.0);
        return;
    }
    ux = warp_sum(ux);
    if (lane == 0) red[t >> 5] = ux;
    // the points: the O, then H1 and H2 of each orientation
    if (t == 0) s_off = atomicAdd(&s.cnt[1], 1 + 2 * nr);
    __syncthreads();
    const double* rot = w.rot + (size_t)ins * kMaxRot * 6;
    for (int k = t; k < 1 + 2 * nr; k += kRT) {
        const size_t p = (size_t)s_off + k;
        const double x = k ? rot[3 * (k - 1)] : o.x, y = k ? rot[3 * (k - 1) + 1] : o.y, z = k ? rot[3 * (k - 1) + 2] : o.z;
        s.xyz[p] = x;
        s.xyz[s.stride + p] = y;
        s.xyz[2 * s.stride + p] = z;
        if (k) {
            double* d = &so[(k - 1) >> 1][3 * ((k - 1) & 1)];
            d[0] = x - o.x;
            d[1] = y - o.y;
            d[2] = z - o.z;
        }
    }
    __syncthreads();
    // both H of an orientation with the sites of one neighbour
    auto sweep = [&](int first, int cnt, bool water) {
        const int total = nr * cnt;
        for (int b = t - lane; b < total; b += kRT) {
            const int i = min(b + lane, total - 1), r = i / cnt, k = first + i - r * cnt, j = nb_j[k];
            double e = 0.0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double x = nb_d[3 * k] + so[r][3 * h], y = nb_d[3 * k + 1] + so[r][3 * h + 1],
                             z = nb_d[3 * k + 2] + so[r][3 * h + 2];
                if (water) {
                    for (int jx = j; jx < j + v.nsi[0]; ++jx) {
                        const double xd = x - v.rsx[jx], yd = y - v.rsy[jx], zd = z - v.rsz[jx];
                        e += v.q[jx] * ewald_g(alfa2 * (xd * xd + yd * yd + zd * zd), v.etab, v.spii);
                    }
                } else {
                    e += v.q[j] * ewald_g(alfa2 * (x * x + y * y + z * z), v.etab, v.spii);
                }
            }
            if (b + lane >= total) e = 0.0;
            const int r1 = min(b + 31, total - 1) / cnt;
            for (int rr = b / cnt; rr <= r1; ++rr) {
                const double sum = warp_sum(r == rr ? e : 0.0);
                if (lane == 0) atomicAdd(&su[rr], sum);
            }
        }
    };
    if (nw) sweep(0, nw, true);
    if (no) sweep(kWNb - no, no, false);
    __syncthreads();
    if (t < nr) {
        double u0 = 0.0;
        for (int k = 0; k < kRT / 32; ++k) u0 += red[k];
        s.u[(size_t)ins * kMaxRot + t] = u0 + fq * w.q1 * su[t];
    }
    if (t == 0) {
        s.off[ins] = s_off;
        w.res[ins] = make_double2(0.0, 0.0);
    }
}

__global__ void k_widom_sum(View v, WArgs w, W64 s, int nins) {
    const int ins = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, r = threadIdx.x & 31;
    if (ins >= nins || w.res[ins].y != 0.0) return;
    double e = 0.0;
    if (r < (int)w.pos[ins].w) {
        const double* rr = w.rot + ((size_t)ins * kMaxRot + r) * 6;
        const double* phi = s.phi + s.off[ins];
        const double oz = w.pos[ins].z;
        const double u_rec = 0.5 * (w.q0 * phi[0] + w.q1 * (phi[1 + 2 * r] + phi[2 + 2 * r]));
        double u = s.u[(size_t)ins * kMaxRot + r] + u_rec;
        u -= w.crf * (w.q0 * oz + w.q1 * rr[2] + w.q1 * rr[5]);
        u += wall_tail(v, w.lr, oz);
        e = exp(-w.beta * u);
    }
    e = warp_sum(e);
    if (r == 0) w.res[ins].x = e;
}

// Mixed form: the orientation loop (real-space erfc terms and the reciprocal term) in FP32 with FP64
// sums per block; the O scan, the wall tail and exp stay FP64.
__global__ void __launch_bounds__(kWT) k_widom(View v, WArgs w) {
    extern __shared__ __align__(16) unsigned char sm[];
    int* nb_j = reinterpret_cast<int*>(sm);
    double* nb_d = reinterpret_cast<double*>(sm + sizeof(int) * kWNb);           // [kWNb][3]
    float2* elf = reinterpret_cast<float2*>(sm + sizeof(int) * kWNb + sizeof(double) * 3 * kWNb);  // [3][nl]
    const int nl = w.KL + 1, nm = 2 * w.KM + 1, nn = 2 * w.KN + 1;
    float2* emf = elf + 3 * nl;        // [3][nm], index m + KM
    float2* enf = emf + 3 * nm;        // [3][nn], index n + KN
    __shared__ double red[kWT / 32];
    __shared__ int s_nnb, s_flag;
    const int ins = blockIdx.x, t = threadIdx.x;
    const double4 o = w.pos[ins];
    const double ox = o.x, oy = o.y, oz = o.z;
    if (t == 0) {
        s_nnb = 0;
        s_flag = 0;
    }
    __syncthreads();
    // ---- the probe's O against every site that is not of the H type
    double ux = 0.0;
    for (int j = t; j < v.ntota; j += kWT) {
        const int jt = v.type[j];
        if (jt == 1) continue;
        const double zio = oz - v.z[j];
        if (fabs(zio) > v.rcut) continue;
        const double xio = minimg(ox - v.x[j], v.lx, v.lxi);
        const double yio = minimg(oy - v.y[j], v.ly, v.lyi);
        const double rsq = xio * xio + yio * yio + zio * zio;
        if (rsq > v.rcutsq) continue;
        if (rsq < w.rwinsmin && (jt == 0 || rsq < w.rinsmin)) {
            atomicOr(&s_flag, 1);
            continue;
        }
        const int ijt = v.ijt[jt];  // it = 1 (the water O type)
        const double rsqi = 1.0 / rsq;
        const double rij = sqrt(rsq);
        const int vk = v.vdw[ijt];
        if (vk == 1) {
            const double r6 = v.sig[ijt] * (rsqi * rsqi * rsqi);
            ux += v.eps[ijt] * r6 * (r6 - 1.0);
        } else if (vk == 2) {
            const double r6 = v.cc[ijt] * (rsqi * rsqi * rsqi);
            ux += v.aa[ijt] * exp(-rij * v.rhoi[ijt]) - r6;
        }
        ux += ewald_e(rij, v.alfa) * (v.facq * w.q0 * v.q[j] / rij);
        const int k = atomicAdd(&s_nnb, 1);
        if (k < kWNb) {
            nb_j[k] = j;
            nb_d[3 * k + 0] = xio;
            nb_d[3 * k + 1] = yio;
            nb_d[3 * k + 2] = zio;
        } else {
            atomicOr(&s_flag, 2);
        }
    }
    ux = block_sum_d(ux, red);
    __syncthreads();
    const int flag = s_flag, nnb = min(s_nnb, kWNb);
    if (flag) {
        if (t == 0) w.res[ins] = make_double2(0.0, (flag & 1) ? 1.0 : 2.0);
        return;
    }
    const double qs3[3] = {w.q0, w.q1, w.q1};
    double acc = 0.0;
    const int nr = (int)o.w;
    for (int r = 0; r < nr; ++r) {
        const double* rr = w.rot + ((size_t)ins * kMaxRot + r) * 6;
        const double sx[3] = {ox, rr[0], rr[3]}, sy[3] = {oy, rr[1], rr[4]}, sz[3] = {oz, rr[2], rr[5]};
        double ur = 0.0, uk = 0.0;
        // ---- real space in FP32: site offsets from the O, neighbour sites from the FP32
        // copy of rs and q
        const float qx3[3] = {(float)(v.facq * qs3[0]), (float)(v.facq * qs3[1]), (float)(v.facq * qs3[2])};
        float dsx[3], dsy[3], dsz[3];
#pragma unroll
        for (int ix = 0; ix < 3; ++ix) {
            dsx[ix] = (float)(sx[ix] - ox);
            dsy[ix] = (float)(sy[ix] - oy);
            dsz[ix] = (float)(sz[ix] - oz);
        }
        const float alfa = (float)v.alfa;
        float urf = 0.f;
        for (int k = t; k < nnb; k += kWT) {
            const int j = nb_j[k];
            const float xio = (float)nb_d[3 * k], yio = (float)nb_d[3 * k + 1], zio = (float)nb_d[3 * k + 2];
            const int jt = v.type[j];
            if (jt == 0) {
                const int njx = v.nsi[jt];
                for (int ix = 0; ix < 3; ++ix) {
                    const float xi = xio + dsx[ix], yi = yio + dsy[ix], zi = zio + dsz[ix];
                    for (int jx = (ix == 0 ? j + 1 : j); jx < j + njx; ++jx) {
                        const float4 qj = w.rsf[jx];
                        const float xd = xi - qj.x, yd = yi - qj.y, zd = zi - qj.z;
                        const float r2 = xd * xd + yd * yd + zd * zd;
                        const float ri = rsqrtf(r2);
                        urf += ewald_ef(r2 * ri, alfa) * (qx3[ix] * qj.w * ri);
                    }
                }
            } else {
                const float qj = w.rsf[j].w;
                for (int ix = 1; ix < 3; ++ix) {
                    const float xi = xio + dsx[ix], yi = yio + dsy[ix], zi = zio + dsz[ix];
                    const float r2 = xi * xi + yi * yi + zi * zi;
                    const float ri = rsqrtf(r2);
                    urf += ewald_ef(r2 * ri, alfa) * (qx3[ix] * qj * ri);
                }
            }
        }
        ur = (double)urf;
        if (t < 9) {
            const int s = t / 3, ax = t % 3;
            const double ang = ax == 0 ? w.pipix * sx[s] : (ax == 1 ? w.pipiy * sy[s] : w.pipiz * sz[s]);
            double cd, sd;
            sincos(ang, &sd, &cd);
            const float2 e1 = make_float2((float)cd, (float)sd);
            if (ax == 0) {
                float2* T = elf + s * nl;
                T[0] = make_float2(1.f, 0.f);
                if (w.KL >= 1) T[1] = e1;
                for (int l = 2; l <= w.KL; ++l)
                    T[l] = make_float2(T[l - 1].x * e1.x - T[l - 1].y * e1.y, T[l - 1].x * e1.y + T[l - 1].y * e1.x);
            } else {
                const int K = ax == 1 ? w.KM : w.KN;
                float2* T = (ax == 1 ? emf + s * nm : enf + s * nn) + K;
                T[0] = make_float2(1.f, 0.f);
                if (K >= 1) T[1] = e1;
                for (int l = 2; l <= K; ++l)
                    T[l] = make_float2(T[l - 1].x * e1.x - T[l - 1].y * e1.y, T[l - 1].x * e1.y + T[l - 1].y * e1.x);
                for (int l = 1; l <= K; ++l) T[-l] = make_float2(T[l].x, -T[l].y);
            }
        }
        __syncthreads();
        const float q3f[3] = {(float)qs3[0], (float)qs3[1], (float)qs3[2]};
        float ukf = 0.f;
        for (int k = t; k < w.nk; k += kWT) {
            const int3 kv = w.kvec[k];
            float xr = 0.f, xi = 0.f;
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const float2 a = elf[s * nl + kv.x], b = emf[s * nm + kv.y + w.KM], cc = enf[s * nn + kv.z + w.KN];
                const float lr_ = q3f[s] * (a.x * b.x - a.y * b.y), li_ = q3f[s] * (a.x * b.y + a.y * b.x);
                xr += lr_ * cc.x - li_ * cc.y;
                xi += lr_ * cc.y + li_ * cc.x;
            }
            const float2 q = w.qsf[k];
            ukf += 0.5f * w.akf[k] * (xr * q.x + xi * q.y);
        }
        uk = (double)ukf;
        const double u_real = block_sum_d(ur, red);
        const double u_rec = block_sum_d(uk, red);
        if (t == 0) {
            double u = u_real + ux + u_rec;
            u -= w.crf * (w.q0 * sz[0] + w.q1 * sz[1] + w.q1 * sz[2]);
            u += wall_tail(v, w.lr, oz);
            acc += exp(-w.beta * u);
        }
        __syncthreads();  // tables are rebuilt for the next orientation
    }
    if (t == 0) w.res[ins] = make_double2(acc, 0.0);
}

// Scratch of the calls: results grow on demand, the rest is sized for one chunk and taken whole or not at all, so
// that the call after one that found no memory starts over.
int widom_scratch(Ctx& c, int64_t nins) {
    const KSet& ks = c.ks;
    const View& v = c.v;
    const size_t mark = c.owned.size();
    const char* oom = "Widom insertion: out of memory";
    if (c.widom_cap < nins) {
        const int64_t cap = std::max<int64_t>(nins, 256);
        double* res = (double*)dalloc(c, sizeof(double) * 2 * cap);
        if (!res) {
            drop_owned(c, mark);
            return set_err(&c, MDG_E_CUDA, oom);
        }
        c.d_widom_res = res;
        c.widom_cap = cap;
    }
    if (c.widom_ready) return MDG_OK;
    const size_t rest = c.owned.size();
    c.d_widom_rot = (double*)dalloc(c, sizeof(double) * kIns * kMaxRot * 6);
    c.d_widom_draw = (double*)dalloc(c, sizeof(double) * kIns * kDraw);
    if (c.precision != MDG_MIXED) {
        // real-space energies, points, potentials (doubles), first points and two counts (int)
        c.d_widom_u = (double*)dalloc(c, (sizeof(double) * (kMaxRot + 4 * kPts) + sizeof(int)) * kIns + 2 * sizeof(int));
        c.d_widom_pm = (double2*)dalloc(c, 2 * sizeof(double2) * std::max(ks.nent, 1));
        c.d_widom_atoms = (float4*)dalloc(c, sizeof(float4) * std::max(v.ntota, 1));
    } else {
        const int nk = std::max(ks.nk, 1);
        c.d_widom_akf = (float*)dalloc(c, sizeof(float) * nk);
        c.d_widom_qsf = (float2*)dalloc(c, sizeof(float2) * nk);
        c.d_widom_rsf = (float4*)dalloc(c, sizeof(float4) * std::max(v.ntota, 1));
    }
    if (!c.h_widom_draw) halloc(c, &c.h_widom_draw, sizeof(double) * 2 * kIns * kDraw);
    for (cudaEvent_t& e : c.widom_read)
        if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            e = nullptr;
            c.alloc_failed = true;
        }
    if (c.alloc_failed) {
        drop_owned(c, rest);
        return set_err(&c, MDG_E_CUDA, oom);
    }
    if (c.precision == MDG_MIXED && ks.nk > 0) {
        std::vector<double> ak(ks.nk);
        std::vector<float> akf(ks.nk);
        MDG_CUDA(cudaMemcpy(ak.data(), ks.ak, sizeof(double) * ks.nk, cudaMemcpyDeviceToHost));
        for (int k = 0; k < ks.nk; ++k) akf[k] = (float)ak[k];
        MDG_CUDA(cudaMemcpy(c.d_widom_akf, akf.data(), sizeof(float) * ks.nk, cudaMemcpyHostToDevice));
    }
    c.widom_ready = true;
    return MDG_OK;
}

}  // namespace

int widom(Ctx& c, const mdg_widom_params* p, double* seed, double* pave, int64_t* inave, int64_t* done) {
    View& v = c.v;
    KSet& ks = c.ks;
    if (c.variant != MDG_SLAB) return set_err(&c, MDG_E_UNSUPPORTED, "Widom insertion: slab variant only");
    if (!p || !seed || !pave || !inave || p->ichmax < 0 || p->lchmax < 1 || !(p->lwmax > p->lwmin))
        return set_err(&c, MDG_E_ARG, "Widom insertion: bad arguments");
    if (done) *done = 0;
    const int64_t nins = p->ichmax;
    if (nins == 0) return MDG_OK;
    // measure_init (src/measure.f90:151-155): distances from the wall -> distances from the centre
    const double lwh = v.lwh;
    const double zlo = lwh - p->lwmax, zhi = lwh - p->lwmin;
    const double facbin = 1.0 / (zhi - zlo) * (double)(float)p->lchmax;
    const double chtemper = p->temper > 0.0 ? p->temper : 300.0;
    const double beta = 1000.0 / ((double)8.31441f * chtemper);
    const double M_PI_R = (double)3.1415926535898f;
    if (const int rc = widom_scratch(c, nins)) return rc;
    double dipz = 0.0;
    if (p->flags & MDG_WIDOM_EW3DC)
        MDG_CUDA(cudaMemcpy(&dipz, v.acc + 2 * v.nijt + ACC_DIPZ, sizeof(double), cudaMemcpyDeviceToHost));
    WArgs w;
    w.pos = reinterpret_cast<const double4*>(c.d_widom_draw);
    w.rot = c.d_widom_rot;
    w.kvec = ks.kvec;
    w.lr = c.d_lr;
    w.nk = ks.nk;
    w.KL = ks.klmax;
    w.KM = ks.kmmax;
    w.KN = ks.knmax;
    w.pipix = ks.pipix;
    w.pipiy = ks.pipiy;
    w.pipiz = ks.pipiz;
    w.beta = beta;
    w.rinsmin = 4.0;                        // 2.0**2
    w.rwinsmin = (double)(2.35f * 2.35f);   // 2.35**2 in default real
    const double crf0 = -2.0 * M_PI_R * v.lzi * v.lxi * v.lyi;
    w.crf = (p->flags & MDG_WIDOM_EW3DC) ? 2.0 * crf0 * v.facq * dipz : 0.0;
    w.q0 = (double)-0.8476f;
    w.q1 = (double)0.4238f;
    const size_t smem = sizeof(int) * kWNb + sizeof(double) * 3 * kWNb +
                        sizeof(float2) * 3 * (size_t)((ks.klmax + 1) + (2 * ks.kmmax + 1) + (2 * ks.knmax + 1));
    const bool mx = c.precision == MDG_MIXED;
    if (!c.widom_attr) {
        MDG_CUDA(allow_max_smem(k_widom));
        c.widom_attr = true;
    }
    w.qsf = nullptr;
    w.akf = nullptr;
    w.rsf = nullptr;
    W64 s{};
    if (mx) {
        const int np = std::max(std::max(ks.nk, v.ntota), 1);
        k_widom_prep<<<std::min((np + 255) / 256, 152 * 4), 256, 0, c.stream>>>(v, ks.s, ks.qw, c.d_widom_qsf, ks.nk,
                                                                             c.d_widom_rsf);
        w.qsf = c.d_widom_qsf;
        w.akf = c.d_widom_akf;
        w.rsf = c.d_widom_rsf;
    } else {
        s.atoms = c.d_widom_atoms;
        s.stride = (size_t)kPts * kIns;
        s.u = c.d_widom_u;
        s.xyz = s.u + (size_t)kMaxRot * kIns;
        s.phi = s.xyz + 3 * s.stride;
        s.off = reinterpret_cast<int*>(s.phi + s.stride);
        s.cnt = s.off + kIns;
        s.lx = (float)v.lx;
        s.ly = (float)v.ly;
        s.lxi = (float)v.lxi;
        s.lyi = (float)v.lyi;
        // FP32 rounding moves a squared distance r^2 by less than 4e-7 r (r + box edge)
        const double box = std::max(v.lx, std::max(v.ly, v.lz));
        s.far2 = (float)(v.rcutsq + 1e-5 * v.rcut * (v.rcut + box));
        s.near2 = (float)(std::min(w.rinsmin, v.rcutsq) - 1e-5 * 2.0 * (2.0 + box));
        MDG_CUDA(cudaMemsetAsync(s.cnt, 0, sizeof(int), c.stream));
        k_widom_atoms<<<(v.ntota + 255) / 256, 256, 0, c.stream>>>(v, s);
        recip_pot_table(c, c.d_widom_pm, c.stream);
    }
    // Chunks: while the device evaluates one the host draws the next, positions and orientations in the
    // reference's order (src/forcem.f90:1256-1377); the states that orientations are made from go to
    // the device (192 bytes per position; the H positions were 964).
    std::vector<double> seed_pos(nins), seed_rot(nins);
    std::vector<int> hn(nins), hil(nins);
    Generator g(*seed);
    for (int64_t base = 0, chunk = 0; base < nins; base += kIns, ++chunk) {
        const int n = (int)std::min<int64_t>(kIns, nins - base);
        double* hp = c.h_widom_draw + (chunk & 1) * kIns * kDraw;
        double* hs = hp + 4 * n;
        if (chunk >= 2) MDG_CUDA(cudaEventSynchronize(c.widom_read[chunk & 1]));
        for (int i = 0; i < n; ++i) {
            const int64_t ic = base + i;
            const double oxr = (g.number() - 0.5) * v.lx;
            const double oyr = (g.number() - 0.5) * v.ly;
            double ozr, sd;
            for (int guard = 0;; ++guard) {
                sd = g.state();
                ozr = ((sd * kRndScale - 0.5) * zhi * 2.0);
                if (std::fabs(ozr) > zlo) break;
                if (guard > 100000000) {
                    cudaStreamSynchronize(c.stream);
                    return set_err(&c, MDG_E_ARG, "Widom insertion: empty band");
                }
            }
            seed_pos[ic] = sd;
            const int il = (int)((std::fabs(ozr) - zlo) * facbin) + 1;
            if (il < 1 || il > p->lchmax) {
                cudaStreamSynchronize(c.stream);
                return set_err(&c, MDG_E_ARG, "Widom insertion: bin outside lchmax");
            }
            hil[ic] = il;
            hn[ic] = il > p->ilmid ? 20 : 1;
            hp[4 * i] = oxr;
            hp[4 * i + 1] = oyr;
            hp[4 * i + 2] = ozr;
            hp[4 * i + 3] = hn[ic];
            for (int ir = 0; ir < hn[ic]; ++ir) {
                double first, ri;
                do {
                    first = g.state();
                    const double a = first * kRndScale - 0.5, b = g.number() - 0.5, d = g.number() - 0.5;
                    ri = a * a + b * b + d * d;
                } while (!(ri < 0.25 && ri > (double)0.001f));
                hs[(size_t)i * kMaxRot + ir] = first;
                sd = g.state();
            }
            seed_rot[ic] = sd;
        }
        w.res = reinterpret_cast<double2*>(c.d_widom_res) + base;
        MDG_CUDA(cudaMemcpyAsync(c.d_widom_draw, hp, sizeof(double) * kDraw * n, cudaMemcpyHostToDevice, c.stream));
        MDG_CUDA(cudaEventRecord(c.widom_read[chunk & 1], c.stream));
        k_widom_rot<<<(n * kMaxRot + 127) / 128, 128, 0, c.stream>>>(w.pos, c.d_widom_draw + 4 * n, c.d_widom_rot, n);
        if (mx) {
            k_widom<<<n, kWT, smem, c.stream>>>(v, w);
        } else {
            MDG_CUDA(cudaMemsetAsync(s.cnt + 1, 0, sizeof(int), c.stream));
            k_widom_real<<<n, kRT, 0, c.stream>>>(v, w, s);
            recip_potential(c, c.d_widom_pm, s.xyz, s.stride, s.cnt + 1, kPts * n, kPts * n / 2 + 1, s.phi, c.stream);
            k_widom_sum<<<(n + 7) / 8, 256, 0, c.stream>>>(v, w, s, n);
        }
    }
    MDG_CUDA(cudaGetLastError());
    std::vector<double> res(2 * nins);
    MDG_CUDA(cudaMemcpyAsync(res.data(), c.d_widom_res, sizeof(double) * 2 * nins, cudaMemcpyDeviceToHost, c.stream));
    MDG_CUDA(cudaStreamSynchronize(c.stream));
    // the reference's accumulation: inave counts the tries of every position drawn, including the
    // one that overlaps; the first overlap ends the call unless overlaps are skipped
    int64_t n = 0;
    for (int64_t ic = 0; ic < nins; ++ic) {
        const int st = (int)res[2 * ic + 1];
        if (st == 2) return set_err(&c, MDG_E_LIST_OVERFLOW, "Widom insertion: more than 1024 sites around the probe");
        inave[hil[ic] - 1] += hn[ic];
        ++n;
        if (st == 1) {
            if (!(p->flags & MDG_WIDOM_SKIP_OVERLAP)) {
                *seed = seed_pos[ic];
                if (done) *done = n;
                return MDG_OK;
            }
            continue;
        }
        pave[hil[ic] - 1] += res[2 * ic];
    }
    *seed = seed_rot[nins - 1];
    if (done) *done = n;
    return MDG_OK;
}

}  // namespace mdg
