// lr_tail.cuh - the analytic long-range tail of the walls, for one system (pair.cu) or the replicas of a batch
// (integrate.cu): block bid of nblk blocks of kLrNT threads.
#pragma once

#include "common.cuh"
#include "ctx.h"

namespace mdg {

// Wall long-range tail, src/forcem.f90:509-543.  lr: [9][nit] tables.  Small blocks: the
// per-atom FP64 work is spread over as many SMs as the atom count allows.
constexpr int kLrNT = 64;
__device__ __forceinline__ void lr_tail_block(const View& v, const double* lr, int bid, int nblk) {
    double ulr = 0.0, fw[2] = {0.0, 0.0};
    const int nit = v.nit;
    for (int i = bid * kLrNT + threadIdx.x; i < v.nmove; i += nblk * kLrNT) {
        const int it = v.type[i];
        if (fabs(v.q[i]) < F32D(0.7)) continue;
        double fz = 0.0;
        for (int j = -1; j <= 1; j += 2) {
            double aux = 0.0;
            const double sgn = (double)j;
            const double dw = v.lwh - sgn * v.z[i];
            if (dw < v.rcut) {
                aux = aux + sgn * lr[1 * nit + it];
                ulr += lr[8 * nit + it];
            } else {
                aux = aux + sgn * lr[0 * nit + it];
                ulr += lr[7 * nit + it];
                const double dwa = 1.0 / (dw * dw);
                const double dwa2 = dwa * dwa;
                aux = aux + sgn * (lr[2 * nit + it] * (dwa2 * dwa2 * dwa) - lr[3 * nit + it] * dwa2);
                const double dw3 = dw * dw * dw;
                ulr += (lr[2 * nit + it] / (9.0 * (dw3 * dw3 * dw3)) - lr[3 * nit + it] / (3.0 * dw3));
                const double t = lr[6 * nit + it];
                const double exp2a = lr[4 * nit + it] * exp(-dw / t);
                aux = aux + sgn * ((t + dw) * exp2a - lr[5 * nit + it] * dwa2);
                ulr += (t * (2.0 * t + dw) * exp2a - lr[5 * nit + it] / (3.0 * dw3));
            }
            fz -= aux;
            if (it + 1 <= v.nltype) fw[(j + 1) / 2] += aux;
        }
        atomicAdd(&v.fz[i], fz);  // the reciprocal sum of the FP64 form may be adding too
    }
    block_atomic_sum<kLrNT>(ulr, &v.acc[2 * v.nijt + ACC_ULR]);
    block_atomic_sum<kLrNT>(fw[0], &v.acc[2 * v.nijt + ACC_FWS + 6 + 0]);
    block_atomic_sum<kLrNT>(fw[1], &v.acc[2 * v.nijt + ACC_FWS + 6 + 2]);
}

}  // namespace mdg
