// hqt_zcol.cuh -- per-step radial (Chebyshev) column kernels.
//
// One thread owns one (x, y) column of all nz radial points.  The column
// lives in registers; the Nz x Nz matrices Lz = 2*chebdif(nz,1) and
// Lz1 = inv(Lz(1:nz-1,1:nz-1)) (scripts/simulation/tevol_driven_cluster.m:49,52)
// are kernel parameters, i.e. constant-bank operands of the fused
// multiply-adds, so the contractions need no loads for the matrix.  The
// compile-time column length NZP >= nz is zero-padded: padded rows and
// columns of Lz and Lz1 are zero, so the first nz outputs are exactly those
// of the nz-point operators.
//
// k_zcol_misc computes d_z A_t and k_zcol_O O alone (set-up and diagnostics).  The
// RK stages run in k_zstage and the post-combine constraint in k_zcons,
// both on block tiles and FP64 tensor-core products (hqt_zstage.cuh, hqt_zcons.cuh).
#pragma once
#include "hqt_dev.cuh"
#include "hqt_args.h"

namespace hqt {

// d_z A_t of a given potential
template <typename T, int NZP>
__global__ void __launch_bounds__(128, 4) k_zcol_misc(ZColArgs<T> a, ZOps<T, NZP> op) {
    pdl_wait();
    const long long site = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (site >= a.plane) return;
    const int nz = a.nz;
    const long long P = a.plane;
    T v[NZP];
#pragma unroll
    for (int j = 0; j < NZP; ++j) v[j] = j < nz ? a.at[(long long)j * P + site] : T(0);
#pragma unroll
    for (int i = 0; i < NZP; ++i) {
        if (i < nz) {
            T s = T(0);
#pragma unroll
            for (int j = 0; j < NZP; ++j) s = fma(op.Lz[i][j], v[j], s);
            a.atd[(long long)i * P + site] = mk2<T>(v[i], s);
        }
    }
}

// Boundary order parameter of Psi: the last row of Lz.  Bound by the reads in flight, so
// a kernel of its own with 32 to 40 registers: as a second part of the one above, which
// takes 92 at 21 levels and 108 at 25, it took 162 us at 1024x1024x25, so 86.
template <typename T, int NZP>
__global__ void __launch_bounds__(128) k_zcol_O(ZColArgs<T> a, ZOps<T, NZP> op) {
    pdl_wait();
    const long long site = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (site >= a.plane) return;
    const int nz = a.nz;
    T orr = T(0), oi = T(0);
    const C2<T> *psi = a.psi + site;
#pragma unroll
    for (int j = 0; j < NZP; ++j, psi += a.plane) {
        if (j < nz) {
            const C2<T> p = *psi;
            orr = fma(op.lzb[j], p.x, orr);
            oi = fma(op.lzb[j], p.y, oi);
        }
    }
    a.O[site] = mk2<T>(orr, oi);
}

}  // namespace hqt
