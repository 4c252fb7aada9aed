// hqt_zstage.cuh -- one RK stage of the radial (Chebyshev) column work in a
// single kernel: F1, F3, F4 and the boundary row of F2
// (scripts/simulation/tevol_driven_cluster.m:72-76), the radial integration
// func_Lzr (:63-65), k = h*F with k(:,:,nz) = 0 and the RK4 bookkeeping
// (:120-124,128).
//
// Every radial operator is an Nz x Nz matrix applied to all columns, run on the
// FP64 tensor cores (mma.sync m8n8k4 f64).  A block of four warps takes tiles of
// 16 adjacent (x, y) columns; a warp owns 4 of them, and the mma's 8 columns are
// (column, part) pairs: the real and imaginary parts of Psi, or the x and y
// components of the gauge field.  The operators are A fragments in registers for
// the life of the (persistent) block, the column data is the B operand.
//
// Lz = 2 chebdif(nz) is centro-antisymmetric (Lz(n'-i, n'-j) = -Lz(i, j), n' =
// nz - 1), so a product is two of half the size: with e_j = x_j + x_{n'-j} and
// o_j = x_j - x_{n'-j}, P = Le e and Q = Lo o (rows i <= n'/2), the results are
// y_i = P_i + Q_i and y_{n'-i} = Q_i - P_i.  A product of 21 levels takes 12 mma
// instead of 18, of 33 levels 22 instead of 45, and the fragments of both
// operators fit in registers at 33 levels too (108 instead of 180).
//
// e and o mix the two ends of a column, where the entries of Lz are about 2/3 n'^2: a
// field that vanishes at the boundary would pick up there the rounding of its
// horizon values (F1 of a nearly static state 3 to 5 times less exact than by the
// full product).  So the line through the end values is taken out first, x = w +
// x_{n'} + z d with d = x_0 - x_{n'}: w vanishes at both ends, Lz x = Lz w + d, and
//   e_j = (x_j - x_0) + (x_{n'-j} - x_{n'}),
//   o_j = (x_j - x_0) - (x_{n'-j} - x_{n'}) + 2 (1 - z_j) d.
// e_0 = o_0 = 0, so the slot j = 0 of o carries d, with ones in Lo.
//
// A tile's fields come in by TMA, one box per field, in two groups with an mbarrier
// each: the main inputs, and the RK state and accumulator.  A group's region is
// refilled with the next tile's as soon as every warp is done with it.  Fields
// whose level rows are not a multiple of 16 bytes apart (a real field or FP32
// pairs with an odd nx*ny) come as two or four groups of levels (ZsSplit).  (By
// cp.async of all threads, 4 or 8 bytes each, a launch took 1044 us at 1001x1001x20,
// now 924, and of 301x301x21 in mixed precision 123, now 109.)
//
// What bounds it: the copies.  TMA takes about 8.5 cycles per box row whatever its
// width up to 256 bytes, so 8-column tiles (128-byte rows) loaded 4.5 TB/s however
// many were in flight, and dropping all products changed nothing; 16 columns load
// 5.8-6.2 TB/s (loads alone, 13 FP64 pair fields, 512x512x25 .. 1001x1001x20).  A
// row is one column wider than the tile (272 bytes): rows then start 16 bytes
// further into the banks each, which a 256-byte row or TMA's 128-byte swizzle
// (128-byte rows only) could not give.
//
// Fragment layouts (g = lane/4, q = lane%4): A a0 = L[row g][4s+q]; B b0 =
// V[level 4s+q][column of g/2].part(g%2); C c_i = out[row g][column of q].part(i).
// Row g of tile m stands for level 8m + zs_row(g), column index k of a warp for
// column zs_col(k): with them the mma operand reads (4 levels x 4 columns), the
// pointwise reads (levels 2 apart) and the stores (whole 32-byte sectors) are
// all free of bank conflicts and half sectors.
//
// Phases of a tile (MODE 1..4 = RK stage, MODE 0 = right-hand side only); the
// gauge field's and Psi's products run side by side, which doubles the independent
// mma chains of a warp:
//   1  g = d A_t + f Lz A, dp = Lz Psi
//   2  S = 1/2 Lz g -+ 1/2 d B + Im(conj(Psi) d Psi) - A |Psi|^2 (:74-75), S1 of
//      d2 = Lz dp (:72-73), Lz(nz,:) div A; then the next tile's main inputs
//   3  F3, F4 = Lzr(S), F1 = Lzr(S1), RK updates; then the next tile's state
#pragma once
#include <cuda.h>

#include <type_traits>

#include "hqt_args.h"
#include "hqt_dev.cuh"
#include "hqt_zdims.h"

namespace hqt {

constexpr int kZsThreads = 128;

// d += a * b on one 8x8x4 FP64 tensor-core tile
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}
// Sum over the 8 lane groups g = lane/4 (same column q): after the shuffles
// every lane holds the total of its column.
__device__ __forceinline__ double zf_colsum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    return v;
}

__device__ __forceinline__ int zs_col(int warp, int k) { return ((k & 1) << 2) + (k >> 1) + 2 * (warp & 1) + 8 * (warp >> 1); }

// Shared-memory layout of a block.
template <typename TD, int NZP, int MODE> struct ZsLay {
    static constexpr int up(int b) { return (b + 127) / 128 * 128; }
    static constexpr int rc = up(NZP * kZsRow);
    // (a group of levels each, ZsSplit)
    static constexpr int rd = up(NZP * zs_row_td<TD>()) + (sizeof(TD) == 8 ? 0 : 128);
    static constexpr int rr = up(NZP * zs_row_r<TD>()) + (sizeof(TD) == 8 ? 128 : 384);
    // state and accumulator staged (DIRECT: read from global memory where they are
    // used; stage 1: the state is the stage input, copied aside for the update)
    static constexpr bool k = MODE >= 2 && !ZsDims<NZP>::direct;
    static constexpr bool z = k || (MODE == 1 && !ZsDims<NZP>::direct);
    static constexpr int oPS = 0, oAXY = rc, oATD = 2 * rc, oDX = 3 * rc, oDY = oDX + rd;
    static constexpr int oDT = oDY + rd, oB = oDT + rd, oXX = oB + rd, oYY = oXX + rd;
    static constexpr int oDIV = oYY + rd, oZA = oDIV + rr, oZP = oZA + (z ? rc : 0);
    static constexpr int oKA = oZP + (z ? rc : 0), oKP = oKA + (k ? rc : 0);
    static constexpr int oVA = oKP + (k ? rc : 0), rv = up(ZsDims<NZP>::VR * kZsRow);
    static constexpr int oVB = oVA + rv, oTAB = oVB + rv;  // z, f, Lz(nz,:), line
    static constexpr int oROW = oTAB + up(ZsDims<NZP>::ntab * 8);  // rows of div A
    static constexpr int oBAR = oROW + up(NZP * 4);
    static constexpr int bytes = oBAR + 64 + 128;  // + alignment of the base
};

// ---- mbarriers and copies ---------------------------------------------------
__device__ __forceinline__ void zs_bar_init(unsigned bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void zs_expect(unsigned bar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// Waits for a phase, `polls` times about a microsecond; false if it did not complete.
__device__ __forceinline__ bool zs_wait(unsigned bar, int parity, int polls) {
    unsigned ok = 0;
    for (int i = 0; i < polls && !ok; ++i)
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"(1000)
            : "memory");
    return ok;
}
// After a wait in vain (`lost`) a thread waits no more and counts no further phases, and
// the thread that issues the block's copies issues none: the block runs to its end on
// whatever its buffers hold.  There that thread waits once more for the phases that were
// in flight (zs_drain), which must not outlive the block, and the fault flag goes up.
// (To wait for them, or to leave, where the first wait gave up cost 1-2% of a launch at
// 301x301x21: a call or a loop in the tile's code, a barrier with a reduction.)
__device__ __forceinline__ void zs_drain(unsigned bar, int parity) {
    zs_wait(bar, parity, kZsPolls);
}
// Ahead of a barrier behind which a region is refilled: this thread's reads of it (and
// writes, of a copy set aside) come before the refill, which another proxy writes.  A
// value read before the barrier has to be used before it too: loads are only ordered by
// their use.
__device__ __forceinline__ void zs_release() {
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
// box of a tile's columns x nz levels at element x of a field's level rows
__device__ __forceinline__ void zs_tma(unsigned dst, const CUtensorMap *map, int x, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, "
        "{%2, %3}], [%4];\n" ::"r"(dst),
        "l"(map), "r"(x), "r"(0), "r"(bar)
        : "memory");
}
// Element (level, column) of the FP64 pair field at byte OFF; (row offset, column) of a
// field of TD pairs or real TD.
template <int OFF> __device__ __forceinline__ double2 &zs_at(unsigned char *sm, int l, int c) {
    return *reinterpret_cast<double2 *>(sm + OFF + l * kZsRow + c * 16);
}
template <int OFF, typename TD>
__device__ __forceinline__ C2<TD> zs_pair(unsigned char *sm, int row, int c) {
    return *reinterpret_cast<const C2<TD> *>(sm + OFF + row + c * (int)sizeof(C2<TD>));
}
template <int OFF, typename TD>
__device__ __forceinline__ double zs_real(unsigned char *sm, int row, int c) {
    return double(*reinterpret_cast<const TD *>(sm + OFF + row + c * (int)sizeof(TD)));
}

// The operators as A fragments (the context's tables, one value a lane and
// fragment) and their products with the four columns of a warp.
template <int NZP> struct ZsOps {
    using D = ZsDims<NZP>;
    static constexpr int MH = D::MH, MP = D::MP, KE = D::KE, KO = D::KO, M1 = D::M1, K1 = D::K1;
    double Fe[MP][KE], Fo[MH][KO], F1[M1][K1];
    int q, cop, part, n1;

    __device__ __forceinline__ ZsOps(const double *frag, int lane, int warp, int nz)
        : q(lane & 3), cop(zs_col(warp, lane >> 3)), part(((lane >> 2) & 1) * 8), n1(nz - 1) {
        const double *f = frag + lane;
#pragma unroll
        for (int m = 0; m < MP; ++m)
#pragma unroll
            for (int s = 0; s < KE; ++s, f += 32) Fe[m][s] = __ldg(f);
#pragma unroll
        for (int m = 0; m < MH; ++m)
#pragma unroll
            for (int s = 0; s < KO; ++s, f += 32) Fo[m][s] = __ldg(f);
#pragma unroll
        for (int m = 0; m < M1; ++m)
#pragma unroll
            for (int s = 0; s < K1; ++s, f += 32) F1[m][s] = __ldg(f);
    }
    // operand (level j) of the FP64 pair field at OFF
    template <int OFF> __device__ __forceinline__ double operand(unsigned char *sm, int j) const {
        return *reinterpret_cast<const double *>(
            reinterpret_cast<unsigned char *>(&zs_at<OFF>(sm, j, cop)) + part);
    }
    // (yA, yB)[m] = Lz x at levels i = 8m + zs_row(g) and n1 - i for the operands
    // x(level) (into y) and v(level) (into w): two sets of independent mma chains;
    // line[j]: factor of the end values' difference in o_j
    template <typename X, typename V>
    __device__ __forceinline__ void lz2(X x, V v, const double *line, double (&yA)[MH][2],
                                        double (&yB)[MH][2], double (&wA)[MH][2],
                                        double (&wB)[MH][2]) const {
#pragma unroll
        for (int m = 0; m < MH; ++m)
            yA[m][0] = yA[m][1] = yB[m][0] = yB[m][1] = wA[m][0] = wA[m][1] = wB[m][0] =
                wB[m][1] = 0.0;
        const double x0 = x(0), xn = x(n1), dx = x0 - xn, v0 = v(0), vn = v(n1), dv = v0 - vn;
#pragma unroll
        for (int s = 0; s < KE; ++s) {
            const int j = min(4 * s + q, n1), jm = max(n1 - 4 * s - q, 0);
            const double x1 = x(j) - x0, x2 = x(jm) - xn, v1 = v(j) - v0, v2 = v(jm) - vn;
            const double t = line[4 * s + q];
            const double e = x1 + x2, o = fma(t, dx, x1 - x2);
            const double ve = v1 + v2, vo = fma(t, dv, v1 - v2);
#pragma unroll
            for (int m = 0; m < MP; ++m) {
                dmma(yA[m][0], yA[m][1], Fe[m][s], e);
                dmma(wA[m][0], wA[m][1], Fe[m][s], ve);
            }
            if (s < KO) {
#pragma unroll
                for (int m = 0; m < MH; ++m) {
                    dmma(yB[m][0], yB[m][1], Fo[m][s < KO ? s : 0], o);
                    dmma(wB[m][0], wB[m][1], Fo[m][s < KO ? s : 0], vo);
                }
            }
        }
        merge(yA, yB);
        merge(wA, wB);
    }
    // ... for one
    template <typename X>
    __device__ __forceinline__ void lz(X x, const double *line, double (&yA)[MH][2],
                                       double (&yB)[MH][2]) const {
#pragma unroll
        for (int m = 0; m < MH; ++m) yA[m][0] = yA[m][1] = yB[m][0] = yB[m][1] = 0.0;
        const double x0 = x(0), xn = x(n1), dx = x0 - xn;
#pragma unroll
        for (int s = 0; s < KE; ++s) {
            const int j = min(4 * s + q, n1), jm = max(n1 - 4 * s - q, 0);
            const double x1 = x(j) - x0, x2 = x(jm) - xn;
            const double e = x1 + x2, o = fma(line[4 * s + q], dx, x1 - x2);
#pragma unroll
            for (int m = 0; m < MP; ++m) dmma(yA[m][0], yA[m][1], Fe[m][s], e);
            if (s < KO) {
#pragma unroll
                for (int m = 0; m < MH; ++m) dmma(yB[m][0], yB[m][1], Fo[m][s < KO ? s : 0], o);
            }
        }
        merge(yA, yB);
    }
    // P in yA, Q in yB: y_i = P + Q, y_{n1-i} = Q - P
    __device__ __forceinline__ static void merge(double (&yA)[MH][2], double (&yB)[MH][2]) {
#pragma unroll
        for (int m = 0; m < MH; ++m)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const double p = yA[m][i], r = yB[m][i];
                yA[m][i] = r + p;
                yB[m][i] = r - p;
            }
    }
    // F[m] = Lz1 x at levels 8m + zs_row(g) (zero at nz - 1 and past it)
    template <int OFF>
    __device__ __forceinline__ void lz1(unsigned char *sm, double (&F)[M1][2]) const {
#pragma unroll
        for (int m = 0; m < M1; ++m) F[m][0] = F[m][1] = 0.0;
#pragma unroll
        for (int s = 0; s < K1; ++s) {
            const double b = operand<OFF>(sm, 4 * s + q);
#pragma unroll
            for (int m = 0; m < M1; ++m) dmma(F[m][0], F[m][1], F1[m][s], b);
        }
    }
    template <int OFF, int OFF2>
    __device__ __forceinline__ void lz1_2(unsigned char *sm, double (&F)[M1][2],
                                          double (&G)[M1][2]) const {
#pragma unroll
        for (int m = 0; m < M1; ++m) F[m][0] = F[m][1] = G[m][0] = G[m][1] = 0.0;
#pragma unroll
        for (int s = 0; s < K1; ++s) {
            const double b = operand<OFF>(sm, 4 * s + q), c = operand<OFF2>(sm, 4 * s + q);
#pragma unroll
            for (int m = 0; m < M1; ++m) {
                dmma(F[m][0], F[m][1], F1[m][s], b);
                dmma(G[m][0], G[m][1], F1[m][s], c);
            }
        }
    }
    // f(m, level, F) for every level of this lane's rows of Lz1, and for the
    // boundary level (F = 0, m = M1) where it lies past them
    template <typename Fn>
    __device__ __forceinline__ void rows(const double (&F)[M1][2], int g, Fn f) const {
#pragma unroll
        for (int m = 0; m < M1; ++m) {
            const int i = 8 * m + zs_row(g);
            if (i <= n1) f(m, i, F[m][0], F[m][1]);
        }
        if (n1 >= 8 * M1 && g == 0) f(M1, n1, 0.0, 0.0);
    }
};

template <typename TD, int NZP, int MODE>
__global__ void __launch_bounds__(kZsThreads, ZsDims<NZP>::min_blocks)
    k_zstage(const __grid_constant__ ZStageArgs<TD> a) {
    using Lay = ZsLay<TD, NZP, MODE>;
    using D = ZsDims<NZP>;
    using PD = C2<TD>;
    constexpr int MH = D::MH, M1 = D::M1;
    constexpr bool kK = Lay::k, kDirect = MODE >= 1 && D::direct;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int nz = a.nz, n1 = nz - 1, h = (nz + 1) / 2;
    const long long P = a.plane;
    unsigned char *sm = g_smem + ((128 - ((unsigned)__cvta_generic_to_shared(g_smem) & 127)) & 127);
    const unsigned sb = (unsigned)__cvta_generic_to_shared(sm);
    const unsigned barM = sb + Lay::oBAR, barZ = barM + 8;
    double *tab = reinterpret_cast<double *>(sm + Lay::oTAB);
    int *rowr = reinterpret_cast<int *>(sm + Lay::oROW);
    const ZsSplit spair(nz, P * (long long)sizeof(PD), zs_row_td<TD>());
    const ZsSplit sreal(nz, P * (long long)sizeof(TD), zs_row_r<TD>());
    const int odd = spair.n > 1 ? spair.start(1) + spair.shift(1) : 0;
    // row of level i in a field of TD pairs
    auto rowp = [&](int i) {
        return sizeof(TD) == 8 ? i * kZsRow
                               : (i >> spair.lg) * zs_row_td<TD>() + (i & spair.lg) * odd;
    };
    const bool leader = threadIdx.x == 0;  // issues the copies
    // z, f = 1 - z^3, Lz(nz,:) and the line's factors; V rows past nz are zero in every product
    for (int i = threadIdx.x; i < D::ntab; i += kZsThreads) tab[i] = __ldg(a.ztab + i);
    for (int i = threadIdx.x; i < nz; i += kZsThreads) rowr[i] = sreal.at(i);
    for (int i = threadIdx.x; i < 2 * Lay::rv / 16; i += kZsThreads)
        reinterpret_cast<double2 *>(sm + Lay::oVA)[i] = make_double2(0.0, 0.0);
    if (threadIdx.x == 0) {
        zs_bar_init(barM, 1);  // the leader's expected bytes
        zs_bar_init(barZ, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    pdl_wait();

    // main inputs; state and accumulator.  All by the leader.
    const int bc = nz * kZsRow;
    auto load_split = [&](int off, const CUtensorMap *map, const ZsSplit &sp, int x) {
        for (int ph = 0; ph < sp.n && ph < nz; ++ph) zs_tma(sb + off + sp.start(ph), map + ph, x, barM);
    };
    auto load_M = [&](long long s0) {
        if (!leader) return;
        const int x = (int)(2 * s0);
        zs_expect(barM, 3 * bc + nz * (6 * zs_row_td<TD>() + zs_row_r<TD>()));
        zs_tma(sb + Lay::oPS, &a.mPS, x, barM);
        zs_tma(sb + Lay::oAXY, &a.mAXY, x, barM);
        zs_tma(sb + Lay::oATD, &a.mATD, x, barM);
        load_split(Lay::oDX, a.mDX, spair, x);
        load_split(Lay::oDY, a.mDY, spair, x);
        load_split(Lay::oDT, a.mDT, spair, x);
        load_split(Lay::oB, a.mB, spair, x);
        load_split(Lay::oXX, a.mXX, spair, x);
        load_split(Lay::oYY, a.mYY, spair, x);
        load_split(Lay::oDIV, a.mDIV, sreal, (int)s0);
    };
    auto load_Z = [&](long long s0) {
        if (kK && leader) {
            zs_expect(barZ, 4 * bc);
            zs_tma(sb + Lay::oZA, &a.mZA, (int)(2 * s0), barZ);
            zs_tma(sb + Lay::oKA, &a.mKA, (int)(2 * s0), barZ);
            zs_tma(sb + Lay::oZP, &a.mZP, (int)(2 * s0), barZ);
            zs_tma(sb + Lay::oKP, &a.mKP, (int)(2 * s0), barZ);
        }
    };

    const int col = zs_col(warp, q);
    const int gr = zs_row(g);
    const ZsOps<NZP> ops(a.frag, lane, warp, nz);
    const long long ntiles = (P + kZsCols - 1) / kZsCols;
    int lost = 0;  // 1: waited in vain for main inputs; 2, 3: for the state, with and
                   // without the next tile's main inputs in flight
    if ((long long)blockIdx.x < ntiles) {
        load_M((long long)blockIdx.x * kZsCols);
        load_Z((long long)blockIdx.x * kZsCols);
    }
    int parity = 0;
#pragma unroll 1
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, parity ^= !lost) {
        const long long site = tile * kZsCols + col;  // of this lane's results
        const bool more = tile + gridDim.x < ntiles;
        const long long next = (tile + gridDim.x) * kZsCols;
        // state and accumulator at this lane's rows of Lz1 (DIRECT), requested
        // ahead of a product
        auto state = [&](const double2 *zsrc, const double2 *ksrc, double2 (&zd)[M1 + 1],
                         double2 (&kd)[M1 + 1]) {
#pragma unroll
            for (int m = 0; m <= M1; ++m) {
                const int i = m < M1 ? 8 * m + gr : n1;
                if (site < P && (m < M1 ? i <= n1 : n1 >= 8 * M1 && g == 0)) {
                    zd[m] = zsrc[(long long)i * P + site];
                    if (MODE >= 2) kd[m] = ksrc[(long long)i * P + site];
                }
            }
        };
        if (!lost && !zs_wait(barM, parity, a.polls)) lost = 1;

        // ---- g = d A_t + f Lz A -> VA, dp = Lz Psi -> VB ---------------------
        double dA[MH][2], dB[MH][2];  // dp
        {
            double yA[MH][2], yB[MH][2];
            ops.lz2([&](int j) { return ops.template operand<Lay::oAXY>(sm, j); },
                    [&](int j) { return ops.template operand<Lay::oPS>(sm, j); }, tab + 3 * NZP,
                    yA, yB, dA, dB);
            auto put = [&](int i, const double (&y)[2], const double (&d)[2]) {
                const PD dt = zs_pair<Lay::oDT, TD>(sm, rowp(i), col);
                const double f = tab[NZP + i];
                zs_at<Lay::oVA>(sm, i, col) =
                    make_double2(double(dt.x) + f * y[0], double(dt.y) + f * y[1]);
                zs_at<Lay::oVB>(sm, i, col) = make_double2(d[0], d[1]);
            };
#pragma unroll
            for (int m = 0; m < MH; ++m) {
                const int i = 8 * m + gr;
                if (i < h) {
                    put(i, yA[m], dA[m]);
                    if (n1 - i != i) put(n1 - i, yB[m], dB[m]);
                }
            }
        }
        __syncwarp();
        // ---- S of Lz g -> VA, S1 of d2 = Lz dp -> VB, boundary row of F2 ------
        double kb = 0.0;  // Lz(nz,:) div A of the column
        {
            double yA[MH][2], yB[MH][2], eA[MH][2], eB[MH][2];
            ops.lz2([&](int j) { return ops.template operand<Lay::oVA>(sm, j); },
                    [&](int j) { return ops.template operand<Lay::oVB>(sm, j); }, tab + 3 * NZP,
                    yA, yB, eA, eB);
            __syncwarp();  // VA and VB are read: the sources overwrite them
            auto put = [&](int i, const double (&y)[2], const double (&d1)[2],
                           const double (&d2)[2]) {
                const double2 ps = zs_at<Lay::oPS>(sm, i, col), av = zs_at<Lay::oAXY>(sm, i, col);
                const int rp = rowp(i);
                const PD dx = zs_pair<Lay::oDX, TD>(sm, rp, col), dy = zs_pair<Lay::oDY, TD>(sm, rp, col);
                const double dxr = double(dx.x), dxi = double(dx.y), dyr = double(dy.x),
                             dyi = double(dy.y);
                const bool in = i < n1;
                {  // S = 1/2 Lz g -+ 1/2 d B + Im(conj(Psi) d Psi) - A |Psi|^2
                    const PD bf = zs_pair<Lay::oB, TD>(sm, rp, col);
                    const double p2 = ps.x * ps.x + ps.y * ps.y;
                    const double vx = 0.5 * y[0] + 0.5 * -double(bf.x) +
                                      (ps.x * dxi - ps.y * dxr) - av.x * p2;
                    const double vy = 0.5 * y[1] + 0.5 * double(bf.y) +
                                      (ps.x * dyi - ps.y * dyr) - av.y * p2;
                    zs_at<Lay::oVA>(sm, i, col) = make_double2(in ? vx : 0.0, in ? vy : 0.0);
                }
                const double2 atd = zs_at<Lay::oATD>(sm, i, col);
                const PD lxx = zs_pair<Lay::oXX, TD>(sm, rp, col), lyy = zs_pair<Lay::oYY, TD>(sm, rp, col);
                const double lpx = double(lxx.x) + double(lyy.x), lpy = double(lxx.y) + double(lyy.y);
                const double dv = zs_real<Lay::oDIV, TD>(sm, rowr[i], col);
                kb = fma(tab[2 * NZP + i], dv, kb);
                const double z = tab[i], f = tab[NZP + i], hh = 0.5;
                const double a2 = av.x * av.x + av.y * av.y;
                const double u = av.x * dxr + av.y * dyr;
                const double w = av.x * dxi + av.y * dyi;
                const double s0 = -atd.x * d1[1] - hh * atd.y * ps.y + hh * f * d2[0] -
                                  1.5 * z * z * d1[0] - hh * z * ps.x - hh * a2 * ps.x + hh * lpx +
                                  hh * dv * ps.y + w;
                const double s1 = atd.x * d1[0] + hh * atd.y * ps.x + hh * f * d2[1] -
                                  1.5 * z * z * d1[1] - hh * z * ps.y - hh * a2 * ps.y + hh * lpy -
                                  hh * dv * ps.x - u;
                zs_at<Lay::oVB>(sm, i, col) = make_double2(in ? s0 : 0.0, in ? s1 : 0.0);
                // stage 1: the state is the stage input, copied aside for the update,
                // which comes after its region refills.  (Held in registers it was
                // read behind the barrier, as the next tile's values: a load need
                // not be done at a barrier that none of its results has to pass.)
                if (MODE == 1 && !kDirect) {
                    zs_at<Lay::oZA>(sm, i, col) = av;
                    zs_at<Lay::oZP>(sm, i, col) = ps;
                }
            };
#pragma unroll
            for (int m = 0; m < MH; ++m) {
                const int i = 8 * m + gr;
                if (i < h) {
                    put(i, yA[m], dA[m], eA[m]);
                    if (n1 - i != i) put(n1 - i, yB[m], dB[m], eB[m]);
                }
            }
        }
        kb = zf_colsum(kb);
        zs_release();
        __syncthreads();  // every warp is done with the main inputs
        if (more && !lost) load_M(next);

        // ---- F3, F4 = Lzr(S), F1 = Lzr(S1) and the RK updates ------------------
        auto update_A = [&](int i, double fx, double fy, double2 z, double2 K) {
            if (site >= P) return;
            const long long gi = (long long)i * P + site;
            if (MODE == 0) {
                a.f3[gi] = fx;
                a.f4[gi] = fy;
                return;
            }
            const double kx = a.h * fx, ky = a.h * fy;
            if (MODE == 4) {
                a.wA[gi] = make_double2(z.x + (1.0 / 6.0) * (K.x + kx),
                                        z.y + (1.0 / 6.0) * (K.y + ky));
                return;
            }
            a.kA[gi] = MODE == 1 ? make_double2(kx, ky) : make_double2(K.x + 2 * kx, K.y + 2 * ky);
            const double nx = (MODE == 3) ? z.x + kx : z.x + kx / 2;
            const double ny = (MODE == 3) ? z.y + ky : z.y + ky / 2;
            a.nA[gi] = make_double2(nx, ny);
            if constexpr (!std::is_same<TD, double>::value) {
                const double mx = a.slice_mean[5 * i + 3], my = a.slice_mean[5 * i + 4];
                a.nA_d[gi] = mk2<TD>(TD(nx - mx), TD(ny - my));
            }
        };
        auto update_psi = [&](int i, double fx, double fy, double2 z, double2 K) {
            if (site >= P) return;
            const long long gi = (long long)i * P + site;
            if (MODE == 0) {
                a.f1[gi] = make_double2(fx, fy);
                return;
            }
            const double2 k = make_double2(a.h * fx, a.h * fy);
            if (MODE == 4) {
                const double s = 1.0 / 6.0;
                a.wpsi[gi] = make_double2(z.x + s * (K.x + k.x), z.y + s * (K.y + k.y));
                return;
            }
            a.kpsi[gi] = MODE == 1 ? k : make_double2(K.x + 2 * k.x, K.y + 2 * k.y);
            const double2 nv = (MODE == 3) ? make_double2(z.x + k.x, z.y + k.y)
                                           : make_double2(z.x + k.x / 2, z.y + k.y / 2);
            a.npsi[gi] = nv;
            if constexpr (!std::is_same<TD, double>::value) {
                const double mr = a.slice_mean[5 * i], mi = a.slice_mean[5 * i + 1];
                a.npsi_d[gi] = mk2<TD>(TD(nv.x - mr), TD(nv.y - mi));
            }
        };
        const double2 none = make_double2(0.0, 0.0);
        if constexpr (kDirect) {
            double F[M1][2];
            double2 zd[M1 + 1], kd[M1 + 1];
            state(a.zA, a.kA, zd, kd);
            ops.template lz1<Lay::oVA>(sm, F);
            ops.rows(F, g, [&](int m, int i, double fx, double fy) {
                update_A(i, fx, fy, zd[m], MODE >= 2 ? kd[m] : none);
            });
            state(a.zpsi, a.kpsi, zd, kd);
            ops.template lz1<Lay::oVB>(sm, F);
            ops.rows(F, g, [&](int m, int i, double fx, double fy) {
                update_psi(i, fx, fy, zd[m], MODE >= 2 ? kd[m] : none);
            });
        } else {
            double F[M1][2], G[M1][2];
            ops.template lz1_2<Lay::oVA, Lay::oVB>(sm, F, G);
            if (kK && !lost && !zs_wait(barZ, parity, a.polls)) lost = more ? 2 : 3;
            ops.rows(F, g, [&](int, int i, double fx, double fy) {
                update_A(i, fx, fy, MODE ? zs_at<Lay::oZA>(sm, i, col) : none,
                         kK ? zs_at<Lay::oKA>(sm, i, col) : none);
            });
            ops.rows(G, g, [&](int, int i, double fx, double fy) {
                update_psi(i, fx, fy, MODE ? zs_at<Lay::oZP>(sm, i, col) : none,
                           kK ? zs_at<Lay::oKP>(sm, i, col) : none);
            });
        }
        if (g == 0 && site < P) {
            if (MODE == 0) {
                a.f2b[site] = kb;
            } else {
                const double k = a.h * kb;
                if (MODE == 1)
                    a.krho[site] = k;
                else if (MODE == 2 || MODE == 3)
                    a.krho[site] = a.krho[site] + 2 * k;
                else  // rhoi = rhoi - k2(:,:,nz), k2 = (1/6)(k21+2k22+2k23+k24)
                    a.wrho[site] = a.zrho[site] - (1.0 / 6.0) * (a.krho[site] + k);
            }
        }
        if (kK) zs_release();
        __syncthreads();  // every warp is done with the state (and VA, VB)
        if (more && !lost) load_Z(next);
    }
    if (lost) {
        if (leader && lost != 3) zs_drain(barM, lost == 1 ? parity : parity ^ 1);
        if (leader && kK) zs_drain(barZ, parity);
        *a.fault = 1;
    }
}

}  // namespace hqt
