// hqt_zfused.cuh -- the radial (Chebyshev) work after the RK combine: the
// constraint, the A_t rebuild and the boundary rows
// (scripts/simulation/tevol_driven_cluster.m:129-136).
//
// Every radial operator is an Nz x Nz matrix applied to all columns, i.e. a
// product (Nz x Nz) x (Nz x columns), run on the FP64 tensor cores
// (mma.sync m8n8k4 f64).  A block stages a tile of kZTile = 16 adjacent
// (x, y) columns (128-byte level rows) with cp.async shared by all its
// threads; each of its 4 warps owns kZCols = 4 of the columns.  The mma's 8
// columns are (column, part) pairs: the real and imaginary parts of Psi, or
// the x and y components of the gauge field, so both gauge components share
// one product.  The zero-padded Lz and Lz1 stay in registers as A fragments
// for the life of the (persistent) block; the column data is the B operand,
// read from the shared tile.  Buffers of finished phases are refilled with
// the inputs of later ones (and of the next tile) while the current phase
// computes.
//
// Fragment layouts (g = lane/4, q = lane%4): A a0 = L[8m+g][4s+q];
// B b0 = V[level 4s+q][column g/2].part(g%2); C c_i = out[level 8m+g]
// [column q].part(i).  A lane thus holds whole complex values (or both gauge
// components) of levels 8m+g of column q, where the pointwise terms are
// evaluated.  Each tile field is [level][kZTile columns] with a per-level
// XOR swizzle of the 4-column groups (zswz), so both access shapes are free
// of bank conflicts.

#pragma once
#include <type_traits>

#include "hqt_dev.cuh"
#include "hqt_args.h"

namespace hqt {

constexpr int kZCols = 4;   // columns per warp (x 2 parts = the mma's n extent)
constexpr int kZWarps = 4;  // warps per block; a block stages kZTile columns
constexpr int kZTile = kZCols * kZWarps;

// d += a * b on one 8x8x4 FP64 tensor-core tile
__device__ __forceinline__ void dmma(double &d0, double &d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

template <int NZP> struct ZmDims {
    static constexpr int MT = (NZP + 7) / 8;  // 8-row output tiles
    static constexpr int KS = (NZP + 3) / 4;  // 4-deep reduction steps
    static constexpr int MP = 8 * MT, KP = 4 * KS;
    static constexpr int LV = MP > KP ? MP : KP;  // levels stored per tile field
};

// Column swizzle of level row l for elements of B bytes: the 4-column group
// of a column is XORed with a function of l, so that the level rows a warp
// touches at once (rows 8m+g of its 4 columns in the pointwise terms, rows
// 4s+q of the mma B operand) fall on disjoint shared-memory banks.  A
// 4-aligned group of columns stays contiguous and in order.
template <int B> __host__ __device__ constexpr int zswz(int l) {
    return B == 16 ? (l & 1) << 2 : B == 8 ? (l & 3) << 2 : ((l >> 1) & 3) << 2;
}
// Field of a tile in shared memory: element (level l, column c) at
// l*kZTile + (c ^ zswz(l)).  A warp's view carries its first column c0.
template <typename V> struct ZTileF {
    V *p;
    int c0 = 0;
    __device__ __forceinline__ V &operator()(int l, int c) const {
        return p[l * kZTile + ((c0 + c) ^ zswz<(int)sizeof(V)>(l))];
    }
    __device__ __forceinline__ ZTileF<V> cols(int c) const { return ZTileF<V>{p, c0 + c}; }
};

constexpr int kZThreads = 32 * kZWarps;

// Sum over the 8 lane groups g = lane/4 (same column q): after the shuffles
// every lane holds the total of its column.
__device__ __forceinline__ double zf_colsum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    return v;
}

// out = L V for a pair tile V (levels >= nz hold zero): C[m][i] is part i of
// level 8m+g, column q
template <int MT, int KS>
__device__ __forceinline__ void zm_pair(const double (&A)[MT][KS], ZTileF<double2> V,
                                        double (&C)[MT][2], int lane) {
    const double *v = reinterpret_cast<const double *>(V.p);
    const int g = lane >> 2, q = lane & 3;
    // level 4s+q, column c0 + g/2, part g%2 (the row's swizzle depends on q only)
    const int cg = 2 * (V.c0 ^ zswz<16>(q)) + g;
#pragma unroll
    for (int m = 0; m < MT; ++m) C[m][0] = C[m][1] = 0.0;
#pragma unroll
    for (int s = 0; s < KS; ++s) {
        const double b = v[(4 * s + q) * 2 * kZTile + cg];
#pragma unroll
        for (int m = 0; m < MT; ++m) dmma(C[m][0], C[m][1], A[m][s], b);
    }
}

// Constraint, A_t rebuild, boundary rows and O after the RK combine
// (scripts/simulation/tevol_driven_cluster.m:129-136) on the same tiles and
// FP64 tensor-core products as k_zstage:
//   cons = Lz(div A) - 2 Im(conj(Psi) Lz Psi),  v = Lzr(cons) - rhoi,
//   A_t = Lzr(v) + mu (A_t(nz) = mu),  d_z A_t = Lz A_t,
//   Psi(nz) = A_x(nz) = 0, A_y(nz) = -vy,  O = Lz(nz,:) Psi (Psi(nz) = 0).
// A block takes 32 sites, a warp 8: sites 8w+j and 8w+j+4 (j = 0..3) share
// pair column 4w+j.  Psi needs two pair tiles (PA: sites 8w+j, PB: 8w+4+j);
// the real fields (div A, cons, v, A_t) pack both sites into one pair tile
// (x: site 8w+j, y: site 8w+4+j), so the real chain costs one product per 8
// sites.  Lane (g, q) owns sites 8w+q and 8w+4+q at levels 8m+g.
// The input tiles (PA, PB, div A) are double-buffered: a tile's inputs are
// requested while the previous tile computes.
constexpr int kZConsTiles = 8;  // pair tiles: 2 x (PA, PB, div A), two scratch
constexpr int kZConsSites = 2 * kZTile;
template <int NZP>
__host__ __device__ constexpr int zcons_smem_bytes() {
    return kZConsTiles * ZmDims<NZP>::LV * kZTile * 16;
}

template <int NZP>
__global__ void __launch_bounds__(kZThreads)
    k_zcons_tc(const __grid_constant__ ZConsArgs<double> a,
               const __grid_constant__ ZOps<double, NZP> op) {
    using D = ZmDims<NZP>;
    constexpr int MT = D::MT, KS = D::KS, L = D::LV * kZTile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int cw = kZCols * warp;  // pair column base of this warp
    const int nz = a.nz;
    const long long P = a.plane;
    double2 *sm = reinterpret_cast<double2 *>(g_smem);
    for (int i = tid; i < kZConsTiles * L; i += kZThreads) sm[i] = make_double2(0.0, 0.0);
    double ALz[MT][KS], ALz1[MT][KS], lzr[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const int i = 8 * m + g;
        lzr[m] = i < NZP ? op.lzb[i < NZP ? i : 0] : 0.0;
#pragma unroll
        for (int s = 0; s < KS; ++s) {
            const int j = 4 * s + q;
            const bool in = (i < NZP) && (j < NZP);
            ALz[m][s] = in ? op.Lz[in ? i : 0][in ? j : 0] : 0.0;
            ALz1[m][s] = in ? op.Lz1[in ? i : 0][in ? j : 0] : 0.0;
        }
    }
    __syncthreads();
    pdl_wait();
    const ZTileF<double2> V1{sm + 6 * L}, V2{sm + 7 * L};
    const auto V1w = V1.cols(cw), V2w = V2.cols(cw);
    const long long ntiles = (P + kZConsSites - 1) / kZConsSites;
    // inputs of the tile at site0 into buffer set b
    auto fetch = [&](long long site0, int b) {
        const ZTileF<double2> PA{sm + 3 * b * L}, PB{sm + (3 * b + 1) * L}, DV{sm + (3 * b + 2) * L};
        // site c of the tile -> pair column 4(c/8) + c%4, half (c/4)%2
#pragma unroll
        for (int it = 0; it < (NZP * kZConsSites + kZThreads - 1) / kZThreads; ++it) {
            const int e = tid + kZThreads * it, l = e / kZConsSites, c = e % kZConsSites;
            const int pc = 4 * (c >> 3) + (c & 3), h = (c >> 2) & 1;
            if (l < nz && site0 + c < P) {
                const long long gi = l * P + site0 + c;
                cp_async<16>(h ? &PB(l, pc) : &PA(l, pc), a.psi + gi);
                cp_async<8>(h ? &DV(l, pc).y : &DV(l, pc).x, a.divA + gi);
            }
        }
    };
    if ((long long)blockIdx.x < ntiles) fetch((long long)blockIdx.x * kZConsSites, 0);
    cp_commit();
    int buf = 0;
#pragma unroll 1
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, buf ^= 1) {
        const long long site0 = tile * kZConsSites;
        const long long next = tile + gridDim.x;
        if (next < ntiles) fetch(next * kZConsSites, buf ^ 1);
        cp_commit();
        cp_wait<1>();  // this tile's inputs; the next tile's may be in flight
        __syncthreads();
        const ZTileF<double2> PA{sm + 3 * buf * L}, PB{sm + (3 * buf + 1) * L},
            DV{sm + (3 * buf + 2) * L};
        const auto PAw = PA.cols(cw), PBw = PB.cols(cw), DVw = DV.cols(cw);
        const long long sA = site0 + 8 * warp + q, sB = sA + 4;  // this lane's two sites
        const bool okA = sA < P, okB = sB < P;
        {  // cons (levels < nz-1 enter Lzr)
            double cA[MT][2], cB[MT][2], c2[MT][2];
            zm_pair<MT, KS>(ALz, PAw, cA, lane);
            zm_pair<MT, KS>(ALz, PBw, cB, lane);
            zm_pair<MT, KS>(ALz, DVw, c2, lane);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int i = 8 * m + g, ic = i < nz ? i : 0;
                const double2 pa = PA(ic, cw + q), pb = PB(ic, cw + q);
                const double xA = c2[m][0] - 2.0 * (pa.x * cA[m][1] - pa.y * cA[m][0]);
                const double xB = c2[m][1] - 2.0 * (pb.x * cB[m][1] - pb.y * cB[m][0]);
                const bool in = i < nz - 1;
                V1(i, cw + q) = make_double2(in ? xA : 0.0, in ? xB : 0.0);
            }
        }
        __syncwarp();
        const double rA = okA ? a.rho[sA] : 0.0, rB = okB ? a.rho[sB] : 0.0;
        {  // v = Lzr(cons) - rhoi
            double v[MT][2];
            zm_pair<MT, KS>(ALz1, V1w, v, lane);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int i = 8 * m + g;
                const bool in = i < nz - 1;
                V2(i, cw + q) = make_double2(in ? v[m][0] - rA : 0.0, in ? v[m][1] - rB : 0.0);
            }
        }
        __syncwarp();
        {  // A_t = Lzr(v) + mu, A_t(nz) = mu
            double t[MT][2];
            zm_pair<MT, KS>(ALz1, V2w, t, lane);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int i = 8 * m + g;
                const double atA = i < nz - 1 ? t[m][0] + a.mu : (i == nz - 1 ? a.mu : 0.0);
                const double atB = i < nz - 1 ? t[m][1] + a.mu : (i == nz - 1 ? a.mu : 0.0);
                V1(i, cw + q) = make_double2(atA, atB);
            }
        }
        __syncwarp();
        {  // d_z A_t of the rebuilt potential (step-constant during the next step)
            double d[MT][2];
            zm_pair<MT, KS>(ALz, V1w, d, lane);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int i = 8 * m + g;
                if (i < nz) {
                    const double2 at = V1(i, cw + q);
                    if (okA) a.atd[(long long)i * P + sA] = make_double2(at.x, d[m][0]);
                    if (okB) a.atd[(long long)i * P + sB] = make_double2(at.y, d[m][1]);
                }
            }
        }
        // O = (Lz Psi)(nz) with Psi(nz) = 0 (:136), then the boundary rows (:133)
        double oar = 0.0, oai = 0.0, obr = 0.0, obi = 0.0;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int i = 8 * m + g, ic = i < nz - 1 ? i : 0;
            const double w = i < nz - 1 ? lzr[m] : 0.0;
            const double2 pa = PA(ic, cw + q), pb = PB(ic, cw + q);
            oar = fma(w, pa.x, oar);
            oai = fma(w, pa.y, oai);
            obr = fma(w, pb.x, obr);
            obi = fma(w, pb.y, obi);
        }
        oar = zf_colsum(oar);
        oai = zf_colsum(oai);
        obr = zf_colsum(obr);
        obi = zf_colsum(obi);
        if (g == 0) {
            const long long gb = (long long)(nz - 1) * P;
            if (okA) {
                if (a.O) a.O[sA] = make_double2(oar, oai);
                a.psi[gb + sA] = make_double2(0.0, 0.0);
                a.A[gb + sA] = make_double2(0.0, -a.vy);
            }
            if (okB) {
                if (a.O) a.O[sB] = make_double2(obr, obi);
                a.psi[gb + sB] = make_double2(0.0, 0.0);
                a.A[gb + sB] = make_double2(0.0, -a.vy);
            }
        }
        __syncthreads();  // every warp is done with this buffer set: it refills next
    }
    cp_wait<0>();
}

}  // namespace hqt
