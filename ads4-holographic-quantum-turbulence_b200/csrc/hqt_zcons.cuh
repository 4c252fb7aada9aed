// hqt_zcons.cuh -- the radial (Chebyshev) work after the RK combine: the
// constraint, the A_t rebuild and the boundary rows
// (scripts/simulation/tevol_driven_cluster.m:129-136).
//   cons = Lz(div A) - 2 Im(conj(Psi) Lz Psi),  v = Lzr(cons) - rhoi,
//   A_t = Lzr(v) + mu (A_t(nz) = mu),  d_z A_t = Lz A_t,
//   Psi(nz) = A_x(nz) = 0, A_y(nz) = -vy,  O = Lz(nz,:) Psi (Psi(nz) = 0).
//
// Operators, fragments and copies as in hqt_zstage.cuh.  A block of four warps takes
// tiles of 32 sites, a warp 8 of them in two halves of 4: Psi is two operands (an
// mma's 8 columns are 4 sites x 2 parts), the real fields (div A, cons, v, A_t) are
// one, (site of the first half, site of the second) as a pair, in two scratch fields
// of pairs.  Inputs are double-buffered: two tiles ahead, one box of Psi and one of
// div A each.
//
// Shared-memory rows: Psi 34 pairs (544 bytes), div A 36 values (288 bytes).  With
// these pitches and the sites a warp takes (zc_site) the mma operand reads (4 levels
// x 2 sites x 2 parts a half warp) and the pointwise reads are free of bank
// conflicts.
//
// Bound: 40 bytes a site through HBM at up to 25 levels, the FP64 tensor cores beside
// it at 33 (152 mma for 8 columns of 33 levels); the chain of four dependent products
// a tile, with 8 to 12 warps on an SM, keeps it at 2 to 2.5 times that.  Measured, us
// a launch, with full-size products of tiles copied by cp.async -> this kernel:
// 301x301x21 46 -> 35, 512x512x25 136 -> 92 (2.8 TB/s), 1001x1001x20 306 -> 287,
// 1024x1024x33 1430 -> 536.
#pragma once
#include "hqt_zstage.cuh"

namespace hqt {

// site k of a warp's first (half 0) or second 4
__device__ __forceinline__ int zc_site(int warp, int k, int half) {
    return 16 * (warp >> 1) + 4 * (warp & 1) + (k & 1) + (half ? 2 + 6 * (k >> 1) : 10 * (k >> 1));
}

template <int NZP> struct ZcLay {
    static constexpr int up(int b) { return (b + 127) / 128 * 128; }
    static constexpr int rp = up(NZP * kZcRowP), rd = up(NZP * kZcRowD) + 128;
    static constexpr int rv = up(ZsDims<NZP>::VR * kZsRow);
    static constexpr int oV1 = 2 * (rp + rd), oV2 = oV1 + rv, oTAB = oV2 + rv;
    static constexpr int oBAR = oTAB + up(ZsDims<NZP>::ntab * 8);
    static constexpr int bytes = oBAR + 64 + 128;  // + alignment of the base
    static constexpr int min_blocks = NZP > 25 ? 2 : 3;
};

template <int NZP>
__global__ void __launch_bounds__(kZsThreads, ZcLay<NZP>::min_blocks)
    k_zcons(const __grid_constant__ ZConsArgs<double> a) {
    using Lay = ZcLay<NZP>;
    using D = ZsDims<NZP>;
    constexpr int MH = D::MH, M1 = D::M1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int nz = a.nz, n1 = nz - 1, h = (nz + 1) / 2;
    const long long P = a.plane;
    unsigned char *sm = g_smem + ((128 - ((unsigned)__cvta_generic_to_shared(g_smem) & 127)) & 127);
    const unsigned sb = (unsigned)__cvta_generic_to_shared(sm), bar = sb + Lay::oBAR;
    double *tab = reinterpret_cast<double *>(sm + Lay::oTAB);
    for (int i = threadIdx.x; i < D::ntab; i += kZsThreads) tab[i] = __ldg(a.ztab + i);
    for (int i = threadIdx.x; i < 2 * Lay::rv / 16; i += kZsThreads)
        reinterpret_cast<double2 *>(sm + Lay::oV1)[i] = make_double2(0.0, 0.0);
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) zs_bar_init(bar + 8 * b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    const double *line = tab + 3 * NZP;
    const ZsSplit sreal(nz, P * 8, kZcRowD);
    const int odd = sreal.n > 1 ? sreal.start(1) + sreal.shift(1) : 0;
    auto rowd = [&](int i) { return (i >> sreal.lg) * kZcRowD + (i & sreal.lg) * odd; };
    const ZsOps<NZP> ops(a.frag, lane, warp, nz);
    pdl_wait();

    const long long ntiles = (P + kZcSites - 1) / kZcSites;
    auto load = [&](long long tile, int b) {
        if (tile >= ntiles) return;
        const long long s0 = tile * kZcSites;
        const int ps = b * (Lay::rp + Lay::rd), dv = ps + Lay::rp;
        if (threadIdx.x == 0) {
            zs_expect(bar + 8 * b, nz * (kZcRowP + kZcRowD));
            zs_tma(sb + ps, &a.mPS, (int)(2 * s0), bar + 8 * b);
            for (int ph = 0; ph < sreal.n; ++ph)
                zs_tma(sb + dv + sreal.start(ph), a.mDIV + ph, (int)s0, bar + 8 * b);
        }
    };
    load(blockIdx.x, 0);
    load((long long)blockIdx.x + gridDim.x, 1);
    const int kk = lane >> 3, part = (lane >> 2) & 1;      // operand column of this lane
    const int oA = zc_site(warp, kk, 0) * 16 + part * 8, oB = zc_site(warp, kk, 1) * 16 + part * 8;
    const int oD = zc_site(warp, kk, part) * 8;
    const int cA = zc_site(warp, q, 0), cB = zc_site(warp, q, 1);  // its result columns
    const int col = zs_col(warp, q), gr = zs_row(g);
    int lost = 0;  // 1, 2: waited in vain, with and without the next tile in flight
    int buf = 0, parity = 0;
#pragma unroll 1
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long sA = tile * kZcSites + cA, sB = tile * kZcSites + cB;
        const bool okA = sA < P, okB = sB < P;
        const unsigned char *ps = sm + buf * (Lay::rp + Lay::rd), *dv = ps + Lay::rp;
        auto psi = [&](int i, int c) {
            return *reinterpret_cast<const double2 *>(ps + i * kZcRowP + c * 16);
        };
        const double rA = okA ? a.rho[sA] : 0.0, rB = okB ? a.rho[sB] : 0.0;
        if (!lost && !zs_wait(bar + 8 * buf, parity, a.polls))
            lost = tile + gridDim.x < ntiles ? 1 : 2;

        // ---- cons -> V1 (levels < nz - 1 enter Lzr), O -------------------------
        double oar = 0.0, oai = 0.0, obr = 0.0, obi = 0.0;
        {
            double tA[MH][2], tB[MH][2];
            ops.lz([&](int j) { return *reinterpret_cast<const double *>(dv + rowd(j) + oD); },
                   line, tA, tB);
            double yA[MH][2], yB[MH][2], wA[MH][2], wB[MH][2];
            ops.lz2([&](int j) { return *reinterpret_cast<const double *>(ps + j * kZcRowP + oA); },
                    [&](int j) { return *reinterpret_cast<const double *>(ps + j * kZcRowP + oB); },
                    line, yA, yB, wA, wB);
            auto put = [&](int i, const double (&t)[2], const double (&y)[2],
                           const double (&w)[2]) {
                const double2 pa = psi(i, cA), pb = psi(i, cB);
                const bool in = i < n1;
                const double xA = t[0] - 2.0 * (pa.x * y[1] - pa.y * y[0]);
                const double xB = t[1] - 2.0 * (pb.x * w[1] - pb.y * w[0]);
                zs_at<Lay::oV1>(sm, i, col) = make_double2(in ? xA : 0.0, in ? xB : 0.0);
                if (in) {
                    const double c = tab[2 * NZP + i];
                    oar = fma(c, pa.x, oar);
                    oai = fma(c, pa.y, oai);
                    obr = fma(c, pb.x, obr);
                    obi = fma(c, pb.y, obi);
                }
            };
#pragma unroll
            for (int m = 0; m < MH; ++m) {
                const int i = 8 * m + gr;
                if (i < h) {
                    put(i, tA[m], yA[m], wA[m]);
                    if (n1 - i != i) put(n1 - i, tB[m], yB[m], wB[m]);
                }
            }
        }
        zs_release();
        __syncthreads();  // every warp is done with this buffer
        if (!lost) load(tile + 2 * (long long)gridDim.x, buf);
        {  // v = Lzr(cons) - rhoi -> V2
            double F[M1][2];
            ops.template lz1<Lay::oV1>(sm, F);
            ops.rows(F, g, [&](int, int i, double fx, double fy) {
                const bool in = i < n1;
                zs_at<Lay::oV2>(sm, i, col) = make_double2(in ? fx - rA : 0.0, in ? fy - rB : 0.0);
            });
        }
        __syncwarp();
        {  // A_t = Lzr(v) + mu -> V1
            double F[M1][2];
            ops.template lz1<Lay::oV2>(sm, F);
            ops.rows(F, g, [&](int, int i, double fx, double fy) {
                const bool in = i < n1;
                zs_at<Lay::oV1>(sm, i, col) =
                    make_double2(in ? fx + a.mu : a.mu, in ? fy + a.mu : a.mu);
            });
        }
        __syncwarp();
        {  // d_z A_t of the rebuilt potential (step-constant during the next step)
            double yA[MH][2], yB[MH][2];
            ops.lz([&](int j) { return ops.template operand<Lay::oV1>(sm, j); }, line, yA, yB);
            auto put = [&](int i, const double (&d)[2]) {
                const double2 at = zs_at<Lay::oV1>(sm, i, col);
                if (okA) a.atd[(long long)i * P + sA] = make_double2(at.x, d[0]);
                if (okB) a.atd[(long long)i * P + sB] = make_double2(at.y, d[1]);
            };
#pragma unroll
            for (int m = 0; m < MH; ++m) {
                const int i = 8 * m + gr;
                if (i < h) {
                    put(i, yA[m]);
                    if (n1 - i != i) put(n1 - i, yB[m]);
                }
            }
        }
        __syncwarp();  // V1 is read: the next tile overwrites it
        oar = zf_colsum(oar);
        oai = zf_colsum(oai);
        obr = zf_colsum(obr);
        obi = zf_colsum(obi);
        if (g == 0) {
            const long long gb = (long long)n1 * P;
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
        if (!lost) {
            parity ^= buf;
            buf ^= 1;
        }
    }
    if (lost) {
        if (threadIdx.x == 0) zs_drain(bar + 8 * buf, parity);
        if (threadIdx.x == 0 && lost == 1) zs_drain(bar + 8 * (buf ^ 1), parity ^ buf);
        *a.fault = 1;
    }
}

}  // namespace hqt
