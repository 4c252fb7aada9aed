// hqt_pfa.cuh -- line transforms of length N = P*Q (gcd(P, Q) = 1) by the
// prime-factor (Good-Thomas) algorithm, with the large factor on the tensor
// cores.
//
// With the input map n = (Q n1 + P n2) mod N and the output map
// k1 = k mod P, k2 = k mod Q, the N-point DFT is a Q-point DFT along n2 for
// every n1 followed by a P-point DFT along n1 for every k2, with no twiddle
// factors.
//   stage A (Q-point): the real-pair fold a_t = x_t + x_{Q-t},
//     b_t = x_t - x_{Q-t} is formed while loading the operand fragments; products
//     with cosine and sine matrices give P_k, Q_k and X_k = P_k -+ i Q_k,
//     X_{Q-k} = P_k +- i Q_k.
//     FP64 (mma.sync m8n8k4 f64), Q = 43: in the order of powers of 3 (Rader:
//     3 generates the residues of 43) the 21 x 21 cosine matrix depends on the sum
//     of its indices modulo 21 only, the sine matrix too up to signs.  With
//     index r + 7p (p = 0..2) the sums over p are cyclic convolutions of three
//     terms, whose constant part takes one 7 x 7 product with
//     s_r = x_0 + x_1 + x_2 and whose rest takes one 14 x 14 product with
//     x_0 - x_2, x_1 - x_2 for the outputs p = 0, 1 (the three rests add to zero,
//     which gives p = 2).  Padded to the mma that is 10 products of 8 x 8 x 4 per
//     operand tile instead of 18 for the whole 22 x 22, and 20 fragments in
//     registers instead of 36.
//     FP32 (the mixed-precision step): the whole matrices, as mma.sync m16n8k8
//     tf32 in the 3xTF32 form A_hi B_hi + A_hi B_lo + A_lo B_hi (hi = the TF32
//     rounding, lo = the TF32 rounding of the rest), accumulated in FP32.
//   stage B (P-point, P <= 8): on the CUDA cores, a lane per column, in the
//     real-pair form; as a padded tensor-core product it cost several times
//     the arithmetic.  A spectral derivative runs forward stage B, its
//     multiplier (i s1 k or s2 k^2, with the 1/N of the inverse folded in)
//     and inverse stage B in the lane's registers, so the spectrum never
//     goes to memory.
// The stage-A matrices live in registers as A fragments for the whole kernel
// (per-lane tables built by pfa_fragments / pfa_fragments32, uploaded at
// init); the data is the B operand, read from the warp's shared memory in
// split real/imaginary planes.
//
// One warp transforms kPfaLines lines at a time and shares nothing with
// other warps, so only __syncwarp orders its stages.
#pragma once
#include <cmath>
#include <cstring>
#include <type_traits>

#include "hqt_dev.cuh"
#include "hqt_args.h"

namespace hqt {

constexpr int kPfaLines = 2;  // lines per warp

__host__ __device__ constexpr int pfa_modinv(int a, int m) {
    for (int x = 1; x < m; ++x)
        if ((a * x) % m == 1) return x;
    return 1;
}

template <int P_, int Q_> struct PfaDims {
    static constexpr int P = P_, Q = Q_, N = P_ * Q_, M = (Q_ - 1) / 2;
    static constexpr int U = kPfaLines * P;      // stage-A columns: (line, n1)
    static constexpr int NTA = (2 * U + 7) / 8;  // ... times (re, im), 8 per tile
    static constexpr int CB = kPfaLines * Q;     // stage-B columns: (line, k2)
    static constexpr int QIP = pfa_modinv(Q_ % P_, P_), PIQ = pfa_modinv(P_ % Q_, Q_);
    // FP64 stage A: m8n8k4 tiles of the constant part (1 x 2 reduction steps) and
    // of the rest (2 x 4), cos and sin
    static constexpr int NFRAG = 2 * (2 + 8);
    // FP32 stage A: m16n8k8 tiles; per lane 4 registers per tile, hi and lo
    static constexpr int MT32 = (M + 1 + 15) / 16, KS32 = (M + 1 + 7) / 8;
    static constexpr int NFRAG32 = 2 * 2 * MT32 * KS32 * 4;  // cos/sin x hi/lo
    static_assert(2 * P_ <= 16 && Q_ == 43, "P <= 8; Q = 43 (powers of 3, 21 = 3 * 7)");
};

// Storage of the Q entries of a column u in shared memory.  FP32: in order, Q
// apart.  FP64: entry 3^i mod 43 at position i, entry 0 at 42, columns 44 apart:
// stage A's operand rows and results (powers r + 7p, and r + 7p + 21 for the
// negative) are then runs of adjacent elements at fixed offsets, and its accesses
// nearly free of bank conflicts (per 43-point stage of two lines 264 wavefronts
// instead of 431, of 192 without any).
template <typename T, int P, int Q> struct PfaStore {
    static constexpr bool kPow = std::is_same<T, double>::value;
    static constexpr int PITCH = kPow ? 44 : Q;
    static constexpr int SIZE = kPfaLines * P * PITCH;  // complex elements of a buffer
};

// One buffer in shared memory: values of [u][t], u = line*P + n1.  FP64:
// interleaved (16-byte copies, reads and writes); FP32: split planes.
template <typename T> struct PfaBuf;
template <> struct PfaBuf<double> {
    double2 *c;
    __device__ __forceinline__ double *re(int i) const { return &c[i].x; }
    __device__ __forceinline__ double *im(int i) const { return &c[i].y; }
    __device__ __forceinline__ double2 get(int i) const { return c[i]; }
    __device__ __forceinline__ void put(int i, double x, double y) const { c[i] = make_double2(x, y); }
    // cp.async of a complex value
    __device__ __forceinline__ void copy(int i, const double2 *src) const { cp_async<16>(c + i, src); }
};
template <> struct PfaBuf<float> {
    float *r, *m;
    __device__ __forceinline__ float *re(int i) const { return r + i; }
    __device__ __forceinline__ float *im(int i) const { return m + i; }
    __device__ __forceinline__ float2 get(int i) const { return make_float2(r[i], m[i]); }
    __device__ __forceinline__ void put(int i, float x, float y) const {
        r[i] = x;
        m[i] = y;
    }
    __device__ __forceinline__ void copy(int i, const float2 *src) const {
        cp_async<4>(r + i, &src->x);
        cp_async<4>(m + i, &src->y);
    }
};

// d += a * b on one 8x8x4 FP64 tensor-core tile
__device__ __forceinline__ void pfa_mma(double &d0, double &d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}
// d += a * b on one 16x8x8 TF32 tile (FP32 accumulators)
__device__ __forceinline__ void pfa_mma_tf32(float (&d)[4], const unsigned (&a)[4], unsigned b0,
                                             unsigned b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pfa_tf32(float x) {
    unsigned r;
    asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
    return r;
}

// Combine P_k, Q_k into X_k (at k) and X_{Q-k} (at kn) (SIGN -1 forward).
template <int SIGN, typename T, typename Put>
__device__ __forceinline__ void pfa_unfold(int u, int k, int kn, T pr, T pi, T qr, T qi, Put put) {
    if (SIGN < 0) {
        put(u, k, pr + qi, pi - qr);
        put(u, kn, pr - qi, pi + qr);
    } else {
        put(u, k, pr - qi, pi + qr);
        put(u, kn, pr + qi, pi - qr);
    }
}

template <typename T, int P, int Q> struct PfaStageA;

// 3^i mod 43: the order of the FP64 stage A
__host__ __device__ constexpr int pfa_pow3(int i) {
    int v = 1;
    for (int k = 0; k < i; ++k) v = v * 3 % 43;
    return v;
}

// FP64 stage A.  Lane (g, q): operand rows r = 4s + q (s = 0, 1; r = 7 stands for
// x_0), result row r' = g (7: X_0) of column u = 4nt + q, parts re and im.
template <int P, int Q> struct PfaStageA<double, P, Q> {
    using D = PfaDims<P, Q>;
    static constexpr int PITCH = PfaStore<double, P, Q>::PITCH;
    double Cd[2], Cw[2][4], Sd[2], Sw[2][4];  // constant part, rest; cos, sin

    __device__ __forceinline__ void init(const double *frag, int lane) {
        const double *f = frag + lane;
#pragma unroll
        for (int s = 0; s < 2; ++s, f += 32) Cd[s] = *f;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int s = 0; s < 4; ++s, f += 32) Cw[m][s] = *f;
#pragma unroll
        for (int s = 0; s < 2; ++s, f += 32) Sd[s] = *f;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int s = 0; s < 4; ++s, f += 32) Sw[m][s] = *f;
    }

    // Two operand tiles per pass: twice the independent accumulator chains
    // in flight.  Tiles past NTA read as zero and put nothing (uc, u >= U).
    // LEVEL (for a derivative): of the lines less one of their elements.  A constant
    // drops out anyway, but its rounding does not: A_x, which the derivative of a
    // nearly uniform A_t drives, was a third less exact after ten steps than with
    // 43 products a row.
    template <int SIGN, bool LEVEL, typename Put>
    __device__ __forceinline__ void run(PfaBuf<double> in, Put put, int g, int q) const {
        static_assert(kPfaLines == 2, "levels of two lines");
        double level[2] = {0.0, 0.0};
        if (LEVEL) {
            level[0] = in.re(42)[g & 1];
            level[1] = in.re(P * PITCH + 42)[g & 1];
        }
#pragma unroll 1
        for (int n0 = 0; n0 < D::NTA; n0 += 2) {
            double pc[2][3][2], ps[2][3][2];  // u, w_0, w_1 of the cos and sin products
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int m = 0; m < 3; ++m)
                    pc[j][m][0] = pc[j][m][1] = ps[j][m][0] = ps[j][m][1] = 0.0;
#pragma unroll
            for (int s = 0; s < 2; ++s) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int uc = 4 * (n0 + j) + (g >> 1);  // operand column (u, part g&1)
                    // rows r = 4s + q (row 7: entries of other rows, times zero)
                    const double *x = in.re((uc < D::U ? uc : 0) * PITCH + 4 * s + q) + (g & 1);
                    const double c = uc < P ? level[0] : level[1];
                    double a[3], b[3];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        double xt = x[2 * (7 * p)], xr = x[2 * (7 * p + 21)];
                        if (LEVEL) {
                            xt -= c;
                            xr -= c;
                        }
                        a[p] = xt + xr;
                        b[p] = xt - xr;
                    }
                    // row 7 of the constant part is x_0 itself
                    const double sa = s == 1 && q == 3 ? x[2 * (42 - 7)] - (LEVEL ? c : 0.0)
                                                       : a[0] + a[1] + a[2];
                    const double sb = b[0] - b[1] + b[2];
                    const double a0 = a[0] - a[2], a1 = a[1] - a[2];
                    const double b0 = b[0] - b[2], b1 = b[1] + b[2];
                    pfa_mma(pc[j][0][0], pc[j][0][1], Cd[s], sa);
                    pfa_mma(ps[j][0][0], ps[j][0][1], Sd[s], sb);
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        pfa_mma(pc[j][1 + m][0], pc[j][1 + m][1], Cw[m][s], a0);
                        pfa_mma(ps[j][1 + m][0], ps[j][1 + m][1], Sw[m][s], b0);
                    }
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        pfa_mma(pc[j][1 + m][0], pc[j][1 + m][1], Cw[m][2 + s], a1);
                        pfa_mma(ps[j][1 + m][0], ps[j][1 + m][1], Sw[m][2 + s], b1);
                    }
                }
            }
            // The tiles write only their own columns, after all their reads:
            // stage A may run in place.
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int u = 4 * (n0 + j) + q;
                if (u >= D::U) continue;
                const double(&c)[3][2] = pc[j];
                const double(&e)[3][2] = ps[j];
                if (g == 7) {
                    put(u, 42, c[0][0], c[0][1]);
                    continue;
                }
                double pr[3], pi[3], qr[3], qi[3];
                pr[0] = c[0][0] + c[1][0];
                pi[0] = c[0][1] + c[1][1];
                pr[1] = c[0][0] + c[2][0];
                pi[1] = c[0][1] + c[2][1];
                pr[2] = c[0][0] - (c[1][0] + c[2][0]);
                pi[2] = c[0][1] - (c[1][1] + c[2][1]);
                qr[0] = e[0][0] + e[1][0];
                qi[0] = e[0][1] + e[1][1];
                qr[1] = -(e[0][0] + e[2][0]);
                qi[1] = -(e[0][1] + e[2][1]);
                qr[2] = e[0][0] - (e[1][0] + e[2][0]);
                qi[2] = e[0][1] - (e[1][1] + e[2][1]);
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    pfa_unfold<SIGN>(u, g + 7 * p, g + 7 * p + 21, pr[p], pi[p], qr[p], qi[p],
                                     put);
            }
        }
    }
};

// FP32 stage A in the 3xTF32 form: fragments a0 = L[16m+g][8s+q],
// a1 = L[16m+g+8][8s+q], a2 = L[16m+g][8s+q+4], a3 = L[16m+g+8][8s+q+4];
// operand b0 = V[8s+q][col g], b1 = V[8s+q+4][col g]; result
// c0, c1 = out[16m+g][col 2q, 2q+1], c2, c3 = out[16m+g+8][col 2q, 2q+1].
template <int P, int Q> struct PfaStageA<float, P, Q> {
    using D = PfaDims<P, Q>;
    static constexpr int M = D::M, MT = D::MT32, KS = D::KS32;
    unsigned Ch[MT][KS][4], Cl[MT][KS][4], Sh[MT][KS][4], Sl[MT][KS][4];

    __device__ __forceinline__ void init(const float *frag, int lane) {
        int j = 0;
        auto ld = [&](unsigned (&A)[MT][KS][4]) {
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int s = 0; s < KS; ++s)
#pragma unroll
                    for (int r = 0; r < 4; ++r) A[m][s][r] = __float_as_uint(frag[32 * j++ + lane]);
        };
        ld(Ch);
        ld(Cl);
        ld(Sh);
        ld(Sl);
    }

    // Two operand tiles per pass, as in FP64.
    template <int SIGN, bool, typename Put>
    __device__ __forceinline__ void run(PfaBuf<float> in, Put put, int g, int q) const {
#pragma unroll 1
        for (int n0 = 0; n0 < D::NTA; n0 += 2) {
            float pa[2][MT][4], qa[2][MT][4];
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int r = 0; r < 4; ++r) pa[j][m][r] = qa[j][m][r] = 0.0f;
            const float *pl = (g & 1) ? in.m : in.r;
#pragma unroll
            for (int s = 0; s < KS; ++s) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int uc = 4 * (n0 + j) + (g >> 1);
                    float av[2], bv[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int t = 8 * s + q + 4 * h;
                        float a = 0.0f, b = 0.0f;
                        if (uc < D::U && t <= M) {
                            const float xt = pl[uc * Q + t];
                            if (t == 0) {
                                a = xt;
                            } else {
                                const float xr = pl[uc * Q + (Q - t)];
                                a = xt + xr;
                                b = xt - xr;
                            }
                        }
                        av[h] = a;
                        bv[h] = b;
                    }
                    const unsigned ah0 = pfa_tf32(av[0]), ah1 = pfa_tf32(av[1]);
                    const unsigned al0 = pfa_tf32(av[0] - __uint_as_float(ah0));
                    const unsigned al1 = pfa_tf32(av[1] - __uint_as_float(ah1));
                    const unsigned bh0 = pfa_tf32(bv[0]), bh1 = pfa_tf32(bv[1]);
                    const unsigned bl0 = pfa_tf32(bv[0] - __uint_as_float(bh0));
                    const unsigned bl1 = pfa_tf32(bv[1] - __uint_as_float(bh1));
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        pfa_mma_tf32(pa[j][m], Cl[m][s], ah0, ah1);
                        pfa_mma_tf32(pa[j][m], Ch[m][s], al0, al1);
                        pfa_mma_tf32(pa[j][m], Ch[m][s], ah0, ah1);
                        pfa_mma_tf32(qa[j][m], Sl[m][s], bh0, bh1);
                        pfa_mma_tf32(qa[j][m], Sh[m][s], bl0, bl1);
                        pfa_mma_tf32(qa[j][m], Sh[m][s], bh0, bh1);
                    }
                }
            }
            __syncwarp();  // in-place safe, as in FP64
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int u = 4 * (n0 + j) + q;
                if (u < D::U) {
#pragma unroll
                    for (int m = 0; m < MT; ++m)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int k = 16 * m + g + 8 * h;
                            if (k > M) continue;
                            if (k == 0)
                                put(u, 0, pa[j][m][2 * h], pa[j][m][2 * h + 1]);
                            else
                                pfa_unfold<SIGN>(u, k, Q - k, pa[j][m][2 * h],
                                                 pa[j][m][2 * h + 1], qa[j][m][2 * h],
                                                 qa[j][m][2 * h + 1], put);
                        }
                }
            }
        }
    }
};

template <typename T, int P, int Q> struct PfaWarp {
    using D = PfaDims<P, Q>;
    using S = PfaStore<T, P, Q>;
    static constexpr int N = D::N;
    PfaStageA<T, P, Q> sa;
    int lane, g, q;
    const unsigned short *k2tab;  // FP64: entry at each position

    __device__ __forceinline__ void init(const T *frag, const unsigned short *k2) {
        k2tab = k2;
        lane = threadIdx.x & 31;
        g = lane >> 2;
        q = lane & 3;
        sa.init(frag, lane);
    }

    // Stage A along t for every column u of `in`; SIGN -1 forward, +1 inverse.
    // The result X(u, k) goes to put(u, e, re, im), e the position of k.
    // LEVEL: for a derivative (FP64: less a constant, PfaStageA).
    template <int SIGN, bool LEVEL = false, typename Put>
    __device__ __forceinline__ void stage_a(PfaBuf<T> in, Put put) const {
        sa.template run<SIGN, LEVEL>(in, put, g, q);
    }
    // entry at position e of a column
    __device__ __forceinline__ int entry(int e) const {
        if constexpr (S::kPow)
            return __ldg(k2tab + e);
        else
            return e;
    }

    // Stage B on the CUDA cores, a lane per column (line, k2), in the
    // real-pair form with cos/sin(2 pi j/P) in `cs`: values v(n1) of `in`
    // (rows u = line*P + n1) -> forward P-point DFT if FWD -> mul(line, k1,
    // k2, re, im) on every entry -> inverse P-point DFT if INV -> `out`
    // (same rows).  The spectrum never goes to memory between the two DFTs.
    template <bool FWD, bool INV, typename Mul>
    __device__ __forceinline__ void stage_b(PfaBuf<T> in, PfaBuf<T> out, const T (&cs)[2][P],
                                            Mul mul) const {
        constexpr int H = (P - 1) / 2;
#pragma unroll 1
        for (int col = lane; col < D::CB; col += 32) {
            const int ln = col / Q, e2 = col - ln * Q, k2 = entry(e2);
            T zr[P], zi[P], xr[P], xi[P];
            load(in, ln, e2, zr, zi);
            if (FWD) {
                dft_real_pair<-1, H>(zr, zi, xr, xi, cs);
            } else {
#pragma unroll
                for (int k1 = 0; k1 < P; ++k1) {
                    xr[k1] = zr[k1];
                    xi[k1] = zi[k1];
                }
            }
#pragma unroll
            for (int k1 = 0; k1 < P; ++k1) mul(ln, k1, k2, xr[k1], xi[k1]);
            if (INV) {
                dft_real_pair<+1, H>(xr, xi, zr, zi, cs);
            } else {
#pragma unroll
                for (int k1 = 0; k1 < P; ++k1) {
                    zr[k1] = xr[k1];
                    zi[k1] = xi[k1];
                }
            }
            store(out, ln, e2, zr, zi);
        }
    }
    __device__ __forceinline__ static void load(PfaBuf<T> b, int ln, int e2, T (&zr)[P], T (&zi)[P]) {
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) {
            const int e = (ln * P + n1) * S::PITCH + e2;
            const C2<T> v = b.get(e);
            zr[n1] = v.x;
            zi[n1] = v.y;
        }
    }
    __device__ __forceinline__ static void store(PfaBuf<T> b, int ln, int e2, const T (&zr)[P],
                                                 const T (&zi)[P]) {
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) {
            const int e = (ln * P + n1) * S::PITCH + e2;
            b.put(e, zr[n1], zi[n1]);
        }
    }

    // natural index k of spectral entry (k1, k2): k = k1 mod P, k = k2 mod Q
    __device__ __forceinline__ static int crt(int k1, int k2) {
        return (Q * D::QIP * k1 + P * D::PIQ * k2) % N;
    }
    // its signed wavenumber (k or k - N)
    __device__ __forceinline__ static T wavenumber(int k1, int k2) {
        const int k = crt(k1, k2);
        return (T)(2 * k < N ? k : k - N);
    }

    // derivative ORDER (1: i*s1*kk, 2: s2*kk^2) of a field after stage A
    template <int ORDER>
    __device__ __forceinline__ void stage_b_deriv(PfaBuf<T> in, PfaBuf<T> out, T s1, T s2,
                                                  const T (&cs)[2][P]) const {
        stage_b<true, true>(in, out, cs, [&](int, int k1, int k2, T &re, T &im) {
            const T w = wavenumber(k1, k2);
            if (ORDER == 1) {  // (i s1 w X): re = -s1 w X.im, im = s1 w X.re
                const T m = s1 * w, r = re;
                re = -m * im;
                im = m * r;
            } else {
                const T m = s2 * w * w;
                re *= m;
                im *= m;
            }
        });
    }

    // first and second derivative of a field after stage A in one pass over its
    // spectrum: the first into `out`, the second in place
    __device__ __forceinline__ void stage_b_deriv12(PfaBuf<T> in, PfaBuf<T> out, T s1, T s2,
                                                    const T (&cs)[2][P]) const {
        constexpr int H = (P - 1) / 2;
#pragma unroll 1
        for (int col = lane; col < D::CB; col += 32) {
            const int ln = col / Q, e2 = col - ln * Q, k2 = entry(e2);
            T zr[P], zi[P], xr[P], xi[P], yr[P], yi[P];
            load(in, ln, e2, zr, zi);
            dft_real_pair<-1, H>(zr, zi, xr, xi, cs);
#pragma unroll
            for (int k1 = 0; k1 < P; ++k1) {
                const T w = wavenumber(k1, k2), m = s1 * w, m2 = s2 * w * w;
                yr[k1] = -m * xi[k1];
                yi[k1] = m * xr[k1];
                xr[k1] *= m2;
                xi[k1] *= m2;
            }
            dft_real_pair<+1, H>(yr, yi, zr, zi, cs);
            store(out, ln, e2, zr, zi);
            dft_real_pair<+1, H>(xr, xi, zr, zi, cs);
            store(in, ln, e2, zr, zi);
        }
    }

    // P-point DFT of (xr, xi) into (yr, yi), sign SIGN, real-pair form.
    template <int SIGN, int H>
    __device__ __forceinline__ static void dft_real_pair(const T (&xr)[P], const T (&xi)[P],
                                                         T (&yr)[P], T (&yi)[P],
                                                         const T (&cs)[2][P]) {
        T ar[H + 1], ai[H + 1], br[H + 1], bi[H + 1];
#pragma unroll
        for (int t = 1; t <= H; ++t) {
            ar[t] = xr[t] + xr[P - t];
            ai[t] = xi[t] + xi[P - t];
            br[t] = xr[t] - xr[P - t];
            bi[t] = xi[t] - xi[P - t];
        }
        T sr = xr[0], si = xi[0];
#pragma unroll
        for (int t = 1; t <= H; ++t) {
            sr += ar[t];
            si += ai[t];
        }
        yr[0] = sr;
        yi[0] = si;
#pragma unroll
        for (int k = 1; k <= H; ++k) {
            T pr = xr[0], pi = xi[0], qr = T(0), qi = T(0);
#pragma unroll
            for (int t = 1; t <= H; ++t) {
                const int j = (t * k) % P;
                pr = fma(ar[t], cs[0][j], pr);
                pi = fma(ai[t], cs[0][j], pi);
                qr = fma(br[t], cs[1][j], qr);
                qi = fma(bi[t], cs[1][j], qi);
            }
            // SIGN -1: X_k = P - iQ, X_{P-k} = P + iQ; SIGN +1: the reverse
            const T s = (T)SIGN;
            yr[k] = pr - s * qi;
            yi[k] = pi + s * qr;
            yr[P - k] = pr + s * qi;
            yi[P - k] = pi - s * qr;
        }
    }
};

// Host side: cos/sin of the stage-A matrices at exactly reduced arguments.
template <int P, int Q> double pfa_matrix(int part, int k, int t) {
    const int M = (Q - 1) / 2;
    const double two_pi = 6.283185307179586476925286766559;
    if (k > M || t > M) return 0.0;
    if (part == 0) return t == 0 ? 1.0 : std::cos(two_pi * ((t * k) % Q) / Q);
    return (t == 0 || k == 0) ? 0.0 : std::sin(two_pi * ((t * k) % Q) / Q);
}

// Host side: the per-lane FP64 fragment table (NFRAG x 32 doubles): constant part
// and rest of the cos, then of the sin matrix, in the order of powers of 3.
template <int P, int Q> void pfa_fragments(double *tab) {
    const long double two_pi = 6.283185307179586476925286766559005768L;
    // c(n) = cos(2 pi 3^n/43), period 21; s(n) = (-1)^n sin(2 pi 3^n/43), period 21
    auto kern = [&](int part, int n) -> long double {
        n %= 21;
        const long double t = two_pi * pfa_pow3(n) / Q;
        return part == 0 ? std::cos(t) : (n % 2 ? -std::sin(t) : std::sin(t));
    };
    auto mean = [&](int part, int m) {
        return (kern(part, m) + kern(part, m + 7) + kern(part, m + 14)) / 3;
    };
    int j = 0;
    for (int part = 0; part < 2; ++part) {
        // sin: rows and columns carry (-1)^index, the p = 1 terms another sign
        auto sg = [&](int i) { return part == 1 && i % 2 ? -1.0L : 1.0L; };
        for (int s = 0; s < 2; ++s, ++j)
            for (int lane = 0; lane < 32; ++lane) {
                const int i = lane >> 2, r = 4 * s + (lane & 3);
                long double v;
                if (i < 7 && r < 7)
                    v = sg(i) * sg(r) * mean(part, i + r);
                else
                    v = part == 0 ? 1 : 0;  // x_0 in every P_k, all of it in X_0
                tab[32 * j + lane] = (double)v;
            }
        for (int m = 0; m < 2; ++m)
            for (int s = 0; s < 4; ++s, ++j)
                for (int lane = 0; lane < 32; ++lane) {
                    const int i = lane >> 2, r = 4 * (s & 1) + (lane & 3), d = s >> 1;
                    long double v = 0;
                    if (i < 7 && r < 7)
                        v = sg(i) * sg(r) * (part == 1 && d == 1 ? -1 : 1) *
                            (kern(part, i + r + 7 * (m + d)) - mean(part, i + r));
                    tab[32 * j + lane] = (double)v;
                }
    }
}

// TF32 rounding (to nearest, ties away from zero) of a float on the host:
// the value cvt.rna.tf32.f32 gives, 10 explicit mantissa bits.
inline float pfa_host_tf32(float x) {
    unsigned u;
    std::memcpy(&u, &x, 4);
    if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & 0xffffe000u;
    float r;
    std::memcpy(&r, &u, 4);
    return r;
}

// Host side: the per-lane FP32 fragment table (NFRAG32 x 32 floats): cos hi,
// cos lo, sin hi, sin lo, each [m][s][register].
template <int P, int Q> void pfa_fragments32(float *tab) {
    using D = PfaDims<P, Q>;
    int j = 0;
    for (int part = 0; part < 2; ++part)
        for (int hl = 0; hl < 2; ++hl)
            for (int m = 0; m < D::MT32; ++m)
                for (int s = 0; s < D::KS32; ++s)
                    for (int r = 0; r < 4; ++r, ++j)
                        for (int lane = 0; lane < 32; ++lane) {
                            const int g = lane >> 2, q = lane & 3;
                            const int k = 16 * m + g + 8 * (r & 1), t = 8 * s + q + 4 * (r >> 1);
                            const double v = pfa_matrix<P, Q>(part, k, t);
                            const float hi = pfa_host_tf32((float)v);
                            const float lo = pfa_host_tf32((float)(v - (double)hi));
                            tab[32 * j + lane] = hl == 0 ? hi : lo;
                        }
}

}  // namespace hqt
