// hqt_lineplan.h -- plans of the in-place line transforms (hqt_line.cuh):
// shared by the host (tables) and the kernels.
#pragma once
#include "hqt_common.cuh"

namespace hqt {

constexpr int kLMaxPass = 6;
constexpr int kLThreads = 512;  // largest block

// n = R[0] .. R[np-1]; s[p] = R[p+1] .. R[np-1]; tw[p] = offset of pass p's
// twiddles, (R[p] - 1) * s[p] entries [k][j] = exp(-2 pi i j k / (R[p] s[p])),
// k >= 1 (the last pass has none); ntw = their total.  np = 0: no plan.
struct LPlan {
    int n, np, ntw;
    int R[kLMaxPass], s[kLMaxPass], tw[kLMaxPass];
};

// Radices of a pass: up to 13; larger primes have no in-place pass.  (An FP64
// radix 16 as the first pass spilled in 128 registers: y_rhs of 128x128x17
// 15.4 -> 21.0 us, of 1024x1024x17 1053 -> 1157 us, against 8*4*4 and
// 8*8*4*4.)

struct LSearch {
    int np, mx, sum, last;
    int cur[kLMaxPass], best[kLMaxPass];
};
__host__ __device__ constexpr void lplan_search(LSearch &S, int m, int d, int mx, int sum) {
    if (m == 1) {
        if (d < 2 || S.cur[d - 1] > S.last) return;
        const bool better = S.np == 0 || d < S.np || (d == S.np && mx < S.mx) ||
                            (d == S.np && mx == S.mx && sum < S.sum);
        if (!better) return;
        S.np = d;
        S.mx = mx;
        S.sum = sum;
        for (int i = 0; i < d; ++i) S.best[i] = S.cur[i];
        return;
    }
    if (d == kLMaxPass) return;
    const int radices[] = {13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    for (int r : radices) {
        if (m % r != 0 || (d > 0 && r > S.cur[d - 1])) continue;
        S.cur[d] = r;
        lplan_search(S, m / r, d + 1, d == 0 ? r : mx, sum + r);
    }
}
// Fewest passes, then the smallest largest radix, then the smallest sum; the
// radices fall.  The last is at most 10 where such a plan exists.
__host__ __device__ constexpr LPlan lplan(int n) {
    LPlan p{};
    p.n = n;
    LSearch S{};
    for (int last : {10, 13}) {
        if (S.np) break;
        S.last = last;
        lplan_search(S, n, 0, 0, 0);
    }
    p.np = S.np;
    int s = n;
    for (int i = 0; i < S.np; ++i) {
        p.R[i] = S.best[i];
        s /= p.R[i];
        p.s[i] = s;
        p.tw[i] = p.ntw;
        if (i + 1 < S.np) p.ntw += (p.R[i] - 1) * s;
    }
    return p;
}

// Mask of the element swizzle (hqt_line.cuh): along x 8 elements fill 128 bytes;
// along y 128 bytes hold this many elements of 2^nbl lines.  0 where a line has no
// groups of 8.  (FP64)
__host__ __device__ constexpr int lswz(int n, int nbl, bool along_x) {
    return n % 8 != 0 ? 0 : along_x ? 7 : nbl < 3 ? (8 >> nbl) - 1 : 0;
}
// Threads of a block with 2^nbl lines: one radix-8 butterfly each.
__host__ __device__ constexpr int lthreads(int n, int nbl) {
    const int t = (((n << nbl) / 8 + 31) / 32) * 32;
    return t < 32 ? 32 : (t > kLThreads ? kLThreads : t);
}

// ... with a runtime plan, whose n / R butterflies seldom fill whole rounds of the
// threads: the multiple of 32 with the least time per block and share of the SM (128
// registers a thread, nbuf buffers a block), where a round of radix R counts R + 4.
// From 96 on, or the count above: with smaller blocks the many of them crowd the L1
// out (384x384x15, filter_x_fwd 100, 72, 86, 85 us with 64, 96, 128, 192 threads).
// The choice is within 5% of the best of a sweep of 64..512 for the passes of 384,
// 250x180, 600, 1001, 96x100; 192 or 512 threads for all, as the rule above has it,
// cost up to a third more (1001x1001x10, filter_x_inv 338 us by this rule, 452
// by that).
inline int lthreads_rt(const LPlan &p, int nbl, int nbuf) {
    const int lo = lthreads(p.n, nbl) < 96 ? lthreads(p.n, nbl) : 96;
    int best = lo;
    double least = 0;
    for (int t = lo; t <= kLThreads; t += 32) {
        const int fit = (int)(227 * 1024ll / ((16ll * p.n * nbuf << nbl) + 1024));
        int blocks = kLThreads / t < fit ? kLThreads / t : fit;
        double time = 0;
        for (int i = 0; i < p.np; ++i) {
            const int cnt = (p.n / p.R[i]) << nbl;
            const int one = (cnt + t - 1) / t, all = (cnt * nbuf + t - 1) / t;
            time += (one + (i + 1 < p.np ? all : nbuf * one)) * (p.R[i] + 4.0);
        }
        time /= blocks < 1 ? 1 : blocks;
        if (least == 0 || time < least) {
            least = time;
            best = t;
        }
    }
    return best;
}

// Compile-time geometry: N points, 2^NBL lines per block.
// The passes with one buffer (One) take blocks of at most 256 threads: with 512, a
// block of 1024-point y lines was the only one on its SM (1024x1024x33: filter y 1247
// -> 1060, y_d1 320 -> 300 us; 1024x1024x17: 647 -> 557, 223 -> 178 us).
template <int N_, int NBL_, int MAXT = kLThreads> struct SGeo;
// Runtime geometry, a kernel argument.
struct RGeo {
    using One = RGeo;
    static constexpr bool kStatic = false;
    static constexpr int kN = 0;
    static constexpr int kMaxThreads = kLThreads;
    int n_, nbl_, np_, swz_;
    int th_[2];    // threads of a block with one and two buffers
    unsigned mn_;  // ceil(2^32 / n)
    int R_[kLMaxPass], s_[kLMaxPass], tw_[kLMaxPass];
    unsigned mg_[kLMaxPass], mr_[kLMaxPass];  // ceil(2^32 / s), ceil(2^32 / (n / R))
    __host__ __device__ __forceinline__ int n() const { return n_; }
    __host__ __device__ __forceinline__ int nbl() const { return nbl_; }
    __host__ __device__ __forceinline__ int np() const { return np_; }
    int block(int nbuf) const { return th_[nbuf - 1]; }
    template <typename T, bool AX> __host__ __device__ __forceinline__ int swz() const {
        return swz_;
    }
    __host__ __device__ __forceinline__ unsigned mn() const { return mn_; }
    __host__ __device__ __forceinline__ unsigned mr(int p) const { return mr_[p]; }
    __host__ __device__ __forceinline__ int R(int p) const { return R_[p]; }
    __host__ __device__ __forceinline__ int s(int p) const { return s_[p]; }
    __host__ __device__ __forceinline__ int tw(int p) const { return tw_[p]; }
    __host__ __device__ __forceinline__ unsigned mg(int p) const { return mg_[p]; }
};
template <int N_, int NBL_, int MAXT> struct SGeo {
    static constexpr bool kStatic = true;
    static constexpr int N = N_, kN = N_, NBL = NBL_;
    static constexpr int kMaxThreads = lthreads(N_, NBL_) < MAXT ? lthreads(N_, NBL_) : MAXT;
    using One = SGeo<N_, NBL_, 256>;
    static_assert(lplan(N_).np >= 2, "no in-place plan for this length");
    __host__ __device__ static constexpr int np() { return lplan(N_).np; }
    __host__ __device__ SGeo(const RGeo &) {}
    __host__ __device__ static constexpr int n() { return N_; }
    __host__ __device__ static constexpr int nbl() { return NBL_; }
    static constexpr int block(int) { return kMaxThreads; }
    __host__ __device__ static constexpr int threads() { return kMaxThreads; }
    template <typename T, bool AX> __host__ __device__ static constexpr int swz() {
        return lswz(N_, NBL_, AX);
    }
    __host__ __device__ static constexpr unsigned mn() { return 0u; }
};

// Device tables of one axis and the runtime plan.
template <typename T> struct LineTab {
    const C2<T> *tw;
    const int *freq;  // [n / R_last]: lowest mode of the last pass's butterfly
    const int *pos;   // [n]: row of mode k
    RGeo g;
};

// log2 of the lines per block.  Two buffers of the block's lines stay within 66 KB (two
// or three blocks per SM, as the threads' registers allow); y lines are adjacent columns,
// of which 8 fill a 128-byte row, and take up to 130 KB for 4 of them (one block from 900 points on).
__host__ __device__ constexpr int lnbl(int n, bool along_y) {
    int b = along_y ? 3 : 2;
    while (b > 0 && (n * 32ll << b) > (along_y && b <= 2 ? 130 : 66) * 1024ll) --b;
    return b;
}

// Runtime geometry of a plan; `half`: half the lines per block.
inline RGeo rgeo(const LPlan &p, bool along_y, bool half) {
    RGeo g{};
    int nbl = lnbl(p.n, along_y);
    if (half && nbl > 0) --nbl;
    g.n_ = p.n;
    g.nbl_ = nbl;
    g.np_ = p.np;
    for (int i = 0; i < 2; ++i) g.th_[i] = lthreads_rt(p, nbl, i + 1);
    g.swz_ = lswz(p.n, nbl, !along_y);
    auto magic = [](int d) { return (unsigned)(((1ull << 32) + d - 1) / d); };
    g.mn_ = magic(p.n);
    for (int i = 0; i < p.np; ++i) {
        g.R_[i] = p.R[i];
        g.s_[i] = p.s[i];
        g.tw_[i] = p.tw[i];
        g.mg_[i] = magic(p.s[i]);
        g.mr_[i] = magic(p.n / p.R[i]);
    }
    return g;
}

}  // namespace hqt
