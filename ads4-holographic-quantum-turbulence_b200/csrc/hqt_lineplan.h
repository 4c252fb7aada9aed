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

// Row swizzle mask (hqt_line.cuh): 128 bytes hold this many rows of 2^nbl
// elements; 0 where rows have no groups of 8.
__host__ __device__ constexpr int lswz(int n, int nbl, int esize) {
    const int rows = (128 / esize) >> nbl;
    return n % 8 == 0 && rows > 1 ? (rows > 8 ? 7 : rows - 1) : 0;
}
// Threads of a block with 2^nbl lines: one radix-8 butterfly each.
__host__ __device__ constexpr int lthreads(int n, int nbl) {
    const int t = (((n << nbl) / 8 + 31) / 32) * 32;
    return t < 32 ? 32 : (t > kLThreads ? kLThreads : t);
}

// Compile-time geometry: N points, 2^NBL lines per block.
template <int N_, int NBL_> struct SGeo;
// Runtime geometry, a kernel argument.
struct RGeo {
    static constexpr bool kStatic = false;
    static constexpr int kMaxThreads = kLThreads;
    int n_, nbl_, np_, th_, swz_;
    int R_[kLMaxPass], s_[kLMaxPass], tw_[kLMaxPass];
    unsigned mg_[kLMaxPass];  // ceil(2^32 / s)
    __host__ __device__ __forceinline__ int n() const { return n_; }
    __host__ __device__ __forceinline__ int nbl() const { return nbl_; }
    __host__ __device__ __forceinline__ int np() const { return np_; }
    __host__ __device__ __forceinline__ int threads() const { return th_; }
    template <typename T> __host__ __device__ __forceinline__ int swz() const { return swz_; }
    __host__ __device__ __forceinline__ int R(int p) const { return R_[p]; }
    __host__ __device__ __forceinline__ int s(int p) const { return s_[p]; }
    __host__ __device__ __forceinline__ int tw(int p) const { return tw_[p]; }
    __host__ __device__ __forceinline__ unsigned mg(int p) const { return mg_[p]; }
};
template <int N_, int NBL_> struct SGeo {
    static constexpr bool kStatic = true;
    static constexpr int N = N_, NBL = NBL_, kMaxThreads = lthreads(N_, NBL_);
    static_assert(lplan(N_).np >= 2, "no in-place plan for this length");
    __host__ __device__ static constexpr int np() { return lplan(N_).np; }
    __host__ __device__ SGeo(const RGeo &) {}
    __host__ __device__ static constexpr int n() { return N_; }
    __host__ __device__ static constexpr int nbl() { return NBL_; }
    __host__ __device__ static constexpr int threads() { return lthreads(N_, NBL_); }
    template <typename T> __host__ __device__ static constexpr int swz() {
        return lswz(N_, NBL_, 2 * (int)sizeof(T));
    }
};

// Device tables of one axis and the runtime plan.
template <typename T> struct LineTab {
    const C2<T> *tw;
    const int *freq;  // [n / R_last]: lowest mode of the last pass's butterfly
    const int *pos;   // [n]: row of mode k
    RGeo g;
};

// log2 of the lines per block.  x lines are contiguous, so 4 lines give a
// warp 128-byte runs; y lines are adjacent columns, of which 8 fill a 128-byte
// row.  Two buffers of the block's lines stay within about 64 KB (three
// blocks per SM); for y lines above HQT_YBIG points four columns (64-byte
// rows) in up to 128 KB.
#ifndef HQT_YBUD
#define HQT_YBUD 130
#endif
__host__ __device__ constexpr int lnbl(int n, bool along_y) {
    int b = along_y ? 3 : 2;
    while (b > 0 && (n * 32ll << b) > (along_y && b == 2 ? HQT_YBUD : 66) * 1024ll) --b;
    return b;
}

}  // namespace hqt
