// hqt_line.cuh -- in-place mixed-radix line transforms: forward decimation in
// frequency, inverse decimation in time, on NB lines held in shared memory.
//
// The passes of a line of n = R0 R1 .. R(m-1) points work on blocks of
// L_p = n/(R0..R(p-1)) elements with stride s_p = L_p/R_p: butterfly (blk, j)
// takes elements blk L_p + j + r s_p (r < R_p), transforms over r in
// registers, multiplies by w_{L_p}^{j k} and writes back where it read.  The
// spectrum is left in digit-reversed order; the inverse runs the same
// butterflies backwards with conjugate twiddles and ends in natural order, so
// nothing is ever reordered.  What follows from that, against a ping-pong
// (Stockham) transform:
//   - the first pass reads global memory into registers and the last inverse
//     pass writes global memory from registers: no staging passes;
//   - the last forward pass, the multiplier of a derivative (or the filter's
//     weight) and the first inverse pass are one pass: a thread holds the
//     spectrum of its butterfly and writes one product per derivative;
//   - one buffer per line and derivative instead of three, no twiddle table
//     in shared memory, a barrier per pass.
// A first and a second derivative of a three-pass line move 12 line lengths
// through shared memory (25 in the Stockham form): W | RW | R WW | RW RW | R R.
// Twiddles come from a table packed per pass as [k][j], so that consecutive
// butterflies read consecutive entries (through L1).
//
// Threads and shared memory.  x lines: threads run along a line, element e of line
// b at b n + e, so a quarter warp's global access is one 128-byte run.  (With
// threads running over the lines first it touched a 128-byte line per line of
// the block: 17 of 57 wavefronts of the L1 data pipe, which bounds these passes,
// at 512x512x25.)  y lines: threads run over the adjacent columns first, element
// e of line b at (e << nbl) + b.  In both, an XOR of e's low bits where n is a
// multiple of 8: the strided rows of the last forward pass otherwise fall on the
// same banks.
//
// The plan is a compile-time constant (SGeo) for the lengths of HQT_LN_LIST
// and a kernel argument (RGeo, divisions by multiply-high) for every other
// length whose prime factors are at most 13.
#pragma once
#include <type_traits>

#include "hqt_args.h"
#include "hqt_dev.cuh"

namespace hqt {

// cos(2 pi k / R) of the radices' real-pair forms, to 20 digits (folded to immediates
// once k is known).
__host__ __device__ constexpr double lf_cos(int R, int k) {
    switch (32 * R + k) {
        case 97: return -0.5;
        case 98: return -0.5;
        case 161: return 0.3090169943749474241;
        case 162: return -0.8090169943749474241;
        case 163: return -0.8090169943749474241;
        case 164: return 0.3090169943749474241;
        case 225: return 0.62348980185873353053;
        case 226: return -0.22252093395631440429;
        case 227: return -0.90096886790241912624;
        case 228: return -0.90096886790241912624;
        case 229: return -0.22252093395631440429;
        case 230: return 0.62348980185873353053;
        case 289: return 0.7660444431189780352;
        case 290: return 0.17364817766693034885;
        case 291: return -0.5;
        case 292: return -0.93969262078590838405;
        case 293: return -0.93969262078590838405;
        case 294: return -0.5;
        case 295: return 0.17364817766693034885;
        case 296: return 0.7660444431189780352;
        case 353: return 0.84125353283118116886;
        case 354: return 0.41541501300188642553;
        case 355: return -0.14231483827328514044;
        case 356: return -0.65486073394528506406;
        case 357: return -0.95949297361449738989;
        case 358: return -0.95949297361449738989;
        case 359: return -0.65486073394528506406;
        case 360: return -0.14231483827328514044;
        case 361: return 0.41541501300188642553;
        case 362: return 0.84125353283118116886;
        case 417: return 0.8854560256532098959;
        case 418: return 0.56806474673115580251;
        case 419: return 0.12053668025532305335;
        case 420: return -0.35460488704253562597;
        case 421: return -0.74851074817110109863;
        case 422: return -0.97094181742605202716;
        case 423: return -0.97094181742605202716;
        case 424: return -0.74851074817110109863;
        case 425: return -0.35460488704253562597;
        case 426: return 0.12053668025532305335;
        case 427: return 0.56806474673115580251;
        case 428: return 0.8854560256532098959;
        default: return 1.0;
    }
}
__host__ __device__ constexpr double lf_sin(int R, int k) {
    switch (32 * R + k) {
        case 97: return 0.86602540378443864676;
        case 98: return -0.86602540378443864676;
        case 161: return 0.95105651629515357212;
        case 162: return 0.58778525229247312917;
        case 163: return -0.58778525229247312917;
        case 164: return -0.95105651629515357212;
        case 225: return 0.78183148246802980871;
        case 226: return 0.97492791218182360702;
        case 227: return 0.43388373911755812048;
        case 228: return -0.43388373911755812048;
        case 229: return -0.97492791218182360702;
        case 230: return -0.78183148246802980871;
        case 289: return 0.64278760968653932632;
        case 290: return 0.98480775301220805937;
        case 291: return 0.86602540378443864676;
        case 292: return 0.34202014332566873304;
        case 293: return -0.34202014332566873304;
        case 294: return -0.86602540378443864676;
        case 295: return -0.98480775301220805937;
        case 296: return -0.64278760968653932632;
        case 353: return 0.54064081745559758211;
        case 354: return 0.90963199535451837141;
        case 355: return 0.98982144188093273238;
        case 356: return 0.75574957435425828377;
        case 357: return 0.28173255684142969771;
        case 358: return -0.28173255684142969771;
        case 359: return -0.75574957435425828377;
        case 360: return -0.98982144188093273238;
        case 361: return -0.90963199535451837141;
        case 362: return -0.54064081745559758211;
        case 417: return 0.46472317204376854566;
        case 418: return 0.82298386589365639458;
        case 419: return 0.9927088740980539928;
        case 420: return 0.93501624268541482344;
        case 421: return 0.66312265824079520238;
        case 422: return 0.23931566428755776715;
        case 423: return -0.23931566428755776715;
        case 424: return -0.66312265824079520238;
        case 425: return -0.93501624268541482344;
        case 426: return -0.9927088740980539928;
        case 427: return -0.82298386589365639458;
        case 428: return -0.46472317204376854566;
        default: return 0.0;
    }
}

template <typename T> __device__ __forceinline__ C2<T> lf_cmul(C2<T> a, C2<T> w) {
    return mk2<T>(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
template <typename T> __device__ __forceinline__ C2<T> lf_cmulc(C2<T> a, C2<T> w) {  // a conj(w)
    return mk2<T>(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y);
}

// ---- R-point DFTs in registers, natural order in and out ------------------
template <typename T, int R, int SIGN> struct LDft;
template <typename T, int R, int SIGN> __device__ __forceinline__ void ldft(C2<T> (&v)[R]) {
    LDft<T, R, SIGN>::run(v);
}
// a * e^{SIGN 2 pi i k/R}
template <typename T, int R, int SIGN> __device__ __forceinline__ C2<T> lrot(C2<T> a, int k) {
    const T c = (T)lf_cos(R, k), s = (T)(SIGN * lf_sin(R, k));
    return mk2<T>(a.x * c - a.y * s, a.x * s + a.y * c);
}
template <typename T, int SIGN> __device__ __forceinline__ C2<T> lmuli(C2<T> a) {  // SIGN i a
    return SIGN < 0 ? mk2<T>(a.y, -a.x) : mk2<T>(-a.y, a.x);
}

template <typename T, int SIGN> struct LDft<T, 2, SIGN> {
    static __device__ __forceinline__ void run(C2<T> (&v)[2]) {
        const C2<T> a = v[0], b = v[1];
        v[0] = a + b;
        v[1] = a - b;
    }
};
template <typename T, int SIGN> struct LDft<T, 4, SIGN> {
    static __device__ __forceinline__ void run(C2<T> (&v)[4]) {
        const C2<T> a = v[0] + v[2], b = v[0] - v[2], c = v[1] + v[3];
        const C2<T> d = lmuli<T, SIGN>(v[1] - v[3]);
        v[0] = a + c;
        v[1] = b + d;
        v[2] = a - c;
        v[3] = b - d;
    }
};
// two 4-point DFTs of the even and odd elements; the turns by +-(1 + SIGN i)/sqrt(2)
// are two adds and two products
template <typename T, int SIGN> struct LDft<T, 8, SIGN> {
    static __device__ __forceinline__ void run(C2<T> (&v)[8]) {
        C2<T> e[4], o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            e[i] = v[2 * i];
            o[i] = v[2 * i + 1];
        }
        ldft<T, 4, SIGN>(e);
        ldft<T, 4, SIGN>(o);
        const T h = (T)0.70710678118654752440;
        const C2<T> q1 = lmuli<T, SIGN>(o[1]), q3 = lmuli<T, SIGN>(o[3]);
        const C2<T> t[4] = {o[0], mk2<T>(h * (o[1].x + q1.x), h * (o[1].y + q1.y)),
                            lmuli<T, SIGN>(o[2]), mk2<T>(h * (q3.x - o[3].x), h * (q3.y - o[3].y))};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = e[k] + t[k];
            v[k + 4] = e[k] - t[k];
        }
    }
};
// odd prime R in the real-pair form: a_j = x_j + x_{R-j}, b_j = x_j - x_{R-j}
template <typename T, int R, int SIGN> struct LDftOdd {
    static __device__ __forceinline__ void run(C2<T> (&v)[R]) {
        constexpr int M = (R - 1) / 2;
        C2<T> a[M + 1], b[M + 1];
#pragma unroll
        for (int j = 1; j <= M; ++j) {
            a[j] = v[j] + v[R - j];
            b[j] = v[j] - v[R - j];
        }
        const C2<T> x0 = v[0];
#pragma unroll
        for (int j = 1; j <= M; ++j) v[0] = v[0] + a[j];
#pragma unroll
        for (int k = 1; k <= M; ++k) {
            C2<T> p = x0, q = mk2<T>(T(0), T(0));
#pragma unroll
            for (int j = 1; j <= M; ++j) {
                const T c = (T)lf_cos(R, (j * k) % R), s = (T)lf_sin(R, (j * k) % R);
                p = mk2<T>(fma(a[j].x, c, p.x), fma(a[j].y, c, p.y));
                q = mk2<T>(fma(b[j].x, s, q.x), fma(b[j].y, s, q.y));
            }
            q = lmuli<T, SIGN>(q);
            v[k] = p + q;
            v[R - k] = p - q;
        }
    }
};
template <typename T, int SIGN> struct LDft<T, 3, SIGN> : LDftOdd<T, 3, SIGN> {};
template <typename T, int SIGN> struct LDft<T, 5, SIGN> : LDftOdd<T, 5, SIGN> {};
template <typename T, int SIGN> struct LDft<T, 7, SIGN> : LDftOdd<T, 7, SIGN> {};
template <typename T, int SIGN> struct LDft<T, 11, SIGN> : LDftOdd<T, 11, SIGN> {};
template <typename T, int SIGN> struct LDft<T, 13, SIGN> : LDftOdd<T, 13, SIGN> {};
template <typename T, int SIGN> struct LDft<T, 9, SIGN> {
    static __device__ __forceinline__ void run(C2<T> (&v)[9]) {
        C2<T> u[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            C2<T> w[3] = {v[i], v[i + 3], v[i + 6]};
            ldft<T, 3, SIGN>(w);
#pragma unroll
            for (int k = 0; k < 3; ++k) u[k][i] = i * k == 0 ? w[k] : lrot<T, 9, SIGN>(w[k], i * k);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            ldft<T, 3, SIGN>(u[k]);
#pragma unroll
            for (int m = 0; m < 3; ++m) v[k + 3 * m] = u[k][m];
        }
    }
};
__host__ __device__ constexpr int lf_modinv(int a, int m) {
    for (int x = 1; x < m; ++x)
        if ((a * x) % m == 1) return x;
    return 1;
}
// R = P Q with gcd(P, Q) = 1: P- and Q-point DFTs without twiddles
template <typename T, int P, int Q, int SIGN> struct LDftPrimeFactor {
    static __device__ __forceinline__ void run(C2<T> (&v)[P * Q]) {
        constexpr int R = P * Q, QI = lf_modinv(Q % P, P), PI = lf_modinv(P % Q, Q);
        C2<T> u[P][Q];
#pragma unroll
        for (int a = 0; a < P; ++a) {
#pragma unroll
            for (int b = 0; b < Q; ++b) u[a][b] = v[(Q * a + P * b) % R];
            ldft<T, Q, SIGN>(u[a]);
        }
#pragma unroll
        for (int b = 0; b < Q; ++b) {
            C2<T> w[P];
#pragma unroll
            for (int a = 0; a < P; ++a) w[a] = u[a][b];
            ldft<T, P, SIGN>(w);
#pragma unroll
            for (int a = 0; a < P; ++a) v[(Q * QI * a + P * PI * b) % R] = w[a];
        }
    }
};
template <typename T, int SIGN> struct LDft<T, 6, SIGN> : LDftPrimeFactor<T, 2, 3, SIGN> {};
template <typename T, int SIGN> struct LDft<T, 10, SIGN> : LDftPrimeFactor<T, 2, 5, SIGN> {};
template <typename T, int SIGN> struct LDft<T, 12, SIGN> : LDftPrimeFactor<T, 4, 3, SIGN> {};

// ---- the transform --------------------------------------------------------
// The threads of a block work on its lines; A and B are its two buffers.  AX: lines
// along x.
template <typename T, class G, bool AX> struct LineEng {
    using C = C2<T>;
    // a runtime plan stays in the kernel's parameters (its dynamic indexing
    // would put a copy on the stack)
    std::conditional_t<G::kStatic, G, const RGeo &> g;
    C *A, *B;
    const C *tw;
    const int *freq, *posn;  // RGeo only: digit reversal of blocks and modes

    __device__ __forceinline__ LineEng(const LineTab<T> &t)
        : g(t.g), A(sptr<T>(0)), B(sptr<T>(0) + (g.n() << g.nbl())), tw(t.tw), freq(t.freq),
          posn(t.pos) {}

    __device__ __forceinline__ int threads() const {
        if constexpr (G::kStatic)
            return G::threads();
        else
            return blockDim.x;
    }
    // element e of line b, its low bits swizzled inside the group of 8
    __device__ __forceinline__ int at(int b, int e) const {
        const int m = g.template swz<T, AX>();
        if (!G::kStatic || m != 0) e ^= ((e >> 3) ^ (e >> 6) ^ (e >> 9)) & m;
        return AX ? b * g.n() + e : (e << g.nbl()) + b;
    }
    __device__ __forceinline__ static int div(unsigned x, int s, unsigned mg) {
        if constexpr (G::kStatic) return (int)x / s;
        return s == 1 ? (int)x : (int)__umulhi(x, mg);
    }
    // f(b, jj) for every butterfly jj < n/R of every line b (mr: the magic of n/R)
    template <int R, typename F> __device__ __forceinline__ void each(unsigned mr, F f) const {
        const int nr = g.n() / R, cnt = nr << g.nbl();
#pragma unroll 1
        for (int t = threadIdx.x; t < cnt; t += threads()) {
            if constexpr (AX) {
                const int b = div(t, nr, mr);
                f(b, t - b * nr);
            } else {
                f(t & ((1 << g.nbl()) - 1), t >> g.nbl());
            }
        }
    }
    // f(integral_constant<int, R>, stride s, magics of s and n/R, twiddle offset) of
    // pass p
    template <int P, typename F> __device__ __forceinline__ void at_static(F f) const {
        constexpr LPlan pl = lplan(G::N);
        constexpr int R = pl.R[P], s = pl.s[P], o = pl.tw[P];
        f(std::integral_constant<int, R>{}, s, 0u, 0u, o);
    }
    template <typename F> __device__ __forceinline__ void at(int p, F f) const {
        const int s = g.s(p), o = g.tw(p);
        const unsigned mg = g.mg(p), mr = g.mr(p);
        switch (g.R(p)) {
#define HQT_LR(RR) \
    case RR: f(std::integral_constant<int, RR>{}, s, mg, mr, o); break;
            HQT_LR(2) HQT_LR(3) HQT_LR(4) HQT_LR(5) HQT_LR(6) HQT_LR(7) HQT_LR(8) HQT_LR(9)
            HQT_LR(10) HQT_LR(11) HQT_LR(12) HQT_LR(13)
#undef HQT_LR
        }
    }
    // pass `P` of the plan: first, last or any of the ones between
    template <typename F> __device__ __forceinline__ void at_first(F f) const {
        if constexpr (G::kStatic)
            at_static<0>(f);
        else
            at(0, f);
    }
    template <typename F> __device__ __forceinline__ void at_last(F f) const {
        if constexpr (G::kStatic)
            at_static<G::np() - 1>(f);
        else
            at(g.np() - 1, f);
    }
    // the passes between, in order (+1) or backwards (-1), a barrier after each
    template <int DIR, int P = 1, typename F> __device__ __forceinline__ void at_mid(F f) const {
        if constexpr (G::kStatic) {
            if constexpr (P < G::np() - 1) {
                at_static<(DIR > 0 ? P : G::np() - 1 - P)>(f);
                __syncthreads();
                at_mid<DIR, P + 1>(f);
            }
        } else {
            const int np = g.np();
#pragma unroll 1
            for (int i = 1; i < np - 1; ++i) {
                at(DIR > 0 ? i : np - 1 - i, f);
                __syncthreads();
            }
        }
    }

    // f(x, b, jj) for every butterfly of A (x = 0) and, if `two`, of B (x = 1).  For
    // runtime plans: their counts leave a part of the block's threads idle, and their
    // larger radices spill with twiddles held for both buffers (y_rhs 1.54 -> 1.75 ms
    // at 1001x1001x20).  A compile-time plan takes A and B in one iteration with the
    // twiddles in registers.
    template <int R, typename F>
    __device__ __forceinline__ void each_of(bool two, unsigned mr, F f) const {
        const int nr = g.n() / R, cnt = nr << g.nbl();
#pragma unroll 1
        for (int t = threadIdx.x; t < (two ? 2 * cnt : cnt); t += threads()) {
            const bool x = t >= cnt;
            const int u = x ? t - cnt : t;
            if constexpr (AX) {
                const int b = div(u, nr, mr);
                f(x, b, u - b * nr);
            } else {
                f(x, u & ((1 << g.nbl()) - 1), u >> g.nbl());
            }
        }
    }
    // twiddles of a butterfly: held in registers, or (runtime plan) loaded at use
    template <int R> struct Twiddles {
        const C *p;
        int s;
        C w[G::kStatic ? R : 1];
        __device__ __forceinline__ Twiddles(const C *p_, int s_) : p(p_), s(s_) {
            if constexpr (G::kStatic) {
#pragma unroll
                for (int r = 1; r < R; ++r) w[r] = __ldg(p + (r - 1) * s);
            }
        }
        __device__ __forceinline__ C operator()(int r) const {
            if constexpr (G::kStatic)
                return w[r];
            else
                return __ldg(p + (r - 1) * s);
        }
    };
    // one butterfly in place at rows e0 + r s
    template <int R, int SIGN>
    __device__ __forceinline__ void fly(C *X, int b, int e0, int s, const Twiddles<R> &w) const {
        C v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = X[at(b, e0 + r * s)];
        if (SIGN > 0) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = lf_cmulc<T>(v[r], w(r));
        }
        ldft<T, R, SIGN>(v);
        if (SIGN < 0) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = lf_cmul<T>(v[r], w(r));
        }
#pragma unroll
        for (int r = 0; r < R; ++r) X[at(b, e0 + r * s)] = v[r];
    }
    // butterflies of one pass in place, of A or (two) of A and B: forward or inverse
    template <int R, int SIGN>
    __device__ __forceinline__ void step(bool two, int s, unsigned mg, unsigned mr, int o) const {
        if constexpr (G::kStatic) {
            each<R>(mr, [&](int b, int jj) {
                const int blk = div(jj, s, mg), j = jj - blk * s;
                const Twiddles<R> w(tw + o + j, s);
#pragma unroll 1
                for (int x = 0; x < (two ? 2 : 1); ++x)
                    fly<R, SIGN>(x ? B : A, b, blk * s * R + j, s, w);
            });
        } else {
            each_of<R>(two, mr, [&](bool x, int b, int jj) {
                const int blk = div(jj, s, mg), j = jj - blk * s;
                fly<R, SIGN>(x ? B : A, b, blk * s * R + j, s, Twiddles<R>(tw + o + j, s));
            });
        }
    }
    // last inverse pass of one butterfly: row j of the plan's first stride s
    template <int R>
    __device__ __forceinline__ void fly_last(const C *X, int b, int j, int s, C (&v)[R],
                                             const Twiddles<R> &w) const {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = X[at(b, j + r * s)];
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = lf_cmulc<T>(v[r], w(r));
        ldft<T, R, 1>(v);
    }
    template <int R, typename Get, typename Sa>
    __device__ __forceinline__ void last_a(int b, int j, int s, const Twiddles<R> &w, Get get,
                                           Sa sa) const {
        constexpr int H = R > 8 ? 4 : R;
        C v[R];
        fly_last<R>(A, b, j, s, v, w);
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += H) {
            decltype(get(0, 0)) x[H];
#pragma unroll
            for (int r = 0; r < H; ++r)
                if (r0 + r < R) x[r] = get(b, j + (r0 + r) * s);
#pragma unroll
            for (int r = 0; r < H; ++r)
                if (r0 + r < R) sa(b, j + (r0 + r) * s, v[r0 + r], x[r]);
        }
    }
    template <int R, typename Sb>
    __device__ __forceinline__ void last_b(int b, int j, int s, const Twiddles<R> &w, Sb sb) const {
        C v[R];
        fly_last<R>(B, b, j, s, v, w);
#pragma unroll
        for (int r = 0; r < R; ++r) sb(b, j + r * s, v[r]);
    }

    // first forward pass from ld(b, e) into X
    template <typename Ld> __device__ __forceinline__ void first(C *X, Ld ld) const {
        first(X, false, [](int) { return mk2<T>(T(1), T(0)); }, ld);
    }
    // ... for a derivative: where the plan has an odd radix, of the line less its
    // first element.  A constant drops out anyway, but an odd radix rounds it into
    // every mode: div A of a nearly uniform flow at 180x180x12 was 4 times less exact
    // than with radices 2, 3 and 5 one by one.  (Powers of two: differences of equal
    // values are exact.)
    static constexpr bool kLevel = !G::kStatic || (G::kN & (G::kN - 1)) != 0;
    template <typename Ld> __device__ __forceinline__ void first_d(C *X, Ld ld) const {
        at_first([&](auto rc, int s, unsigned, unsigned mr, int o) {
            constexpr int R = decltype(rc)::value;
            each<R>(mr, [&](int b, int j) { first_d_fly<R>(X, b, j, s, o, ld); });
        });
    }
    // ... of A and B, by the threads that read them in last2.  (With a barrier ahead of a
    // first_d(B, ..) instead, y_rhs by a runtime plan took 1611 us at 1001x1001x20 and 79.8
    // at 250x180x20; so 1440 and 77.4.)
    template <typename LdA, typename LdB>
    __device__ __forceinline__ void first_d2(LdA lda, LdB ldb) const {
        if constexpr (G::kStatic) {
            first_d(A, lda);
            first_d(B, ldb);
        } else {
            at_first([&](auto rc, int s, unsigned, unsigned mr, int o) {
                constexpr int R = decltype(rc)::value;
                each_of<R>(true, mr, [&](bool x, int b, int j) {
                    if (x)
                        first_d_fly<R>(B, b, j, s, o, ldb);
                    else
                        first_d_fly<R>(A, b, j, s, o, lda);
                });
            });
        }
    }
    template <int R, typename Ld>
    __device__ __forceinline__ void first_d_fly(C *X, int b, int j, int s, int o, Ld ld) const {
        C v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = ld(b, j + r * s);
        if (kLevel) {
            const C x0 = ld(b, 0);
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = v[r] - x0;
        }
        first_fly<R>(X, b, j, s, o, v);
    }
    template <int R>
    __device__ __forceinline__ void first_fly(C *X, int b, int j, int s, int o, C (&v)[R]) const {
        ldft<T, R, -1>(v);
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = lf_cmul<T>(v[r], __ldg(tw + o + (r - 1) * s + j));
#pragma unroll
        for (int r = 0; r < R; ++r) X[at(b, j + r * s)] = v[r];
    }
    // ... times ph(b) if `turn`
    template <typename Ph, typename Ld>
    __device__ __forceinline__ void first(C *X, bool turn, Ph ph, Ld ld) const {
        at_first([&](auto rc, int s, unsigned, unsigned mr, int o) {
            constexpr int R = decltype(rc)::value;
            each<R>(mr, [&](int b, int j) {
                C v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = ld(b, j + r * s);
                if (turn) {
                    const C p = ph(b);
#pragma unroll
                    for (int r = 0; r < R; ++r) v[r] = lf_cmul<T>(v[r], p);
                }
                first_fly<R>(X, b, j, s, o, v);
            });
        });
    }
    // middle passes of A, or of A and B; starts and ends at a barrier
    __device__ __forceinline__ void forward_mid(bool two) const {
        __syncthreads();
        at_mid<1>([&](auto rc, int s, unsigned mg, unsigned mr, int o) {
            step<decltype(rc)::value, -1>(two, s, mg, mr, o);
        });
    }
    __device__ __forceinline__ void inverse_mid(bool two) const {
        __syncthreads();
        at_mid<-1>([&](auto rc, int s, unsigned mg, unsigned mr, int o) {
            step<decltype(rc)::value, 1>(two, s, mg, mr, o);
        });
    }
    template <int P> __device__ __forceinline__ static int mode0_static(int rem, int mult) {
        constexpr LPlan pl = lplan(G::N);
        if constexpr (P < pl.np - 1) {
            constexpr int w = pl.s[P] / pl.R[pl.np - 1], R = pl.R[P];
            return (rem / w) * mult + mode0_static<P + 1>(rem % w, mult * R);
        }
        return 0;
    }
    template <int P> __device__ __forceinline__ static int pos_static(int k) {
        constexpr LPlan pl = lplan(G::N);
        if constexpr (P < pl.np) {
            constexpr int R = pl.R[P], s = pl.s[P];
            return (k % R) * s + pos_static<P + 1>(k / R);
        }
        return 0;
    }
    // mode number of output km of the last pass's butterfly blk: base + km n/R
    __device__ __forceinline__ int mode0(int blk) const {
        if constexpr (G::kStatic) {
            return mode0_static<0>(blk, 1);
        } else {
            return __ldg(freq + blk);
        }
    }
    // row of mode k
    __device__ __forceinline__ int pos(int k) const {
        if constexpr (G::kStatic) {
            return pos_static<0>(k);
        } else {
            return __ldg(posn + k);
        }
    }
    __device__ __forceinline__ T wave(int k) const {  // signed, Nyquist 0
        const int k2 = 2 * k, n = g.n();
        return (T)(k2 < n ? k : (k2 > n ? k - n : 0));
    }
    // Last forward pass of X, f(v, b, k0, step) on the spectrum of a butterfly
    // (v[i] = mode k0 + i step), which writes what it wants with put().
    template <int R> __device__ __forceinline__ void put(C *X, int b, int blk, C (&v)[R]) const {
        ldft<T, R, 1>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) X[at(b, blk * R + r)] = v[r];
    }
    template <typename F> __device__ __forceinline__ void middle(const C *X, F f) const {
        at_last([&](auto rc, int, unsigned, unsigned mr, int) {
            constexpr int R = decltype(rc)::value;
            const int st = g.n() / R;
            each<R>(mr, [&](int b, int blk) {
                C v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = X[at(b, blk * R + r)];
                ldft<T, R, -1>(v);
                f(v, b, blk, mode0(blk), st);
            });
        });
    }
    // A <- d A, B <- d^2 A (spectra times i s1 k and s2 k^2), after forward_mid
    __device__ __forceinline__ void middle_deriv12(T s1, T s2) const {
        middle(A, [&](auto &v, int b, int blk, int k0, int st) {
            constexpr int R = sizeof(v) / sizeof(C);
            C u[R];
            if (R > 8) {  // two of them spill: the spectrum waits in B
#pragma unroll
                for (int i = 0; i < R; ++i) B[at(b, blk * R + i)] = v[i];
            }
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const T m = s1 * wave(k0 + i * st);
                u[i] = mk2<T>(-m * v[i].y, m * v[i].x);
            }
            put<R>(A, b, blk, u);
            if (R > 8) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = B[at(b, blk * R + i)];
            }
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const T k = wave(k0 + i * st), m = s2 * k * k;
                v[i] = mk2<T>(m * v[i].x, m * v[i].y);
            }
            put<R>(B, b, blk, v);
        });
    }
    __device__ __forceinline__ void middle_deriv1(C *X, T s1) const {
        middle(X, [&](auto &v, int b, int blk, int k0, int st) {
            constexpr int R = sizeof(v) / sizeof(C);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const T m = s1 * wave(k0 + i * st);
                v[i] = mk2<T>(-m * v[i].y, m * v[i].x);
            }
            put<R>(X, b, blk, v);
        });
    }
    // X <- (s1 k - s2 k^2) X
    __device__ __forceinline__ void middle_deriv_mix(C *X, T s1, T s2) const {
        middle(X, [&](auto &v, int b, int blk, int k0, int st) {
            constexpr int R = sizeof(v) / sizeof(C);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const T k = wave(k0 + i * st), m = s1 * k - s2 * k * k;
                v[i] = mk2<T>(m * v[i].x, m * v[i].y);
            }
            put<R>(X, b, blk, v);
        });
    }
    // last inverse pass of A: st(b, e, v) for every element
    template <typename St> __device__ __forceinline__ void last(St st) const {
        last2(false, [](int, int) { return 0; }, [&](int b, int e, C v, int) { st(b, e, v); },
              [](int, int, C) {});
    }
    // ... of A and B with the twiddles loaded once: sa(b, e, v, x) with
    // x = get(b, e), sb(b, e, v).  x is read for up to 8 elements ahead of their
    // stores (a read after a store could not move ahead of it).
    // No barrier follows: a first_d(A, ..) may come next, or first_d2, in which each
    // thread takes the butterflies of A and B that it takes here.  (Not a first_d(B, ..):
    // with a runtime plan each_of deals out B's butterflies after A's, from where it is
    // in the round of threads, and first_d from thread 0.)
    template <typename Get, typename Sa, typename Sb>
    __device__ __forceinline__ void last2(bool two, Get get, Sa sa, Sb sb) const {
        at_first([&](auto rc, int s, unsigned, unsigned mr, int o) {
            constexpr int R = decltype(rc)::value;
            if constexpr (G::kStatic) {
                each<R>(mr, [&](int b, int j) {
                    const Twiddles<R> w(tw + o + j, s);
                    last_a<R>(b, j, s, w, get, sa);
                    if (two) last_b<R>(b, j, s, w, sb);
                });
            } else {
                each_of<R>(two, mr, [&](bool x, int b, int j) {
                    const Twiddles<R> w(tw + o + j, s);
                    if (x)
                        last_b<R>(b, j, s, w, sb);
                    else
                        last_a<R>(b, j, s, w, get, sa);
                });
            }
        });
    }
    // f(b, k) over all modes of all lines
    template <typename F> __device__ __forceinline__ void modes(F f) const {
        const int n = g.n(), cnt = n << g.nbl();
#pragma unroll 4
        for (int t = threadIdx.x; t < cnt; t += threads()) {
            if constexpr (AX) {
                const int b = div(t, n, g.mn());
                f(b, t - b * n);
            } else {
                f(t & ((1 << g.nbl()) - 1), t >> g.nbl());
            }
        }
    }
    // forward, spectrum left in A by rows pos(k); starts after first(A, ..)
    __device__ __forceinline__ void forward_rest() const {
        forward_mid(false);
        middle(A, [&](auto &v, int b, int blk, int, int) {
            constexpr int R = sizeof(v) / sizeof(C);
#pragma unroll
            for (int r = 0; r < R; ++r) A[at(b, blk * R + r)] = v[r];
        });
        __syncthreads();
    }
    // inverse of a spectrum in A up to (not including) last(A, ..)
    __device__ __forceinline__ void inverse_begin() const {
        __syncthreads();
        at_last([&](auto rc, int, unsigned, unsigned mr, int) {
            constexpr int R = decltype(rc)::value;
            each<R>(mr, [&](int b, int blk) {
                C v[R];
#pragma unroll
                for (int r = 0; r < R; ++r) v[r] = A[at(b, blk * R + r)];
                put<R>(A, b, blk, v);
            });
        });
        inverse_mid(false);
    }
};

}  // namespace hqt
