// The in-place line kernels on the CPU, one block at a time: the threads of a block
// run one after the other from barrier to barrier, in the order of their numbers or
// against it.  Between two barriers no thread may depend on what another one does, so
// both orders have to leave the same bits; where a barrier is missing they do not.
//
//   order x|y <n> ...   for each length with an in-place plan: the name of every kernel
//                       whose two orders differ ("ok" where none does)
#include <cuda_runtime.h>
#include <ucontext.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

// ---- the device side of the language ----------------------------------------
#undef __noinline__
#undef __launch_bounds__
#undef __grid_constant__
#define __noinline__
#define __launch_bounds__(...)
#define __grid_constant__
static uint3 threadIdx, blockIdx;
static dim3 blockDim, gridDim;
using std::fma;
using std::max;
using std::min;
static ucontext_t g_main;
static std::vector<ucontext_t> g_ctx;
static int g_or;
static void __syncthreads() { swapcontext(&g_ctx[threadIdx.x], &g_main); }
static int __syncthreads_or(int v) {
    g_or |= v != 0;
    __syncthreads();
    return g_or;
}
template <typename T> static T __ldg(const T *p) { return *p; }
static unsigned __umulhi(unsigned a, unsigned b) {
    return (unsigned)(((unsigned long long)a * b) >> 32);
}
static void sincospi(double x, double *s, double *c) {
    *s = std::sin(M_PI * x);
    *c = std::cos(M_PI * x);
}
static void atomicMin(unsigned long long *p, unsigned long long v) { *p = min(*p, v); }
static size_t __cvta_generic_to_shared(const void *) { return 0; }
namespace hqt {
static void pdl_wait() {}
}  // namespace hqt
using std::isfinite;

#include "hqt_line_passes.cuh"
#include "hqt_ops_host.h"

namespace hqt {
alignas(16) unsigned char g_smem[256 * 1024];
}
using namespace hqt;

// ---- a block ------------------------------------------------------------------
static std::function<void()> g_body;
static std::vector<char> g_done;
static void entry() {
    g_body();
    g_done[threadIdx.x] = 1;
    swapcontext(&g_ctx[threadIdx.x], &g_main);
}
static void block(int threads, bool up) {
    constexpr size_t kStack = 256 * 1024;
    static std::vector<char> stacks((size_t)kLThreads * kStack);
    g_ctx.assign(threads, ucontext_t{});
    g_done.assign(threads, 0);
    blockDim = dim3(threads);
    for (int t = 0; t < threads; ++t) {
        getcontext(&g_ctx[t]);
        g_ctx[t].uc_stack.ss_sp = stacks.data() + (size_t)t * kStack;
        g_ctx[t].uc_stack.ss_size = kStack;
        makecontext(&g_ctx[t], entry, 0);
    }
    g_or = 0;
    for (int left = threads; left > 0;) {
        int ended = 0;
        for (int i = 0; i < threads; ++i) {
            threadIdx.x = up ? i : threads - 1 - i;
            swapcontext(&g_main, &g_ctx[threadIdx.x]);
            ended += g_done[threadIdx.x];
        }
        if (ended != 0 && ended != left) {
            std::printf("threads at different barriers\n");
            std::exit(1);
        }
        left -= ended;
    }
}

// ---- the passes of one block, all fields in one array --------------------------
struct Fields {
    std::vector<double2> v;
    size_t n, k = 0;
    explicit Fields(size_t n_) : v(16 * n_), n(n_) {
        unsigned r = 12345;
        for (double2 &x : v) {
            r = r * 1664525u + 1013904223u;
            x.x = (double)(r >> 8) / (1 << 24) - 0.5;
            r = r * 1664525u + 1013904223u;
            x.y = (double)(r >> 8) / (1 << 24) - 0.5;
        }
    }
    double2 *c() { return v.data() + n * k++; }
    double *r() { return &c()->x; }
};

// true where both orders of pass(f) leave the same fields
template <typename F> static bool same(size_t n, int threads, F pass) {
    std::vector<double2> out[2];
    for (int up = 0; up < 2; ++up) {
        Fields f(n);
        std::memset(g_smem, 0, sizeof(g_smem));
        auto body = pass(f);
        g_body = body;
        block(threads, up == 1);
        out[up] = f.v;
    }
    return std::memcmp(out[0].data(), out[1].data(), sizeof(double2) * out[0].size()) == 0;
}

template <class G> static int check_x(const LineTab<double> &lt) {
    const G g(lt.g);
    using O = typename G::One;
    const O o(lt.g);
    const int n = g.n(), lines = 1 << g.nbl();
    const size_t sz = (size_t)n * 2 * lines;
    int bad = 0;
    auto fill = [&](auto &a) {
        a.lt = lt;
        a.nlines = lines;
    };
    auto say = [&](const char *name, bool ok) {
        if (!ok) std::printf("%d %s\n", n, name), ++bad;
    };
    say("x_rhs", same(sz, g.block(2), [&](Fields &f) {
            XRhsArgs<double> a{};
            fill(a);
            a.s1 = 0.1, a.s2 = -0.01;
            a.psi = f.c(), a.A = f.c(), a.dxpsi = f.c(), a.dxxpsi = f.c(), a.E = f.c();
            a.dxxay = f.r();
            return [a] { k_lx_rhs<double, G>(a); };
        }));
    say("x_d1", same(sz, o.block(1), [&](Fields &f) {
            XD1Args<double> a{};
            fill(a);
            a.s1 = 0.1;
            a.in = FieldIn<double>{f.c(), nullptr, nullptr};
            a.out = FieldOut<double>{f.c(), nullptr, nullptr};
            return [a] { k_lx_d1<double, O>(a); };
        }));
    say("x_d1r", same(sz, o.block(1), [&](Fields &f) {
            XD1Args<double> a{};
            fill(a);
            a.nlines = 2 * lines;
            a.s1 = 0.1;
            a.in = FieldIn<double>{nullptr, f.r(), nullptr};
            a.out = FieldOut<double>{nullptr, f.r(), nullptr, 2};
            return [a] { k_lx_d1r<double, O>(a); };
        }));
    say("x_filt_fwd", same(sz, o.block(1), [&](Fields &f) {
            XFiltFwdArgs<double> a{};
            fill(a);
            a.ny = lines;
            a.nf = 3;
            for (int i = 0; i < 3; ++i) {
                a.in[i] = FieldIn<double>{f.c(), nullptr, nullptr};
                a.spec[i] = f.c();
            }
            return [a] { k_lx_filt_fwd<double, O>(a); };
        }));
    say("x_filt_inv", same(sz, o.block(1), [&](Fields &f) {
            XFiltInvArgs<double> a{};
            fill(a);
            a.nf = 3;
            for (int i = 0; i < 3; ++i) {
                a.spec[i] = f.c();
                a.out[i] = FieldOut<double>{f.c(), nullptr, nullptr};
            }
            return [a] { k_lx_filt_inv<double, O>(a); };
        }));
    return bad;
}

template <class G> static int check_y(const LineTab<double> &lt) {
    const G g(lt.g);
    using O = typename G::One;
    const O o(lt.g);
    const int n = g.n(), lines = 1 << g.nbl();
    const size_t sz = (size_t)n * 2 * lines;
    std::vector<double> m(std::max(n, 2 * lines), 1.0);
    int bad = 0;
    auto fill = [&](auto &a) {
        a.lt = lt;
        a.nx = lines;
        a.ny = n;
    };
    auto say = [&](const char *name, bool ok) {
        if (!ok) std::printf("%d %s\n", n, name), ++bad;
    };
    say("y_rhs", same(sz, g.block(2), [&](Fields &f) {
            YRhsArgs<double> a{};
            fill(a);
            a.s1 = 0.1, a.s2 = -0.01;
            a.psi = f.c(), a.A = f.c(), a.E = f.c(), a.dxxay = f.r();
            a.dypsi = f.c(), a.dyypsi = f.c(), a.divA = f.r(), a.B = f.c();
            return [a] { k_ly_rhs<double, G>(a); };
        }));
    say("y_d1", same(sz, o.block(1), [&](Fields &f) {
            YD1Args<double> a{};
            fill(a);
            a.s1 = 0.1;
            a.in = FieldIn<double>{f.c(), nullptr, nullptr};
            a.add_re = f.r();
            a.out = FieldOut<double>{f.c(), nullptr, nullptr};
            return [a] { k_ly_d1<double, O>(a); };
        }));
    say("y_d1r", same(sz, o.block(1), [&](Fields &f) {
            YD1Args<double> a{};
            fill(a);
            a.nx = 2 * lines;
            a.s1 = 0.1;
            a.in = FieldIn<double>{nullptr, f.r(), nullptr};
            a.add_re = f.r();
            a.out = FieldOut<double>{nullptr, f.r(), nullptr};
            return [a] { k_ly_d1r<double, O>(a); };
        }));
    auto filt = [&](Fields &f) {
        YFiltArgs<double> a{};
        fill(a);
        a.nf = 2;
        for (int i = 0; i < 2; ++i) a.spec[i] = f.c();
        a.mx = a.my = m.data();
        a.scale = 1.0 / n;
        return a;
    };
    say("y_filt", same(sz, o.block(1), [&](Fields &f) {
            const YFiltArgs<double> a = filt(f);
            return [a] { k_ly_filt<double, O>(a); };
        }));
    say("y_fwd", same(sz, o.block(1), [&](Fields &f) {
            const YFiltArgs<double> a = filt(f);
            return [a] { k_ly_fwd<double, O>(a); };
        }));
    return bad;
}

int main(int argc, char **argv) {
    if (argc < 3) return 2;
    const bool y = argv[1][0] == 'y';
    int bad = 0;
    for (int i = 2; i < argc; ++i) {
        const int n = std::atoi(argv[i]);
        const LPlan p = lplan(n);
        std::vector<double2> roots(n), tw;
        for (int k = 0; k < n; ++k) {
            const double t = -2.0 * M_PI * k / n;
            roots[k] = make_double2(std::cos(t), std::sin(t));
        }
        std::vector<int> freq, pos;
        make_line_tables(p, roots, tw, freq, pos);
        for (bool half : {false, true}) {
            const LineTab<double> t{tw.data(), freq.data(), pos.data(), rgeo(p, y, half)};
            bad += y ? check_y<RGeo>(t) : check_x<RGeo>(t);
        }
        // the compile-time plans are the same kernels
        const LineTab<double> t{tw.data(), freq.data(), pos.data(), rgeo(p, y, false)};
        if (n == 33) bad += y ? check_y<SGeo<33, lnbl(33, true)>>(t)
                              : check_x<SGeo<33, lnbl(33, false)>>(t);
        if (n == 64) bad += y ? check_y<SGeo<64, lnbl(64, true)>>(t)
                              : check_x<SGeo<64, lnbl(64, false)>>(t);
    }
    if (!bad) std::printf("ok\n");
    return 0;
}
