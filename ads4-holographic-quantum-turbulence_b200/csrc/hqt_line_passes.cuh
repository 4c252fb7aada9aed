// hqt_line_passes.cuh -- the spectral passes of one RK stage and of the
// filter (what each computes: hqt_passes.cuh) on the in-place line transforms
// of hqt_line.cuh.  G is the geometry, compile-time (SGeo) or a kernel
// argument (RGeo).
//
// Bound: each pass streams its fields through HBM once (x_rhs 88, y_rhs 112
// bytes a site in FP64); next come the FP64 units (about 30 operations an
// element and transform) and shared memory.  Two buffers of a block's lines
// take at most 66 KB (64 KB at 512 and 1024 points along x, 256 and 512 along y), and with
// 128 registers a thread 512 threads fit on an SM: two such blocks, one's loads and stores
// behind the other's butterflies.  Four adjacent y lines take up to 130 KB, and from 900
// points on such a block is alone on its SM.
// Measured, us a launch, with threads over the lines first and the twiddles loaded
// for each buffer -> as it is: 512x512x25 x_rhs 196 -> 160 (3.6 TB/s), y_rhs 250 ->
// 244 (3.0 TB/s), filter x forward 154 -> 125, x inverse 183 -> 164; 256x256x25 x_rhs
// 50 -> 38; with a runtime plan 1001x1001x20 x_rhs 853 -> 864, y_rhs 1540 -> 1440,
// filter x forward / y / x inverse 636 / 797 / 981 -> 491 / 588 / 659.
#pragma once
#include "hqt_line.cuh"
#include "hqt_passes.cuh"

namespace hqt {

// The rhs passes get 128 registers a thread (512 threads per SM): an FP64
// radix-8 butterfly with its spectrum and one product fits without spills.
// The others hold one spectrum and get 80 (768 threads); with a runtime plan
// all get 128, for the radices 9..13.
#define HQT_L_BOUNDS(G) __launch_bounds__(G::kMaxThreads, 512 / G::kMaxThreads)
#define HQT_L_BOUNDS1(G) \
    __launch_bounds__(G::kMaxThreads, (G::kStatic && G::kMaxThreads < 512 ? 768 : 512) / G::kMaxThreads)

template <typename T> __device__ __forceinline__ C2<T> lzero() { return mk2<T>(T(0), T(0)); }

template <typename T, class G>
__global__ void HQT_L_BOUNDS(G) k_lx_rhs(const __grid_constant__ XRhsArgs<T> a) {
    const LineEng<T, G, true> w(a.lt);
    const int n = w.g.n(), L0 = blockIdx.x << w.g.nbl(), valid = a.nlines - L0;
    const long long g0 = (long long)L0 * n;
    pdl_wait();
    auto at = [&](int b, int e) { return g0 + (long long)b * n + e; };
    // Psi, then C = A_x + i A_y: first and second derivative
#pragma unroll 1
    for (int f = 0; f < 2; ++f) {
        w.first_d(w.A, [&](int b, int e) {
            if (b >= valid) return lzero<T>();
            const long long g = at(b, e);
            return f == 0 ? a.psi[g] : a.A[g];
        });
        w.forward_mid(false);
        w.middle_deriv12(a.s1, a.s2);
        w.inverse_mid(true);
        C2<T> *d1 = f == 0 ? a.dxpsi : a.E;
        w.last2(
            true, [](int, int) { return 0; },
            [&](int b, int e, C2<T> v, int) {
                if (b < valid) d1[at(b, e)] = v;
            },
            [&](int b, int e, C2<T> v) {
                if (b >= valid) return;
                if (f == 0)
                    a.dxxpsi[at(b, e)] = v;
                else
                    a.dxxay[at(b, e)] = v.y;
            });
    }
}

// The gauge fields travel as two complex lines whose y derivatives are the
// outputs (no split of pair spectra):
//   W1 = E_x + i A_y:  div A = E_x + Im(d_y W1),  d_x B = d_xx A_y - Re(d_y W1);
//   W2 = A_x + i E_y:  d_y B = Im(d_y W2) - Re(d_yy W2)
//      = Re(IFFT((s1 k - s2 k^2) W2^)), one real multiplier.
template <typename T, class G>
__global__ void HQT_L_BOUNDS(G) k_ly_rhs(const __grid_constant__ YRhsArgs<T> a) {
    const LineEng<T, G, false> w(a.lt);
    const int x0 = blockIdx.x << w.g.nbl(), valid = a.nx - x0;
    const long long zoff = (long long)blockIdx.y * a.ny * a.nx + x0;
    pdl_wait();
    auto at = [&](int b, int e) { return zoff + (long long)e * a.nx + b; };
#pragma unroll 1
    for (int f = 0; f < 2; ++f) {
        if (f == 0) {
            w.first_d(w.A, [&](int b, int e) { return b < valid ? a.psi[at(b, e)] : lzero<T>(); });
        } else {
            w.first_d2(
                [&](int b, int e) {
                    if (b >= valid) return lzero<T>();
                    const long long g = at(b, e);
                    return mk2<T>(a.E[g].x, a.A[g].y);
                },
                [&](int b, int e) {
                    if (b >= valid) return lzero<T>();
                    const long long g = at(b, e);
                    return mk2<T>(a.A[g].x, a.E[g].y);
                });
        }
        w.forward_mid(f == 1);
        if (f == 0) {
            w.middle_deriv12(a.s1, a.s2);
        } else {
            w.middle_deriv1(w.A, a.s1);
            w.middle_deriv_mix(w.B, a.s1, a.s2);
        }
        w.inverse_mid(true);
        if (f == 0) {
            w.last2(
                true, [](int, int) { return 0; },
                [&](int b, int e, C2<T> v, int) {
                    if (b < valid) a.dypsi[at(b, e)] = v;
                },
                [&](int b, int e, C2<T> v) {
                    if (b < valid) a.dyypsi[at(b, e)] = v;
                });
        } else {
            w.last2(
                true,
                [&](int b, int e) {
                    if (b >= valid) return lzero<T>();
                    const long long g = at(b, e);
                    return mk2<T>(a.E[g].x, a.dxxay[g]);
                },
                [&](int b, int e, C2<T> v, C2<T> x) {
                    if (b >= valid) return;
                    const long long g = at(b, e);
                    a.divA[g] = x.x + v.y;
                    a.B[g].y = x.y - v.x;
                },
                [&](int b, int e, C2<T> v) {
                    if (b < valid) a.B[at(b, e)].x = v.x;
                });
        }
    }
}

template <typename T, class G>
__global__ void HQT_L_BOUNDS1(G) k_lx_d1(const __grid_constant__ XD1Args<T> a) {
    const LineEng<T, G, true> w(a.lt);
    const int n = w.g.n(), L0 = blockIdx.x << w.g.nbl(), valid = a.nlines - L0;
    const long long g0 = (long long)L0 * n;
    pdl_wait();
    auto at = [&](int b, int e) { return g0 + (long long)b * n + e; };
    w.first_d(w.A, [&](int b, int e) {
        return b < valid ? load_field(a.in, at(b, e)) : lzero<T>();
    });
    w.forward_mid(false);
    w.middle_deriv1(w.A, a.s1);
    w.inverse_mid(false);
    w.last([&](int b, int e, C2<T> v) {
        if (b < valid) store_field(a.out, at(b, e), v);
    });
}

template <typename T, class G>
__global__ void HQT_L_BOUNDS1(G) k_ly_d1(const __grid_constant__ YD1Args<T> a) {
    const LineEng<T, G, false> w(a.lt);
    const int x0 = blockIdx.x << w.g.nbl(), valid = a.nx - x0;
    const long long zoff = (long long)blockIdx.y * a.ny * a.nx + x0;
    pdl_wait();
    auto at = [&](int b, int e) { return zoff + (long long)e * a.nx + b; };
    w.first_d(w.A, [&](int b, int e) {
        return b < valid ? load_field(a.in, at(b, e)) : lzero<T>();
    });
    w.forward_mid(false);
    w.middle_deriv1(w.A, a.s1);
    w.inverse_mid(false);
    w.last2(
        false, [&](int b, int e) { return a.add_re && b < valid ? a.add_re[at(b, e)] : T(0); },
        [&](int b, int e, C2<T> v, T x) {
            v.x += x;
            if (b < valid) store_field(a.out, at(b, e), v);
        },
        [](int, int, C2<T>) {});
}

// First derivative of a real field into a real field, two real lines per
// complex line (real_field_d1): complex line b carries real lines 2b and 2b+1.
template <typename T, class G>
__global__ void HQT_L_BOUNDS1(G) k_lx_d1r(const __grid_constant__ XD1Args<T> a) {
    const LineEng<T, G, true> w(a.lt);
    const int n = w.g.n(), L0 = blockIdx.x << (w.g.nbl() + 1), nr = a.nlines - L0;
    const int si = a.in.st, so = a.out.st;
    const T *src = a.in.re + (long long)L0 * n * si;
    T *dst = a.out.re + (long long)L0 * n * so;
    pdl_wait();
    w.first_d(w.A, [&](int b, int e) {
        const long long g = 2ll * b * n + e;
        return mk2<T>(2 * b < nr ? src[g * si] : T(0), 2 * b + 1 < nr ? src[(g + n) * si] : T(0));
    });
    w.forward_mid(false);
    w.middle_deriv1(w.A, a.s1);
    w.inverse_mid(false);
    w.last([&](int b, int e, C2<T> v) {
        const long long g = 2ll * b * n + e;
        if (2 * b < nr) dst[g * so] = v.x;
        if (2 * b + 1 < nr) dst[(g + n) * so] = v.y;
    });
}

template <typename T, class G>
__global__ void HQT_L_BOUNDS1(G) k_ly_d1r(const __grid_constant__ YD1Args<T> a) {
    const LineEng<T, G, false> w(a.lt);
    const int x0 = blockIdx.x << (w.g.nbl() + 1), nr = a.nx - x0;
    const long long zoff = (long long)blockIdx.y * a.ny * a.nx + x0;
    pdl_wait();
    auto pair = [&](const T *p, int st, int b, int e) {
        const long long g = (zoff + (long long)e * a.nx + 2 * b) * st;
        return mk2<T>(2 * b < nr ? p[g] : T(0), 2 * b + 1 < nr ? p[g + st] : T(0));
    };
    w.first_d(w.A, [&](int b, int e) { return pair(a.in.re, a.in.st, b, e); });
    w.forward_mid(false);
    w.middle_deriv1(w.A, a.s1);
    w.inverse_mid(false);
    w.last2(
        false, [&](int b, int e) { return a.add_re ? pair(a.add_re, 1, b, e) : lzero<T>(); },
        [&](int b, int e, C2<T> v, C2<T> x) {
            const int st = a.out.st;
            const long long g = (zoff + (long long)e * a.nx + 2 * b) * st;
            if (2 * b < nr) a.out.re[g] = v.x + x.x;
            if (2 * b + 1 < nr) a.out.re[g + st] = v.y + x.y;
        },
        [](int, int, C2<T>) {});
}

// Filter, x forward: spectra in natural order, the weight-zeroed columns left
// unwritten.
template <typename T, class G>
__global__ void HQT_L_BOUNDS1(G) k_lx_filt_fwd(const __grid_constant__ XFiltFwdArgs<T> a) {
    const LineEng<T, G, true> w(a.lt);
    const int n = w.g.n(), L0 = blockIdx.x << w.g.nbl(), valid = a.nlines - L0;
    const long long g0 = (long long)L0 * n;
    pdl_wait();
    const int wnd = a.st ? a.st->winding : 0;
    auto at = [&](int b, int e) { return g0 + (long long)b * n + e; };
    // winding phase of line L0 + b (tevol_driven_cluster.m:139)
    auto phase = [&](int b) {
        const int y = (L0 + b) % a.ny;
        const long long q = ((long long)y * wnd) % a.ny;
        double sn, cs;
        sincospi(-2.0 * (double)q / (double)a.ny, &sn, &cs);
        return mk2<T>((T)cs, (T)sn);
    };
#pragma unroll 1
    for (int f = 0; f < a.nf; ++f) {
        // one load expression per kind of field, without branches an element:
        // the loads of a butterfly are in flight together
        const FieldIn<T> in = a.in[f];
        const bool turn = f == 0 && wnd != 0;
        if (in.c) {
            w.first(w.A, turn, phase,
                    [&](int b, int e) { return b < valid ? in.c[at(b, e)] : lzero<T>(); });
        } else {
            const bool pair = in.im != nullptr;
            const T *im = pair ? in.im : in.re;
            w.first(w.A, turn, phase, [&](int b, int e) {
                if (b >= valid) return lzero<T>();
                const long long g = at(b, e);
                const T re = in.re[g], i = im[g];
                return mk2<T>(re, pair ? i : T(0));
            });
        }
        w.forward_rest();
        C2<T> *spec = a.spec[f];
        w.modes([&](int b, int k) {
            if (b < valid && filt_col_live(k, a.dead0, a.dead1))
                spec[at(b, k)] = w.A[w.at(b, w.pos(k))];
        });
        __syncthreads();  // the next field's first pass writes other threads' rows
    }
}

// Filter, y: forward, weight, inverse; blockIdx.z = field
template <typename T, class G>
__global__ void HQT_L_BOUNDS1(G) k_ly_filt(const __grid_constant__ YFiltArgs<T> a) {
    const LineEng<T, G, false> w(a.lt);
    const int n = w.g.n(), NB = 1 << w.g.nbl();
    const int x0 = blockIdx.x * NB, valid = min(NB, a.nx - x0);
    const long long zoff = (long long)blockIdx.y * a.ny * a.nx + x0;
    bool live = false;
    for (int b = 0; b < valid; ++b) live = live || filt_col_live(x0 + b, a.dead0, a.dead1);
    if (!live) return;  // every column filtered out
    pdl_wait();
    C2<T> *spec = a.spec[blockIdx.z];
    auto at = [&](int b, int e) { return zoff + (long long)e * a.nx + b; };
    w.first(w.A, [&](int b, int e) { return b < valid ? spec[at(b, e)] : lzero<T>(); });
    w.forward_mid(false);
    w.middle(w.A, [&](auto &v, int b, int blk, int k0, int st) {
        constexpr int R = sizeof(v) / sizeof(C2<T>);
        const int kx = x0 + min(b, valid - 1), kxm = kx == 0 ? 0 : a.nx - kx;
        const T m0 = __ldg(a.mx + kx), m1 = __ldg(a.mx + kxm);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int ky = k0 + i * st, kym = ky == 0 ? 0 : n - ky;
            const T wgt = T(0.5) * (m0 * __ldg(a.my + ky) + m1 * __ldg(a.my + kym)) * a.scale;
            v[i] = wgt * v[i];
        }
        w.template put<R>(w.A, b, blk, v);
    });
    w.inverse_mid(false);
    w.last([&](int b, int e, C2<T> v) {
        if (b < valid) spec[at(b, e)] = v;
    });
}

// Filter, x inverse; a non-finite value sets the status' first bad step
template <typename T, class G>
__global__ void HQT_L_BOUNDS1(G) k_lx_filt_inv(const __grid_constant__ XFiltInvArgs<T> a) {
    const LineEng<T, G, true> w(a.lt);
    const int n = w.g.n(), L0 = blockIdx.x << w.g.nbl(), valid = a.nlines - L0;
    const long long g0 = (long long)L0 * n;
    pdl_wait();
    int bad = 0;
    auto at = [&](int b, int e) { return g0 + (long long)b * n + e; };
#pragma unroll 1
    for (int f = 0; f < a.nf; ++f) {
        const C2<T> *spec = a.spec[f];
        w.modes([&](int b, int k) {
            w.A[w.at(b, w.pos(k))] =
                b < valid && filt_col_live(k, a.dead0, a.dead1) ? spec[at(b, k)] : lzero<T>();
        });
        w.inverse_begin();
        const FieldOut<T> out = a.out[f];
        w.last([&](int b, int e, C2<T> v) {
            if (!(isfinite(v.x) && isfinite(v.y))) bad = 1;
            if (b < valid) store_field(out, at(b, e), v);
        });
        __syncthreads();  // the next field's load writes other threads' rows
    }
    if (a.st && __syncthreads_or(bad) && threadIdx.x == 0)
        atomicMin(reinterpret_cast<unsigned long long *>(&a.st->first_bad_step),
                  (unsigned long long)(a.st->step + 1));
}

// Forward transform along y of nf complex fields, natural order (spectrum)
template <typename T, class G>
__global__ void HQT_L_BOUNDS1(G) k_ly_fwd(const __grid_constant__ YFiltArgs<T> a) {
    const LineEng<T, G, false> w(a.lt);
    const int x0 = blockIdx.x << w.g.nbl(), valid = a.nx - x0;
    const long long zoff = (long long)blockIdx.y * a.ny * a.nx + x0;
    pdl_wait();
    auto at = [&](int b, int e) { return zoff + (long long)e * a.nx + b; };
#pragma unroll 1
    for (int f = 0; f < a.nf; ++f) {
        C2<T> *spec = a.spec[f];
        w.first(w.A, [&](int b, int e) { return b < valid ? spec[at(b, e)] : lzero<T>(); });
        w.forward_rest();
        w.modes([&](int b, int k) {
            if (b < valid) spec[at(b, k)] = w.A[w.at(b, w.pos(k))];
        });
        __syncthreads();
    }
}

}  // namespace hqt
