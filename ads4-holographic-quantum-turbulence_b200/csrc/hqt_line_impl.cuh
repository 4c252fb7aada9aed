// hqt_line_impl.cuh -- launchers of the in-place line passes for one pair of
// geometries (GX along x, GY along y) and element type.
#pragma once
#include "hqt_launch.h"
#include "hqt_line_passes.cuh"

namespace hqt {

template <typename T, class GX, class GY> struct LineLaunch {
    using OX = typename GX::One;  // of the passes with one buffer
    using OY = typename GY::One;
    static cudaError_t opt(const void *fn, int max_smem, cudaError_t e) {
        cudaFuncAttributes fa{};
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     max_smem - (int)fa.sharedSizeBytes);
        return e;
    }
    static cudaError_t init_x(int max_smem) {
        cudaError_t e = cudaSuccess;
        e = opt((const void *)k_lx_rhs<T, GX>, max_smem, e);
        e = opt((const void *)k_lx_d1<T, OX>, max_smem, e);
        e = opt((const void *)k_lx_d1r<T, OX>, max_smem, e);
        e = opt((const void *)k_lx_filt_fwd<T, OX>, max_smem, e);
        return opt((const void *)k_lx_filt_inv<T, OX>, max_smem, e);
    }
    static cudaError_t init_y(int max_smem) {
        cudaError_t e = cudaSuccess;
        e = opt((const void *)k_ly_rhs<T, GY>, max_smem, e);
        e = opt((const void *)k_ly_d1<T, OY>, max_smem, e);
        e = opt((const void *)k_ly_d1r<T, OY>, max_smem, e);
        e = opt((const void *)k_ly_filt<T, OY>, max_smem, e);
        return opt((const void *)k_ly_fwd<T, OY>, max_smem, e);
    }
    // lines of a pass, in blocks of `per` complex lines of geometry g, nbuf
    // buffers each
    template <class G, class K, class A>
    static cudaError_t go(K k, const A &a, int lines, int ny, int nz, int nbuf, int real,
                          cudaStream_t s) {
        const G g(a.lt.g);
        const int per = (1 << g.nbl()) * real;
        const size_t smem = sizeof(C2<T>) * nbuf * ((size_t)g.n() << g.nbl());
        (void)klaunch(k, dim3((lines + per - 1) / per, ny, nz), dim3(g.block(nbuf)), smem, s, a);
        return cudaGetLastError();
    }
    static cudaError_t launch_x(int kind, const void *args, cudaStream_t s) {
        switch (kind) {
            case CT_X_RHS: {
                const XRhsArgs<T> &a = *(const XRhsArgs<T> *)args;
                return go<GX>(k_lx_rhs<T, GX>, a, a.nlines, 1, 1, 2, 1, s);
            }
            case CT_X_D1: {
                const XD1Args<T> &a = *(const XD1Args<T> *)args;
                if (real_field_d1(a.in, a.out))
                    return go<OX>(k_lx_d1r<T, OX>, a, a.nlines, 1, 1, 1, 2, s);
                return go<OX>(k_lx_d1<T, OX>, a, a.nlines, 1, 1, 1, 1, s);
            }
            case CT_FX_FWD: {
                const XFiltFwdArgs<T> &a = *(const XFiltFwdArgs<T> *)args;
                return go<OX>(k_lx_filt_fwd<T, OX>, a, a.nlines, 1, 1, 1, 1, s);
            }
            case CT_FX_INV: {
                const XFiltInvArgs<T> &a = *(const XFiltInvArgs<T> *)args;
                return go<OX>(k_lx_filt_inv<T, OX>, a, a.nlines, 1, 1, 1, 1, s);
            }
        }
        return cudaErrorInvalidValue;
    }
    // nsl: z slices
    static cudaError_t launch_y(int kind, const void *args, int nsl, cudaStream_t s) {
        switch (kind) {
            case CT_Y_RHS: {
                const YRhsArgs<T> &a = *(const YRhsArgs<T> *)args;
                return go<GY>(k_ly_rhs<T, GY>, a, a.nx, nsl, 1, 2, 1, s);
            }
            case CT_Y_D1: {
                const YD1Args<T> &a = *(const YD1Args<T> *)args;
                if (real_field_d1(a.in, a.out))
                    return go<OY>(k_ly_d1r<T, OY>, a, a.nx, nsl, 1, 1, 2, s);
                return go<OY>(k_ly_d1<T, OY>, a, a.nx, nsl, 1, 1, 1, s);
            }
            case CT_FY: {
                const YFiltArgs<T> &a = *(const YFiltArgs<T> *)args;
                return go<OY>(k_ly_filt<T, OY>, a, a.nx, nsl, a.nf, 1, 1, s);
            }
            case CT_Y_FWD: {
                const YFiltArgs<T> &a = *(const YFiltArgs<T> *)args;
                return go<OY>(k_ly_fwd<T, OY>, a, a.nx, nsl, 1, 1, 1, s);
            }
        }
        return cudaErrorInvalidValue;
    }
};

}  // namespace hqt
