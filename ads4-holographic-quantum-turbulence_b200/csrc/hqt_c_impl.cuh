// hqt_c_impl.cuh -- the line passes of one compile-time length HQT_CN (each
// hqt_c<N>.cu defines HQT_CN and includes this): FP64 in place, FP32 (mixed
// precision) by the Stockham transforms.
#include <vector>

#include "hqt_cpasses.cuh"
#include "hqt_line_impl.cuh"

#ifndef HQT_CN
#error "define HQT_CN"
#endif

namespace hqt {

#if HQT_CN != 301  // 7*43: FP64 on the prime-factor engine
using L64 = LineLaunch<double, SGeo<HQT_CN, lnbl(HQT_CN, false)>,
                       SGeo<HQT_CN, lnbl(HQT_CN, true)>>;
template <> cudaError_t ct_init64<HQT_CN>(int max_smem) {
    const cudaError_t e = L64::init_x(max_smem);
    return e == cudaSuccess ? L64::init_y(max_smem) : e;
}
template <> cudaError_t ct_launch_x64<HQT_CN>(int kind, const void *args, cudaStream_t s) {
    return L64::launch_x(kind, args, s);
}
template <>
cudaError_t ct_launch_y64<HQT_CN>(int kind, const void *args, int nsl, cudaStream_t s) {
    return L64::launch_y(kind, args, nsl, s);
}
#endif

template <>
cudaError_t ct_init<HQT_CN>(const double *tc, const double *ts, int ntab, const double *bc,
                            const double *bs, int nbig, int max_smem) {
    if (ntab != kTabTotal || nbig != kBigTotal) return cudaErrorInvalidValue;
    std::vector<float> fc(tc, tc + ntab), fs(ts, ts + ntab), gc(bc, bc + nbig), gs(bs, bs + nbig);
    cudaError_t e = cudaMemcpyToSymbol(c_tab_cos_f, fc.data(), sizeof(float) * ntab);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_tab_sin_f, fs.data(), sizeof(float) * ntab);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_big_cos_f, gc.data(), sizeof(float) * nbig);
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_big_sin_f, gs.data(), sizeof(float) * nbig);
    auto opt = [&](const void *fn) {
        cudaFuncAttributes fa{};
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     max_smem - (int)fa.sharedSizeBytes);
    };
    opt((const void *)k_x_rhs_c<float, HQT_CN>);
    opt((const void *)k_y_rhs_c<float, HQT_CN>);
    opt((const void *)k_x_d1_c<float, HQT_CN>);
    opt((const void *)k_y_d1_c<float, HQT_CN>);
    opt((const void *)k_x_d1r_c<float, HQT_CN>);
    opt((const void *)k_y_d1r_c<float, HQT_CN>);
    return e;
}

template <>
cudaError_t ct_launch<HQT_CN>(int kind, const void *args, dim3 grid, size_t smem,
                              cudaStream_t s) {
    // block sizes: ct_threads of each kernel's NB (the expressions of the kernels)
    constexpr int N = HQT_CN, EF = (int)sizeof(float2);
    constexpr int TXRf = ct_threads_n(N, ct_lines(N, 3, EF), EF);
    constexpr int TYRf = ct_threads_n(N, ct_lines_y(N, 3, EF), EF);
    constexpr int TX2f = ct_threads_n(N, ct_lines(N, 2, EF), EF);
    constexpr int TY2f = ct_threads_n(N, ct_lines_y(N, 2, EF), EF);
    switch (kind) {
        case CT_X_RHS_F:
            (void)klaunch(k_x_rhs_c<float, HQT_CN>, dim3(grid), dim3(TXRf), smem, s,
                          *(const XRhsArgs<float> *)args);
            break;
        case CT_Y_RHS_F:
            (void)klaunch(k_y_rhs_c<float, HQT_CN>, dim3(grid), dim3(TYRf), smem, s,
                          *(const YRhsArgs<float> *)args);
            break;
        case CT_X_D1_F: {
            const XD1Args<float> &a = *(const XD1Args<float> *)args;
            constexpr int nb2 = 2 * ct_lines(HQT_CN, 2, sizeof(float2));
            if (real_field_d1(a.in, a.out))
                (void)klaunch(k_x_d1r_c<float, HQT_CN>, dim3((a.nlines + nb2 - 1) / nb2),
                              dim3(TX2f), smem, s, a);
            else
                (void)klaunch(k_x_d1_c<float, HQT_CN>, dim3(grid), dim3(TX2f), smem, s, a);
            break;
        }
        case CT_Y_D1_F: {
            const YD1Args<float> &a = *(const YD1Args<float> *)args;
            constexpr int nb2 = 2 * ct_lines_y(HQT_CN, 2, sizeof(float2));
            if (real_field_d1(a.in, a.out))
                (void)klaunch(k_y_d1r_c<float, HQT_CN>, dim3((a.nx + nb2 - 1) / nb2, grid.y),
                              dim3(TY2f), smem, s, a);
            else
                (void)klaunch(k_y_d1_c<float, HQT_CN>, dim3(grid), dim3(TY2f), smem, s, a);
            break;
        }
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace hqt
