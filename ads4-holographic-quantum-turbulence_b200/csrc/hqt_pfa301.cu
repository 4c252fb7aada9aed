// The prime-factor tensor-core line passes of 301 = 7 * 43 points.
#include <vector>

#include "hqt_launch.h"
#define HQT_PFA_P 7
#define HQT_PFA_Q 43
#include "hqt_passes.cuh"
#include "hqt_pfa_passes.cuh"

namespace hqt {

cudaError_t pfa_init_301() {
    std::vector<double> frag(PfaDims<HQT_PFA_P, HQT_PFA_Q>::NFRAG * 32);
    pfa_fragments<HQT_PFA_P, HQT_PFA_Q>(frag.data());
    cudaError_t e = cudaMemcpyToSymbol(g_pfa_frag, frag.data(), sizeof(double) * frag.size());
    std::vector<float> frag32(PfaDims<HQT_PFA_P, HQT_PFA_Q>::NFRAG32 * 32);
    pfa_fragments32<HQT_PFA_P, HQT_PFA_Q>(frag32.data());
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbol(g_pfa_frag32, frag32.data(), sizeof(float) * frag32.size());
    // positions of the FP64 storage order
    constexpr int P = HQT_PFA_P, Q = HQT_PFA_Q, N = P * Q;
    using D = PfaDims<P, Q>;
    constexpr int PITCH = PfaStore<double, P, Q>::PITCH;
    unsigned short at[Q], k2[Q], pos[kPfaLines * N], spos[kPfaLines * N];
    at[0] = Q - 1;
    for (int i = 0; i < Q - 1; ++i) at[pfa_pow3(i)] = (unsigned short)i;
    for (int t = 0; t < Q; ++t) k2[at[t]] = (unsigned short)t;
    for (int n = 0; n < N; ++n)
        for (int ln = 0; ln < kPfaLines; ++ln) {
            pos[kPfaLines * n + ln] = (unsigned short)((ln * P + n * D::QIP % P) * PITCH +
                                                       at[n * D::PIQ % Q]);
            spos[kPfaLines * n + ln] = (unsigned short)((ln * P + n % P) * PITCH + at[n % Q]);
        }
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_pfa_pos, pos, sizeof(pos));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_pfa_spos, spos, sizeof(spos));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_pfa_k2, k2, sizeof(k2));
    return e;
}

cudaError_t pfa_launch_301(int kind, const void *args, int nlines, cudaStream_t s) {
    constexpr int P = HQT_PFA_P, Q = HQT_PFA_Q;
    const int grid = (nlines + kPfaLines - 1) / kPfaLines;  // x passes
    constexpr size_t smem = pfa_smem_bytes<double, P, Q>();
    constexpr size_t smem32 = pfa_smem_bytes<float, P, Q>();
    auto ygrid = [&](int nx, int nz_) {
        return dim3((nx + kPfaLines - 1) / kPfaLines, nz_);
    };
    // real-field first derivatives: kPfaRealLines real lines per warp
    const int rgrid = (nlines + kPfaRealLines - 1) / kPfaRealLines;
    auto yrgrid = [&](int nx, int nz_) {
        return dim3((nx + kPfaRealLines - 1) / kPfaRealLines, nz_);
    };
    switch (kind) {
        case CT_X_RHS:
            (void)klaunch(k_x_rhs_pfa<double, P, Q>, dim3(grid), dim3(32), smem, s,
                          *(const XRhsArgs<double> *)args);
            break;
        case CT_Y_RHS: {
            const YRhsArgs<double> &a = *(const YRhsArgs<double> *)args;
            (void)klaunch(k_y_rhs_pfa<double, P, Q>, dim3(ygrid(a.nx, nlines)), dim3(32), smem, s,
                          a);
            break;
        }
        case CT_X_D1: {
            const XD1Args<double> &a = *(const XD1Args<double> *)args;
            if (real_field_d1(a.in, a.out))
                (void)klaunch(k_x_d1r_pfa<double, P, Q>, dim3(rgrid), dim3(32), smem, s, a);
            else
                (void)klaunch(k_x_d1_pfa<double, P, Q>, dim3(grid), dim3(32), smem, s, a);
            break;
        }
        case CT_Y_D1: {
            const YD1Args<double> &a = *(const YD1Args<double> *)args;
            if (real_field_d1(a.in, a.out))
                (void)klaunch(k_y_d1r_pfa<double, P, Q>, dim3(yrgrid(a.nx, nlines)), dim3(32), smem,
                              s, a);
            else
                (void)klaunch(k_y_d1_pfa<double, P, Q>, dim3(ygrid(a.nx, nlines)), dim3(32), smem,
                              s, a);
            break;
        }
        case CT_X_RHS_F:
            (void)klaunch(k_x_rhs_pfa<float, P, Q>, dim3(grid), dim3(32), smem32, s,
                          *(const XRhsArgs<float> *)args);
            break;
        case CT_Y_RHS_F: {
            const YRhsArgs<float> &a = *(const YRhsArgs<float> *)args;
            (void)klaunch(k_y_rhs_pfa<float, P, Q>, dim3(ygrid(a.nx, nlines)), dim3(32), smem32, s,
                          a);
            break;
        }
        case CT_X_D1_F: {
            const XD1Args<float> &a = *(const XD1Args<float> *)args;
            if (real_field_d1(a.in, a.out))
                (void)klaunch(k_x_d1r_pfa<float, P, Q>, dim3(rgrid), dim3(32), smem32, s, a);
            else
                (void)klaunch(k_x_d1_pfa<float, P, Q>, dim3(grid), dim3(32), smem32, s, a);
            break;
        }
        case CT_Y_D1_F: {
            const YD1Args<float> &a = *(const YD1Args<float> *)args;
            if (real_field_d1(a.in, a.out))
                (void)klaunch(k_y_d1r_pfa<float, P, Q>, dim3(yrgrid(a.nx, nlines)), dim3(32),
                              smem32, s, a);
            else
                (void)klaunch(k_y_d1_pfa<float, P, Q>, dim3(ygrid(a.nx, nlines)), dim3(32), smem32,
                              s, a);
            break;
        }
        case CT_FX_FWD:
            (void)klaunch(k_x_filt_fwd_pfa<P, Q>, dim3(grid), dim3(32), smem, s,
                          *(const XFiltFwdArgs<double> *)args);
            break;
        case CT_FY: {
            const YFiltArgs<double> &a = *(const YFiltArgs<double> *)args;
            (void)klaunch(k_y_filt_pfa<P, Q>,
                          dim3((a.nx + kPfaLines - 1) / kPfaLines, nlines, a.nf), dim3(32), smem, s,
                          a);
            break;
        }
        case CT_FX_INV:
            (void)klaunch(k_x_filt_inv_pfa<P, Q>, dim3(grid), dim3(32), smem, s,
                          *(const XFiltInvArgs<double> *)args);
            break;
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}
}  // namespace hqt
