// hqt_z_impl.cuh -- launchers of the column kernels for one column length
// HQT_ZN (each hqt_z<N>.cu defines HQT_ZN and includes this file).
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "hqt_launch.h"
#include "hqt_zcol.cuh"
#include "hqt_zcons.cuh"
#include "hqt_zstage.cuh"

#ifndef HQT_ZN
#error "define HQT_ZN"
#endif

namespace hqt {

static ZOps<double, HQT_ZN> make_zops(const ZHost &h) {
    ZOps<double, HQT_ZN> op;
    std::memset(&op, 0, sizeof(op));
    const int nz = h.nz;
    for (int i = 0; i < nz; ++i) {
        for (int j = 0; j < nz; ++j) op.Lz[i][j] = h.Lz[(size_t)i * nz + j];
        op.zz[i] = h.zz[i];
        op.fz[i] = 1.0 - h.zz[i] * h.zz[i] * h.zz[i];
        op.lzb[i] = h.Lz[(size_t)(nz - 1) * nz + i];
    }
    for (int i = 0; i < nz - 1; ++i)
        for (int j = 0; j < nz - 1; ++j) op.Lz1[i][j] = h.Lz1[(size_t)i * (nz - 1) + j];
    return op;
}

template <> cudaError_t z_init<HQT_ZN>(int max_smem) {
    cudaError_t e = cudaSuccess;
    auto opt = [&](const void *fn) {
        // the opt-in limit covers static and dynamic shared memory together
        cudaFuncAttributes fa{};
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, fn);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     max_smem - (int)fa.sharedSizeBytes);
    };
    opt((const void *)k_zstage<double, HQT_ZN, 0>);
    opt((const void *)k_zstage<double, HQT_ZN, 1>);
    opt((const void *)k_zstage<double, HQT_ZN, 2>);
    opt((const void *)k_zstage<double, HQT_ZN, 3>);
    opt((const void *)k_zstage<double, HQT_ZN, 4>);
    opt((const void *)k_zstage<float, HQT_ZN, 1>);
    opt((const void *)k_zstage<float, HQT_ZN, 2>);
    opt((const void *)k_zstage<float, HQT_ZN, 3>);
    opt((const void *)k_zstage<float, HQT_ZN, 4>);
    opt((const void *)k_zcons<HQT_ZN>);
    return e;
}

// Operand tables of the radial stage: the fragments per lane ([frag][lane]) of
// Le, Lo (the half-size products of Lz, hqt_zstage.cuh) and Lz1, and z,
// 1 - z^3, Lz(nz,:) padded to HQT_ZN.  Lz enters through its centro-antisymmetric
// part (Lz(i,j) - Lz(n'-i,n'-j))/2, from which it differs by rounding (the
// diagonal is a sum).
template <>
void z_tables<HQT_ZN>(const ZHost &h, std::vector<double> &frag, std::vector<double> &tab) {
    using D = ZsDims<HQT_ZN>;
    const int nz = h.nz, n1 = nz - 1, hf = (nz + 1) / 2;
    auto L = [&](int i, int j) {
        return 0.5 * (h.Lz[(size_t)i * nz + j] - h.Lz[(size_t)(n1 - i) * nz + (n1 - j)]);
    };
    frag.clear();
    auto put = [&](int mt, int kt, auto f) {
        for (int m = 0; m < mt; ++m)
            for (int s = 0; s < kt; ++s)
                for (int lane = 0; lane < 32; ++lane)
                    frag.push_back(f(8 * m + zs_row(lane >> 2), 4 * s + (lane & 3)));
    };
    put(D::MP, D::KE, [&](int i, int j) {
        if (i >= nz / 2 || j >= hf) return 0.0;
        return j == n1 - j ? 0.5 * L(i, j) : 0.5 * (L(i, j) + L(i, n1 - j));
    });
    put(D::MH, D::KO, [&](int i, int j) {
        if (i >= hf || j >= nz / 2) return 0.0;
        if (j == 0) return 1.0;  // the end values' line
        return 0.5 * (L(i, j) - L(i, n1 - j));
    });
    put(D::M1, D::K1, [&](int i, int j) {
        return i < n1 && j < n1 ? h.Lz1[(size_t)i * n1 + j] : 0.0;
    });
    tab.assign(D::ntab, 0.0);
    // 2 (1 - z_j) = 2 sin^2(j pi/2n'): from zz it would be off by the rounding of
    // z near 1, which Lz multiplies by n'^2
    tab[3 * HQT_ZN] = 1.0;
    for (int j = 1; j < nz / 2; ++j) {
        const double s = std::sin(j * 3.14159265358979323846 / (2.0 * n1));
        tab[3 * HQT_ZN + j] = 2.0 * s * s;
    }
    for (int i = 0; i < nz; ++i) {
        tab[i] = h.zz[i];
        tab[HQT_ZN + i] = 1.0 - h.zz[i] * h.zz[i] * h.zz[i];
        tab[2 * HQT_ZN + i] = h.Lz[(size_t)n1 * nz + i];
    }
}

// One launch per stage (hqt_zstage.cuh): persistent blocks, as many as fit on
// the device at once, each looping over tiles of kZsCols columns.
template <typename TD, int M>
static cudaError_t z_stage_mode(const ZStageArgs<TD> &a, cudaStream_t s) {
    constexpr int smem = ZsLay<TD, HQT_ZN, M>::bytes;
    static int per_sm = 0, nsm = 0;
    if (per_sm == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_zstage<TD, HQT_ZN, M>, kZsThreads,
                                                      smem);
        if (per_sm < 1) per_sm = 1;
    }
    const long long tiles = (a.plane + kZsCols - 1) / kZsCols;
    const long long full = (long long)per_sm * (nsm > 0 ? nsm : 1);
    (void)klaunch(k_zstage<TD, HQT_ZN, M>, dim3((int)(tiles < full ? tiles : full)),
                  dim3(kZsThreads), smem, s, a);
    return cudaGetLastError();
}

template <>
cudaError_t z_stage<HQT_ZN>(int mode, const ZStageArgs<double> &a, cudaStream_t s) {
    switch (mode) {
        case 0: return z_stage_mode<double, 0>(a, s);
        case 1: return z_stage_mode<double, 1>(a, s);
        case 2: return z_stage_mode<double, 2>(a, s);
        case 3: return z_stage_mode<double, 3>(a, s);
        case 4: return z_stage_mode<double, 4>(a, s);
    }
    return cudaErrorInvalidValue;
}

template <>
cudaError_t z_stage_mixed<HQT_ZN>(int mode, const ZStageArgs<float> &a, cudaStream_t s) {
    switch (mode) {
        case 1: return z_stage_mode<float, 1>(a, s);
        case 2: return z_stage_mode<float, 2>(a, s);
        case 3: return z_stage_mode<float, 3>(a, s);
        case 4: return z_stage_mode<float, 4>(a, s);
    }
    return cudaErrorInvalidValue;
}

template <>
cudaError_t z_cons<HQT_ZN>(const ZConsArgs<double> &a, cudaStream_t s) {
    static int per_sm = 0, nsm = 0;
    constexpr int smem = ZcLay<HQT_ZN>::bytes;
    if (per_sm == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_zcons<HQT_ZN>, kZsThreads, smem);
        if (per_sm < 1) per_sm = 1;
    }
    const long long tiles = (a.plane + kZcSites - 1) / kZcSites;
    const long long full = (long long)per_sm * (nsm > 0 ? nsm : 1);
    (void)klaunch(k_zcons<HQT_ZN>, dim3((int)(tiles < full ? tiles : full)), dim3(kZsThreads),
                  smem, s, a);
    return cudaGetLastError();
}

template <>
cudaError_t z_misc<HQT_ZN>(const ZColArgs<double> &a, const ZHost &h, int grid, int threads,
                           cudaStream_t s) {
    const ZOps<double, HQT_ZN> op = make_zops(h);
    if (a.at) (void)klaunch(k_zcol_misc<double, HQT_ZN>, dim3(grid), dim3(threads), 0, s, a, op);
    if (a.psi) (void)klaunch(k_zcol_O<double, HQT_ZN>, dim3(grid), dim3(threads), 0, s, a, op);
    return cudaGetLastError();
}

}  // namespace hqt
