// hqt_zdims.h -- sizes and operand tables of the radial stage (hqt_zstage.cuh),
// shared by host and device.
#pragma once
#include "hqt_common.cuh"

namespace hqt {

constexpr int kZsCols = 16;  // columns of a tile
// Row pitches in shared memory (= widths of the TMA boxes) in bytes: kZsRow of an FP64 pair field,
// zs_row_td of a pair of type TD, zs_row_r of a real field of type TD.
constexpr int kZsRow = (kZsCols + 1) * 16;
template <typename TD> __host__ __device__ constexpr int zs_row_td() {
    return sizeof(TD) == 8 ? kZsRow : (kZsCols + 2) * 8;
}
template <typename TD> __host__ __device__ constexpr int zs_row_r() {
    return sizeof(TD) == 8 ? (kZsCols + 2) * 8 : (kZsCols + 4) * 4;
}

// The constraint kernel's tile (hqt_zcons.cuh): sites, row pitches of Psi and div A.
constexpr int kZcSites = 32, kZcRowP = (kZcSites + 2) * 16, kZcRowD = (kZcSites + 4) * 8;

// Levels whose rows of `bytes` bytes are no multiple of 16: TMA takes every n-th, a
// group of levels ph = l mod n per tensor map, whose base is rounded down by shift(ph)
// bytes.  In shared memory the groups follow each other, 128 bytes aligned, and an
// element of group ph lies shift(ph) bytes further into its row of `pitch` bytes.
struct ZsSplit {
    int n, lg, nz, pitch, low;  // groups, log2, levels; bytes mod 16
    __host__ __device__ __forceinline__ ZsSplit(int nz_, long long bytes, int pitch_)
        : lg(bytes % 16 == 0 ? 0 : bytes % 8 == 0 ? 1 : 2), nz(nz_), pitch(pitch_),
          low((int)(bytes % 16)) {
        n = 1 << lg;
    }
    __host__ __device__ __forceinline__ int shift(int ph) const { return (ph * low) & 15; }
    __host__ __device__ __forceinline__ int rows(int ph) const { return (nz - ph + n - 1) >> lg; }
    __host__ __device__ __forceinline__ int start(int ph) const {
        int o = 0;
        for (int p = 0; p < ph; ++p) o += (rows(p) * pitch + 127) / 128 * 128;
        return o;
    }
    __host__ __device__ __forceinline__ int at(int l) const {
        const int ph = l & (n - 1);
        return start(ph) + (l >> lg) * pitch + shift(ph);
    }
};

// Polls of a wait for a copy before it counts as lost: about a second.
constexpr int kZsPolls = 1 << 20;

// Row g of an mma tile stands for level 8m + zs_row(g) (bits 0 and 1 swapped).
__host__ __device__ constexpr int zs_row(int g) { return (g & 4) | ((g & 1) << 1) | ((g >> 1) & 1); }

template <int NZP> struct ZsDims {
    static constexpr int HE = (NZP + 1) / 2, HO = NZP / 2;  // even, odd halves
    static constexpr int MH = (HE + 7) / 8, MP = (HO + 7) / 8;
    static constexpr int KE = (HE + 3) / 4, KO = (HO + 3) / 4;
    static constexpr int M1 = (NZP - 1 + 7) / 8, K1 = (NZP - 1 + 3) / 4;
    static constexpr int ntab = 3 * NZP + 4 * KE;  // z, f, Lz(nz,:), line factors
    static constexpr int VR = NZP > 4 * K1 ? NZP : 4 * K1;  // rows of a scratch field
    static constexpr int nfrag = MP * KE + MH * KO + M1 * K1;
    // state and accumulator are read straight from global memory instead of staged
    // where staging them would leave one block per SM
    static constexpr bool direct = NZP > 25;
    static constexpr int min_blocks = 2;
};

}  // namespace hqt
