// hqt_args.h -- kernel argument blocks (plain structs, host and device).
#pragma once
#include <cuda.h>

#include "hqt_common.cuh"
#include "hqt_lineplan.h"

namespace hqt {

constexpr int kMaxFilt = 4;

template <typename T> struct FieldIn {
    const C2<T> *c;  // interleaved complex source, or
    const T *re;     // split real / imaginary sources (im may be null),
    const T *im;
    int st = 1;  // elements st apart (2: one part of an interleaved pair; only
                 // for a real field, im null)
};

template <typename T> struct FieldOut {
    C2<T> *c;  // interleaved, and/or
    T *re;     // split parts (each may be null),
    T *im;
    int st = 1;  // elements st apart (2: one part of an interleaved pair; only
                 // for a real field, c and im null)
};

// A first derivative of one real field into one real field: the line
// passes then carry two real lines per complex transform (the multiplier
// ik is a real operator, so a transform of A + iB gives dA + i dB).
template <typename T>
__host__ __device__ inline bool real_field_d1(const FieldIn<T> &in, const FieldOut<T> &out) {
    return in.re && !in.im && !in.c && out.re && !out.im && !out.c;
}

template <typename T> struct XRhsArgs {
    LineTab<T> lt;  // in-place transforms
    FFTPlan plan;
    const C2<T> *roots;
    int NB, nlines;
    T s1, s2;
    const C2<T> *psi;
    const C2<T> *A;  // (A_x, A_y)
    C2<T> *dxpsi, *dxxpsi, *E;
    T *dxxay;
};

template <typename T> struct YRhsArgs {
    LineTab<T> lt;  // in-place transforms
    FFTPlan plan;
    const C2<T> *roots;
    int TX, nx, ny;
    T s1, s2;
    const C2<T> *psi;
    const C2<T> *A;  // (A_x, A_y)
    const C2<T> *E;  // d_x A_x + i d_x A_y
    const T *dxxay;
    C2<T> *dypsi, *dyypsi;  // (the radial stage forms lap Psi = d_xx Psi + d_yy Psi)
    T *divA;
    C2<T> *B;  // (d_y B, d_x B)
};

template <typename T> struct XD1Args {
    LineTab<T> lt;  // in-place transforms
    FFTPlan plan;
    const C2<T> *roots;
    int NB, nlines;
    T s1;
    FieldIn<T> in;
    FieldOut<T> out;
};

template <typename T> struct YD1Args {
    LineTab<T> lt;  // in-place transforms
    FFTPlan plan;
    const C2<T> *roots;
    int TX, nx, ny;
    T s1;
    FieldIn<T> in;
    const T *add_re;  // optional: out.re = add_re + Re(d_y in)
    FieldOut<T> out;
};

template <typename T> struct XFiltFwdArgs {
    LineTab<T> lt;  // in-place transforms
    FFTPlan plan;
    const C2<T> *roots;
    int NB, nlines, ny;
    int nf;
    FieldIn<T> in[kMaxFilt];
    C2<T> *spec[kMaxFilt];
    const DevStatus *st;  // phase e^{-2 pi i y w/ny} on field 0 when non-null
    int dead0 = 1, dead1 = 0;  // spectral columns dead0 <= kx <= dead1 may be left
                               // unwritten (prime-factor engine; empty by default)
};

template <typename T> struct YFiltArgs {
    LineTab<T> lt;  // in-place transforms
    FFTPlan plan;
    const C2<T> *roots;
    int TX, nx, ny;
    int nf;
    C2<T> *spec[kMaxFilt];
    const T *mx, *my;  // 1 - fx, 1 - fy
    T scale;           // 1/(nx*ny)
    int dead0 = 1, dead1 = 0;  // columns dead0 <= kx <= dead1 are zero after the weight
    // optional: the weighted (0,0) coefficient of field f's real and imaginary
    // parts, i.e. the slice means of the filtered field, go to
    // slice_mean[5*z + slot[f][c]] (slot < 0: not written)
    T *slice_mean = nullptr;
    int slot[kMaxFilt][2] = {};
};

template <typename T> struct XFiltInvArgs {
    LineTab<T> lt;  // in-place transforms
    FFTPlan plan;
    const C2<T> *roots;
    int NB, nlines;
    int nf;
    const C2<T> *spec[kMaxFilt];
    FieldOut<T> out[kMaxFilt];
    DevStatus *st;  // non-finite check when non-null
    // optional FP32 copies minus the slice means (slice_mean[5*z + slot]):
    // interleaved c32[f], or re32[f]; z = line / ny
    const T *slice_mean = nullptr;
    int slot[kMaxFilt][2] = {};
    int ny = 0;
    C2<float> *c32[kMaxFilt] = {};
    float *re32[kMaxFilt] = {};
    int dead0 = 1, dead1 = 0;  // spectral columns dead0 <= kx <= dead1 read as zero
};

template <typename T, int NZP> struct ZOps {
    T Lz[NZP][NZP];
    T Lz1[NZP][NZP];
    T zz[NZP];
    T fz[NZP];   // 1 - z^3
    T lzb[NZP];  // boundary row Lz(nz, :)
};

// Radial stage (hqt_zstage.cuh).  TD: type of the horizontal-derivative fields
// written by the line passes; all else is FP64.  Pairs of real fields are
// interleaved.  Inputs come by the tensor maps, one per group of levels (ZsSplit).
template <typename TD> struct ZStageArgs {
    CUtensorMap mPS, mAXY;        // stage input Psi, (A_x, A_y)
    CUtensorMap mDX[2], mDY[2];   // d_x Psi, d_y Psi
    CUtensorMap mDT[2], mB[2];    // (d_x A_t, d_y A_t), (d_y B, d_x B)
    CUtensorMap mZA, mKA;         // state and RK accumulator of (A_x, A_y)
    CUtensorMap mATD;             // (A_t, d_z A_t)
    CUtensorMap mXX[2], mYY[2];   // d_xx Psi, d_yy Psi (their sum is lap Psi)
    CUtensorMap mDIV[4];          // div A
    CUtensorMap mZP, mKP;         // state and RK accumulator of Psi
    int nz;
    long long plane;  // nx*ny
    double h;
    const double *frag;  // operator fragments per lane (z_tables)
    const double *ztab;  // z, 1 - z^3, Lz(nz,:), NZP each
    const double2 *ypsi, *yA, *atd;
    const C2<TD> *dxpsi, *dypsi, *dAt, *B, *dxxpsi, *dyypsi;
    const TD *divA;
    const double2 *zpsi, *zA;
    const double *zrho;
    double2 *kpsi, *kA;
    double *krho;
    double2 *npsi, *nA;       // next stage input
    C2<TD> *npsi_d, *nA_d;    // its copy in the derivative type (TD float only),
    // minus the plane means of its z slice (psi re, psi im, A_t, A_x, A_y): the
    // line passes only differentiate, and the smaller magnitude rounds to FP32
    // with a smaller error
    const double *slice_mean;
    double2 *wpsi, *wA;       // new state (stage 4)
    double *wrho;
    double2 *f1;              // right-hand-side outputs (MODE 0)
    double *f3, *f4, *f2b;
    int *fault;               // set when a copy did not arrive
    int polls;                // of a wait for a copy before it counts as lost
};

template <typename T> struct ZConsArgs {
    int nz;
    long long plane;
    T mu, vy;
    C2<T> *psi;
    C2<T> *A;    // (A_x, A_y): boundary row
    C2<T> *atd;  // (A_t, d_z A_t)
    const T *divA;
    const T *rho;  // 2-D
    C2<T> *O;      // 2-D boundary order parameter (may be null)
    const double *frag, *ztab;  // operand tables (hqt_zdims.h)
    int *fault;                 // set when a copy did not arrive
    int polls;                  // of a wait for a copy before it counts as lost
    CUtensorMap mPS, mDIV[2];   // Psi, div A (ZsSplit)
};

template <typename T> struct ZColArgs {
    int nz;
    long long plane;
    const T *at;
    C2<T> *atd;  // (A_t, d_z A_t) of at
    const C2<T> *psi;
    C2<T> *O;
};

}  // namespace hqt
