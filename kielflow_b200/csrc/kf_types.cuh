// kf_types.cuh -- argument blocks shared by the kernels and the host driver.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

#include "kf_fft.cuh"

namespace kf {

// Multipliers applied to a spectral element as it is loaded by a pass.
enum Mul : int {
    MUL_NONE = 0,   // 1
    MUL_P = 1,      // 2/3 dealiasing mask P(k)            (x pass only: needs i, j, k)
    MUL_P_IK = 2,   // P(k) * i k_axis                     (x pass only)
    MUL_IK = 3,     // i k_axis  (k of the pass's own axis)
    MUL_HALF = 4,   // z c2r only: 1/2 for 0 < kz < n/2 (the half-spectrum weight of a transpose)
};

// Term bits (runtime form of rhs_standard.hpp:22-30 plus the added terms).
enum Term : int {
    T_POISSON = 1 << 0, T_DISSIPATION = 1 << 1, T_SVISCOSITY = 1 << 2, T_E_INT = 1 << 3,
    T_PRESSURE = 1 << 4, T_E_EXT = 1 << 5, T_CONTINUITY = 1 << 6, T_ADVECTION = 1 << 7,
    T_PENALIZATION = 1 << 8, T_DIFFUSION = 1 << 9,
};

// One batched 1-D transform along x or y: in -> out with a load multiplier.
struct AxisJob {
    const void *in;
    void *out;
    int mul;
    int pad_;
};

// One z-axis real transform pair: two real rows <-> one complex line.
// c2r: half spectra inA/inB (multiplied by mulA/mulB) -> real rows outA/outB;
// r2c: real rows inA/inB -> half spectra outA/outB.  inB == nullptr: single row.
struct ZJob {
    const void *inA, *inB;
    void *outA, *outB;
    int mulA, mulB;
};

// Grid geometry and axis tables, valid for all three axes of the cubic box.
template <typename T> struct Geo {
    int n, nzc;
    const T *kv;       // k_val_at(i), i < n                        (axis_EqSt.cpp:57-61)
    const double *q2;  // pow(k_val_at(i)/k_val_at(n/2), 2.), i < n  (OP_dealiasing.hpp:24-28)
    double thr;        // smallest double s with sqrt(s) >= 2/3 (see dealias_threshold)
    const int *pb;     // per (j, kz) column: the 2/3 rule along i as a bound (dealias_bounds), or nullptr
};

// Which part of a half spectrum an x / y pass moves (uniform over a launch).
// The 2/3 rule keeps a ball of radius n/3: 16 % of a half spectrum, the columns
// (j, kz) of a disc (35 %) once x is transformed, kz < nkz (67 %) once y is.
// A pass over a masked field reads, transforms and writes only those parts; the
// next pass knows that the rest is zero and does not read it.
enum AxMode : int {
    AX_FULL = 0,  // everything
    AX_XM = 1,    // x pass, masked input: active columns, rows within the column's bound -> every row
    AX_YI = 2,    // y pass after AX_XM: columns kz < nkz, rows j within jb[kz] -> every row
    AX_YF = 3,    // forward y pass whose x pass needs only active columns: every row -> rows within jb[kz]
    AX_XB = 4,    // x pass of which the window's planes are needed: every row -> these, packed
    AX_YB = 5,    // y pass after AX_XB, on the window's planes: every row -> the window's rows, packed
    AX_XF = 6,    // forward x pass after AX_YF: active columns, every row
};
// The window of rows (i, j) on which the mask is not zero, as k_mask_box leaves it
// (min i, max i, min j, max j; nullptr: none).  Kernels read it from there, so
// that captured steps do not depend on it.
struct RowBox {
    int i0, bi, j0, bj;
    __device__ __forceinline__ explicit RowBox(const int *__restrict__ b) : i0(0), bi(0), j0(0), bj(0) {
        if (b && __ldg(b + 1) >= 0) {
            i0 = __ldg(b);
            bi = __ldg(b + 1) - i0 + 1;
            j0 = __ldg(b + 2);
            bj = __ldg(b + 3) - j0 + 1;
        }
    }
    __device__ __forceinline__ bool has(int i, int j) const {
        return (unsigned)(i - i0) < (unsigned)bi && (unsigned)(j - j0) < (unsigned)bj;
    }
    __device__ __forceinline__ int row(int i, int j) const { return (i - i0) * bj + j - j0; }
};

struct AxTrunc {
    int mode;
    int nkz;        // columns kz < nkz are active
    float itpp;     // 1 / column tiles per plane of AX_YI, AX_YF
    const int *jb;  // per kz < nkz: largest min(j, n - j) of an active column
    const int *tl;  // active x-pass tiles: (j << 16) | first kz
    const int *win; // AX_XB, AX_YB: the window's planes i, rows j (RowBox)
    // elements per (i, j) row of the input and the output: n/2 + 1, or for the
    // masked passes' intermediates nkz rounded up to whole tiles, so that tiles are
    // aligned 128-byte segments (a row of n/2 + 1 elements shifts them across lines)
    int ip, op;
};

// sqrt is correctly rounded and monotone, so sqrt(s) < 2/3 holds exactly when
// s < thr for the smallest double thr with sqrt(thr) >= 2/3: the 2/3 rule of
// rhs_standard.cpp:22 on |k~| (OP_dealiasing.hpp:28) without a square root.
inline double dealias_threshold() {
    const double c = 2. / 3.;
    double s = c * c;
    while (!(std::sqrt(s) < c)) s = std::nextafter(s, 0.);
    while (std::sqrt(s) < c) s = std::nextafter(s, 1.);
    return s;
}

// 2/3 rule of rhs_standard.cpp:22 on the exact |k~|^2 = (q2[i] + q2[j]) + q2[k].
__device__ __forceinline__ bool dealias_keep(const double *__restrict__ q2, double thr, int i, int j, int k) {
    return __dadd_rn(__dadd_rn(q2[i], q2[j]), q2[k]) < thr;
}

// The 2/3 rule along the x axis of one (j, kz) column as a bound: keep(i) ==
// (min(i, n - i) <= b), with b from the host table dealias_bounds (which checks
// that equivalence for every i of the column and stores -2 where it does not
// hold); -2 or no table: the exact sum of dealias_keep per element.
__device__ __forceinline__ int dealias_bound(const int *__restrict__ pb, int jj, int kk, int nzc) {
    return pb ? pb[jj * nzc + kk] : -2;
}
__device__ __forceinline__ bool dealias_keep_b(const double *__restrict__ q2, double thr, int b, int n, int i, int j,
                                               int k) {
    if (b >= -1) return (i <= n / 2 ? i : n - i) <= b;
    return dealias_keep(q2, thr, i, j, k);
}

// Everything the spectral linear terms need.
template <typename T> struct RhsArgs {
    typedef typename C2<T>::type T2;
    const T2 *Y[4];     // stage input: u'_x, u'_y, u'_z, s  (half spectra)
    const T2 *phihat;   // r2c(phi), unnormalised
    const T *SV;        // spectral-viscosity table field_SV (rhs_standard.cpp:57-71), cut applied
    const T *PF;        // phi filter exp(-2000 |k~_Q1|^15) (operations.hpp:20-46)
    T tau, theta, M, D;
    int terms;
};

}  // namespace kf
