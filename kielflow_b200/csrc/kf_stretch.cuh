// kf_stretch.cuh -- pointwise kernels of the right-hand side on sine-stretched
// axes (axis_CoSiSt, axis_SiSt.cpp).  There a derivative is the chain-rule
// form of OP_partial_derivative.cpp:104-136,
//   D_d F = r2c( m(x_d) * c2r( P i k_d F ) ),
// m = 1/dS of the axis after the 2/3 filter (OP_partial_derivative.cpp:60-80),
// so every derivative costs a transform pair; the transforms run as batched
// passes (kf_passes.cuh) and these kernels do the pointwise work between them.
#pragma once

#include "kf_passes.cuh"
#include "kf_pointwise.cuh"
#include "kf_types.cuh"

namespace kf {

// -1 x the linear spectral parts of FBuffer (no derivative; rhs_standard.cpp:119-140
// and the added diffusion) and the potential of the E-force/pressure term
// F1 = PF phi^ + s^/theta (rhs_standard.cpp:218-240), one thread per
// half-spectrum element.  Same order of operations as lin_terms.
// herm: with the Hermitian part of the kz = 0 plane, as k_lin.
template <typename T>
__device__ __forceinline__ void sl_lin_terms(const RhsArgs<T> &a, const Geo<T> &g, int i, int j, int k,
                                             typename C2<T>::type *o) {
    typedef typename C2<T>::type T2;
    const long idx = (long)k + (long)g.nzc * ((long)j + (long)i * g.n);
    const int Tm = a.terms;
    const T kx = g.kv[i], ky = g.kv[j], kz = g.kv[k];
    const T sv = a.SV[idx];
    const bool diss = Tm & T_DISSIPATION, svo = Tm & T_SVISCOSITY;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const T2 y = a.Y[q][idx];
        const T cf = q < 3 && diss ? (svo ? a.tau + sv : a.tau) : svo ? sv : (T)0;
        T2 fb = mk<T2>(cf * y.x, cf * y.y);
        if (Tm & T_DIFFUSION) {
            const T k2 = kx * kx + ky * ky + kz * kz;
            fb.x += a.D * k2 * y.x;
            fb.y += a.D * k2 * y.y;
        }
        o[q] = mk<T2>(-fb.x, -fb.y);
    }
}

template <typename T>
__global__ void k_sl_lin(RhsArgs<T> a, Geo<T> g, typename C2<T>::type *l0, typename C2<T>::type *l1,
                         typename C2<T>::type *l2, typename C2<T>::type *l3, typename C2<T>::type *F1o, bool herm) {
    typedef typename C2<T>::type T2;
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long Nc = (long)g.n * g.n * g.nzc;
    if (idx >= Nc) return;
    const int k = (int)(idx % g.nzc);
    const long r = idx / g.nzc;
    const int j = (int)(r % g.n), i = (int)(r / g.n);
    T2 o[4];
    sl_lin_terms(a, g, i, j, k, o);
    if (herm && k == 0 && dealias_keep(g.q2, g.thr, i, j, 0)) {
        T2 m[4];
        sl_lin_terms(a, g, i ? g.n - i : 0, j ? g.n - j : 0, 0, m);
        hermitian_part(o, m);
    }
    l0[idx] = o[0];
    l1[idx] = o[1];
    l2[idx] = o[2];
    l3[idx] = o[3];
    const int Tm = a.terms;
    const T2 s = a.Y[3][idx];
    T2 F1 = mk<T2>((T)0, (T)0);
    const bool pres = Tm & T_PRESSURE, eint = Tm & T_E_INT;
    if (eint) {
        const T pf = pres ? a.PF[idx] : (T)1;
        if (pf != (T)0) F1 = a.phihat[idx];  // (not formed where PF is 0)
        F1.x *= pf;
        F1.y *= pf;
    }
    if (pres) {
        F1.x += s.x / a.theta;
        F1.y += s.y / a.theta;
    }
    F1o[idx] = F1;
}

// The raw derivatives c2r(P i k_d F) times the metric of their direction
// (OP_partial_derivative.cpp:125-127): f[j] along axis j % 3 (j = 3c + d for
// d_d u'_c, 9 + d for d_d s) in place, as the products want them projected once
// more; and what the right-hand side adds of them as they are, before its one
// transform of the sum (rhs_standard.cpp:218-319):
//   S_c = D_c F1 + M D_x u'_c        S_3 = M D_x s + D_x u'_x + D_y u'_y + D_z u'_z
// Memory-bound: 15 fields in, 16 out.
template <typename T> struct ScaleArgs {
    T *f[12], *S[4];
    const T *F1[3], *met;
    T M;
    int n, terms;
    long N;
};

template <typename T>
__global__ void __launch_bounds__(256) k_sl_scale(ScaleArgs<T> a) {
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= a.N) return;
    const int k = (int)(idx % a.n);
    const long r = idx / a.n;
    const int j = (int)(r % a.n), i = (int)(r / a.n);
    const T m[3] = {a.met[i], a.met[j], a.met[k]};
    const bool force = a.terms & (T_PRESSURE | T_E_INT), ext = a.terms & T_E_EXT;
    T f[12], F1[3];
#pragma unroll
    for (int q = 0; q < 12; ++q) f[q] = a.f[q][idx];
#pragma unroll
    for (int q = 0; q < 3; ++q) F1[q] = force ? a.F1[q][idx] : (T)0;
#pragma unroll
    for (int q = 0; q < 12; ++q) {
        f[q] *= m[q % 3];
        a.f[q][idx] = f[q];
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) a.S[q][idx] = F1[q] * m[q] + (ext ? a.M * f[3 * q] : (T)0);
    T s = ext ? a.M * f[9] : (T)0;
    if (a.terms & T_CONTINUITY) s += f[0] + f[4] + f[8];
    a.S[3][idx] = s;
}

// The physical part of the right-hand side, out_q (S_q on entry) ->
//   t_c = S_c + u.grad u_c, t_3 = S_3 + u.grad s   (rhs_standard.cpp:323-436)
// as -t_q or, where the mask H is not zero (on the window of rows that bounds it,
// with l_q = c2r(-lin_q) there), the masking form (effect_penalization.cpp:35)
//   (1-H)(l_q - t_q) + H eta (q_d - q_fix) - l_q,  q_fix = (-M, 0, 0, -10),
// so that the right-hand side is -lin_q plus the transform of out_q.
// Memory-bound: 23 fields a point with all terms.
template <typename T> struct SlProdArgs {
    const T *U[3], *dU[3][3], *ds[3];  // dU[c][d] = D_d U_c, ds[d] = D_d s
    const T *sd, *H, *rl[4];           // penalization: c2r(P s^), the mask, l_q on the window
    T *out[4];
    T M, eta;
    const int *box;  // the mask's window (RowBox)
    int terms, n;
    long N;
};

template <typename T>
__global__ void __launch_bounds__(256) k_sl_products(SlProdArgs<T> a) {
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= a.N) return;
    const bool adv = a.terms & T_ADVECTION, cont = a.terms & T_CONTINUITY;
    T t[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) t[q] = a.out[q][idx];
    const int row = (int)(idx / a.n), i = row / a.n, j = row % a.n;
    const RowBox box(a.box);
    const T h = box.has(i, j) ? a.H[idx] : (T)0;
    T u[3] = {};
    if (adv || cont || h != (T)0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) u[d] = a.U[d][idx];
    }
    if (adv) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            T s = u[0] * a.dU[c][0][idx];
            s += u[1] * a.dU[c][1][idx];
            s += u[2] * a.dU[c][2][idx];
            t[c] += s;
        }
    }
    if (cont) {
        T s = a.ds[0][idx] * u[0];
        s += a.ds[1][idx] * u[1];
        s += a.ds[2][idx] * u[2];
        t[3] += s;
    }
    if (h != (T)0) {
        const T qd[4] = {u[0], u[1], u[2], a.sd[idx]};
        const T qfix[4] = {-a.M, (T)0, (T)0, (T)-10};
        const long w = (long)box.row(i, j) * a.n + idx % a.n;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const T l = a.rl[q][w], r = l - t[q];
            a.out[q][idx] = (((T)1 - h) * r + h * a.eta * (qd[q] - qfix[q])) - l;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) a.out[q][idx] = -t[q];
    }
}

// The 2/3 filter between the two x passes of P r2c(m c2r(..)): one block takes an
// active column tile of one field through the forward transform, drops what the
// rule does not keep and transforms back, so the spectrum itself is never stored.
// As k_xfwd_stage, a block holds one tile in registers and one in shared memory;
// bound by the two transforms' issue.  With the sums in physical space it took a
// 128^3 FP32 step from 6.6 to 5.4 ms.
template <typename T, int N, int V = 0>
__global__ void __launch_bounds__(Tile<T>::TC * PlanV<N, V>::P,
                                  PipeMinBlocks<T, N, V, 1, sizeof(T) == 4 ? 4 : 2, 64>::value)
k_x_filter(const AxisJob *__restrict__ jobs, int njobs, Geo<T> g, const typename C2<T>::type *__restrict__ tw,
           AxTrunc A) {
    typedef typename C2<T>::type T2;
    constexpr int TC = Tile<T>::TC, P = PlanV<N, V>::P, E = N / P, NZC = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *sm = reinterpret_cast<T2 *>(kf_smem);
    const AxisJob J = jobs[blockIdx.x % njobs];
    const int w = A.tl[blockIdx.x / njobs];
    const int c = threadIdx.x % TC, p = threadIdx.x / TC;
    const int kk = (w & 0xffff) + c, col = (w >> 16) * A.op + kk, rs = N * A.op;
    const int b = kk < A.nkz ? g.pb[(w >> 16) * NZC + kk] : -1;
    const T2 *in = static_cast<const T2 *>(J.in);
    T2 v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int row = reg_row<N, P, PlanV<N, V>::R1>(p, e);
        v[e] = b >= 0 ? in[col + row * rs] : mk<T2>((T)0, (T)0);
    }
    PlanV<N, V>::template fft<T2, -1>(v, sm + c, StrideAddr{TC}, p, tw);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int row = reg_row<N, P, PlanV<N, V>::RL>(p, e);
        sm[row * TC + c] = row_freq<N>(row) <= b ? v[e] : mk<T2>((T)0, (T)0);
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = sm[reg_row<N, P, PlanV<N, V>::R1>(p, e) * TC + c];
    __syncthreads();
    PlanV<N, V>::template fft<T2, +1>(v, sm + c, StrideAddr{TC}, p, tw);
    if (b < 0) return;
    T2 *out = static_cast<T2 *>(J.out);
#pragma unroll
    for (int e = 0; e < E; ++e) out[col + reg_row<N, P, PlanV<N, V>::RL>(p, e) * rs] = v[e];
}

}  // namespace kf
