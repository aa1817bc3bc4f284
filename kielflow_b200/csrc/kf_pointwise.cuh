// kf_pointwise.cuh -- linear spectral terms, Poisson source, penalization window.
#pragma once

#include "kf_passes.cuh"
#include "kf_types.cuh"

namespace kf {

// -lin_q in k-space, lin_q being the part of rhs_standard's FBuffer_q (the
// negated right-hand side) that is computed there, in the reference's order of
// accumulation:
//   u_c: (tau+SV) u^ [+ D|k|^2 u^] + i k_c (PF phi^ + s^/theta) + M i k_x P u^
//        (rhs_standard.cpp:119-140, 218-248, 279-295)
//   s  : SV s^ [+ D|k|^2 s^] + M i k_x P s^ + i k.P u^
//        (rhs_standard.cpp:135-139, 304-319)
// k_lin: grid (ceil(nzc/32), n/8, n) of 32 x 8 blocks over (kz, j, i): no index
// division; the four outputs of an element share its loads (state, phi^, tables).
// The damping and diffusion sum's roundings are written out (k_zprod): in u_c the
// diffusion product is rounded first with penalization, the damping one without.
template <typename T>
__device__ __forceinline__ void lin_terms(const RhsArgs<T> &a, const Geo<T> &g, int i, int j, int k,
                                          typename C2<T>::type *o) {
    typedef typename C2<T>::type T2;
    const long idx = (long)k + (long)g.nzc * ((long)j + (long)i * g.n);
    const int Tm = a.terms;
    const bool P = dealias_keep(g.q2, g.thr, i, j, k);
    const T kx = g.kv[i], ky = g.kv[j], kz = g.kv[k];
    const T sv = a.SV[idx];
    const T2 u[3] = {a.Y[0][idx], a.Y[1][idx], a.Y[2][idx]};
    const T2 s = a.Y[3][idx];
    const bool diss = Tm & T_DISSIPATION, svo = Tm & T_SVISCOSITY;
    const bool pres = Tm & T_PRESSURE, eint = Tm & T_E_INT;
    // F1 = PF phi^ + s^/theta, the E-force/pressure potential (rhs_standard.cpp:218-248)
    T2 F1 = mk<T2>((T)0, (T)0);
    if (pres || eint) {
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
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const T cf = diss && svo ? (a.tau + sv) : diss ? a.tau : svo ? sv : (T)0;
        T2 fb = mk<T2>(mul_rn(cf, u[q].x), mul_rn(cf, u[q].y));
        if (Tm & T_DIFFUSION) {
            const T Dk = mul_rn(a.D, kx * kx + ky * ky + kz * kz);
            if (Tm & T_PENALIZATION)
                fb = mk<T2>(fma(cf, u[q].x, mul_rn(Dk, u[q].x)), fma(cf, u[q].y, mul_rn(Dk, u[q].y)));
            else
                fb = mk<T2>(fma(Dk, u[q].x, fb.x), fma(Dk, u[q].y, fb.y));
        }
        if (pres || eint) {
            const T kc = q == 0 ? kx : q == 1 ? ky : kz;
            const T2 d = mul_ik(F1, kc);
            fb.x += d.x;
            fb.y += d.y;
        }
        if ((Tm & T_E_EXT) && P) {
            const T2 d = mul_ik(u[q], kx);
            fb.x += a.M * d.x;
            fb.y += a.M * d.y;
        }
        o[q] = mk<T2>(-fb.x, -fb.y);
    }
    {
        const T cf = (Tm & T_SVISCOSITY) ? sv : (T)0;
        T2 fb = mk<T2>(mul_rn(cf, s.x), mul_rn(cf, s.y));
        if (Tm & T_DIFFUSION) {
            const T Dk = mul_rn(a.D, kx * kx + ky * ky + kz * kz);
            fb = mk<T2>(fma(Dk, s.x, fb.x), fma(Dk, s.y, fb.y));
        }
        if ((Tm & T_E_EXT) && P) {
            const T2 d = mul_ik(s, kx);
            fb.x += a.M * d.x;
            fb.y += a.M * d.y;
        }
        if ((Tm & T_CONTINUITY) && P) {
            const T2 dx = mul_ik(u[0], kx);
            const T2 dy = mul_ik(u[1], ky);
            const T2 dz = mul_ik(u[2], kz);
            fb.x += dx.x; fb.y += dx.y;
            fb.x += dy.x; fb.y += dy.y;
            fb.x += dz.x; fb.y += dz.y;
        }
        o[3] = mk<T2>(-fb.x, -fb.y);
    }
}

// The Hermitian part of the kz = 0 plane, which is what a way through physical
// space leaves of it (penalization): o holds four values of element (i, j, 0), m
// those of (-i, -j, 0)
template <typename T2> __device__ __forceinline__ void hermitian_part(T2 *o, const T2 *m) {
    typedef decltype(T2::x) T;
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = mk<T2>((T)0.5 * (o[q].x + m[q].x), (T)0.5 * (o[q].y - m[q].y));
}

// HERM: with the Hermitian part of the kz = 0 plane (hermitian_part) inside the 2/3
// rule, where the result is used.
template <typename T, bool HERM>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 8 : 4) k_lin(RhsArgs<T> a, Geo<T> g, typename C2<T>::type *o0,
                                             typename C2<T>::type *o1, typename C2<T>::type *o2,
                                             typename C2<T>::type *o3) {
    typedef typename C2<T>::type T2;
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= g.nzc || j >= g.n) return;
    const long idx = (long)k + (long)g.nzc * ((long)j + (long)i * g.n);
    // Where the Hermitian part is formed, the mirror's values go through the
    // element's own place, so that few registers live across the terms' code
    const bool h = HERM && k == 0 && dealias_keep(g.q2, g.thr, i, j, 0);
#pragma unroll 1
    for (int mirror = h ? 1 : 0; mirror >= 0; --mirror) {
        T2 o[4];
        lin_terms(a, g, mirror && i ? g.n - i : i, mirror && j ? g.n - j : j, k, o);
        if (h && !mirror) {
            const T2 m[4] = {o0[idx], o1[idx], o2[idx], o3[idx]};
            hermitian_part(o, m);
        }
        o0[idx] = o[0];
        o1[idx] = o[1];
        o2[idx] = o[2];
        o3[idx] = o[3];
    }
}

// The (i, j) rows on which the penalization mask is not zero, as the window
// box = {min i, max i, min j, max j} (started from {n, -1, n, -1}): outside it
// the penalization has no effect, so c2r(-lin_q) is needed on the window only.
template <typename T>
__global__ void __launch_bounds__(256) k_mask_box(const T *__restrict__ H, int n, int *__restrict__ box) {
    const int j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (j >= n) return;
    bool any = false;
    for (int k = threadIdx.x; k < n; k += 32) any |= H[((long)i * n + j) * n + k] != (T)0;
    if (any) {
        atomicMin(box + 0, i);
        atomicMax(box + 1, i);
        atomicMin(box + 2, j);
        atomicMax(box + 3, j);
    }
}

// rho = exp(s_d) + n_d in FP64 (rhs_standard.cpp:108-111)
template <typename T>
__global__ void k_rho(const T *__restrict__ sd, const double *__restrict__ nd, double *__restrict__ rho, long N) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) rho[i] = exp((double)sd[i]) + nd[i];
}

// x <- exp(x) (fn 0) or log(x) (fn 1) in place, evaluated in FP64: the
// density's linear <-> log scale (kielflow.cpp:172-182, 293-296)
template <typename T>
__global__ void k_explog(T *__restrict__ x, int fn, long N) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const double v = (double)x[i];
    x[i] = (T)(fn == 0 ? exp(v) : log(v));
}

// The real-space fields of an output file (IO.cpp save_field_imag and
// save_slice write iFFT of the spectra): u'_c, n = exp(s) from the c2r of the
// state, and phi, as FP64; all points (k0 < 0, o[q][id]) or the plane z
// index k0 only (o[q][j + n i]).
template <typename T>
__global__ void k_out_real(const T *__restrict__ ux, const T *__restrict__ uy, const T *__restrict__ uz,
                           const T *__restrict__ s, const double *__restrict__ phi, double *__restrict__ o0,
                           double *__restrict__ o1, double *__restrict__ o2, double *__restrict__ o3,
                           double *__restrict__ o4, int n, int k0, long M) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= M) return;
    const long src = k0 >= 0 ? i * n + k0 : i;
    o0[i] = (double)ux[src];
    o1[i] = (double)uy[src];
    o2[i] = (double)uz[src];
    o3[i] = exp((double)s[src]);
    o4[i] = phi[src];
}

// rho = n_background + n_d (the frontend's Poisson source)
__global__ void k_add_const(double *__restrict__ out, const double *__restrict__ in, double a, long N) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) out[i] = a + in[i];
}

// frontend.cpp:245-248: the Boltzmann ion density n = exp(-theta phi)
template <typename T>
__global__ void k_boltzmann(T *__restrict__ out, const double *__restrict__ phi, double theta, long N) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) out[i] = (T)exp(-theta * phi[i]);
}

// X *= f elementwise over a half spectrum (dealiasing_undesignated with a
// precomputed filter table, operations.hpp:20-46)
template <typename T>
__global__ void k_filter(typename C2<T>::type *__restrict__ X, const T *__restrict__ f, long Nc) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= Nc) return;
    typename C2<T>::type x = X[i];
    const T w = f[i];
    x.x *= w;
    x.y *= w;
    X[i] = x;
}

// FP64 <-> bulk precision conversion of interleaved complex / real arrays
template <typename T>
__global__ void k_from_f64(T *__restrict__ dst, const double *__restrict__ src, long M) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M) dst[i] = (T)src[i];
}
template <typename T>
__global__ void k_to_f64(double *__restrict__ dst, const T *__restrict__ src, long M) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < M) dst[i] = (double)src[i];
}

}  // namespace kf
