// kf_jacobi.cuh -- the reference's nonlinear Jacobi relaxation
// (solver_poisson_jacobi_nlin.cpp:50-265) with its sweep loop on the device.
//
// A sweep is one kernel: the point updates, the sweep's statistics reduced in a
// fixed order (block trees, then one tree over the blocks' partials by the block
// that finishes last), Carre's over-relaxation factor and the stop test.  The
// loop is a conditional WHILE node whose body holds JC_UNROLL sweeps, which
// return at once when an earlier one has stopped; the host reads the record back
// once per solve.  A host-driven sweep (two launches, a copy and a
// synchronisation) took 27 us at 32^3.
#pragma once

#include "kf_poisson.cuh"

namespace kf {

// The relaxation's record (members of solver_poisson_jacobi_nlin.hpp:66-95):
// norm_max ... omega carry over between sweeps and solves.
struct JacState {
    double norm_max, norm_sum, norm_max_old, norm_sum_old, sup, inf, omega, rlast;
    int iteration, done, converged, nan;
    unsigned ticket, pad;
};

struct JacStop {
    int max_it, resstop;
    double limit, tol;  // relative-update limit; residual target (resstop)
};

// num / den with r = 1 / den rounded to nearest: Markstein's correction
// (P. Markstein, IBM J. Res. Dev. 34, 1990): with q within an ulp,
// q + r (num - q den) is num / den correctly rounded; one step brings num r there.
__device__ __forceinline__ double div_by(double num, double den, double r) {
    double q = __dmul_rn(num, r);
    q = __fma_rn(__fma_rn(-q, den, num), r, q);
    return __fma_rn(__fma_rn(-q, den, num), r, q);
}

// point_coeffs: the same quotients and sums, the divisors' reciprocals from tables
__device__ __forceinline__ void point_coeffs_div(const double *__restrict__ p, const double *__restrict__ rho,
                                                 const Lev &L, int i, int j, int k, double &A, double &D) {
    const int n = L.n;
    D = __dadd_rn(__dadd_rn(L.dd[i], L.dd[j]), L.dd[k]);
    A = div_by(p[lidx(wrapi(i + 1, n), j, k, n)], L.dp[i], L.rp[i]);
    A = __dadd_rn(A, div_by(p[lidx(wrapi(i - 1, n), j, k, n)], L.dm[i], L.rm[i]));
    A = __dadd_rn(A, div_by(p[lidx(i, wrapi(j + 1, n), k, n)], L.dp[j], L.rp[j]));
    A = __dadd_rn(A, div_by(p[lidx(i, wrapi(j - 1, n), k, n)], L.dm[j], L.rm[j]));
    A = __dadd_rn(A, div_by(p[lidx(i, j, wrapi(k + 1, n), n)], L.dp[k], L.rp[k]));
    A = __dadd_rn(A, div_by(p[lidx(i, j, wrapi(k - 1, n), n)], L.dm[k], L.rm[k]));
    A = __dmul_rn(2., A);
    A = __dadd_rn(A, rho[lidx(i, j, k, n)]);
}

// newton_method::solve (newton_method.hpp:16-63), eps 0.05, Nmax 20, g 0.8; f0 =
// f(x) at entry.  The method's first pass moves by omega * 0, so it repeats the
// evaluation it starts from: f(x), its step and exp(x) are formed once.
__device__ __forceinline__ double newton_point(double x, double A, double D, double &f0) {
    const double g = 0.8;
    double ex = exp(x);
    f0 = __dsub_rn(__dsub_rn(A, __dmul_rn(D, x)), ex);
    double dx = f0 / __dsub_rn(-D, ex), dx_alt = dx;
    double omega = __dadd_rn(1. - g, g * 1.);
    for (int i = 1; fabs(dx) > 0.05 && i < 20; ++i) {
        x = __dsub_rn(x, __dmul_rn(omega, dx));
        ex = exp(x);
        dx = __dsub_rn(__dsub_rn(A, __dmul_rn(D, x)), ex) / __dsub_rn(-D, ex);
        omega = fabs(dx) > fabs(dx_alt) ? __dmul_rn(g, omega) : __dadd_rn(__dmul_rn(1. - g, omega), g * 1.);
        dx_alt = dx;
    }
    return __dsub_rn(x, dx);
}

// Block partials of a sweep's statistics: [0] max|dP|, [1] sum|dP|, [2] max P_new,
// [3] min P_new, [4] max|f(P_old)|.  Tree over BS values per slot, t taking t + w
// for w = BS/2, ..., 1, the last five levels by warp shuffle.
template <int BS>
__device__ __forceinline__ void jac_tree(double v[KF_RED], double (*sh)[BS]) {
    const int t = threadIdx.x;
    for (int s = 0; s < KF_RED; ++s) sh[s][t] = v[s];
    __syncthreads();
#pragma unroll
    for (int w = BS / 2; w >= 32; w >>= 1) {
        if (t < w) {
            v[0] = nmax(v[0], sh[0][t + w]);
            v[1] = __dadd_rn(v[1], sh[1][t + w]);
            v[2] = nmax(v[2], sh[2][t + w]);
            v[3] = nmin(v[3], sh[3][t + w]);
            v[4] = nmax(v[4], sh[4][t + w]);
            if (w > 32)
                for (int s = 0; s < KF_RED; ++s) sh[s][t] = v[s];
        }
        if (w > 32) __syncthreads();
    }
    if (t < 32) {
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
            v[0] = nmax(v[0], __shfl_down_sync(0xffffffffu, v[0], w));
            v[1] = __dadd_rn(v[1], __shfl_down_sync(0xffffffffu, v[1], w));
            v[2] = nmax(v[2], __shfl_down_sync(0xffffffffu, v[2], w));
            v[3] = nmin(v[3], __shfl_down_sync(0xffffffffu, v[3], w));
            v[4] = nmax(v[4], __shfl_down_sync(0xffffffffu, v[4], w));
        }
    }
}

// One sweep in -> out.  cond: the last sweep of the loop's body sets the WHILE
// condition h.
template <int BS>
__global__ void __launch_bounds__(BS) k_jacobi(const double *__restrict__ in, double *__restrict__ out,
                                               const double *__restrict__ rho, Lev L, JacStop S,
                                               double *__restrict__ partial, JacState *js, int cond,
                                               cudaGraphConditionalHandle h) {
    __shared__ double sh[KF_RED][BS];
    __shared__ bool last;
    if (js->done) {
        if (cond && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(h, 0u);
        return;
    }
    const double omega = js->omega;
    const int n = L.n;
    const long N = (long)n * n * n;
    double v[KF_RED] = {0., 0., -INFINITY, INFINITY, 0.};
    if (blockIdx.x == 0 && threadIdx.x == 0) v[2] = v[3] = in[0];  // supremum = infinum = in.val[0] (:158-159)
    for (long id = (long)blockIdx.x * BS + threadIdx.x; id < N; id += (long)gridDim.x * BS) {
        const unsigned u = (unsigned)id;
        const int k = (int)(u % (unsigned)n);
        const unsigned r = u / (unsigned)n;
        const int j = (int)(r % (unsigned)n), i = (int)(r / (unsigned)n);
        double A, D;
        point_coeffs_div(in, rho, L, i, j, k, A, D);
        const double P_old = in[id];
        double f0;
        const double P_new = newton_point(P_old, A, D, f0);
        const double delta = fabs(__dsub_rn(P_new, P_old));
        out[id] = __dadd_rn(__dmul_rn(1. - omega, P_old), __dmul_rn(omega, P_new));
        v[0] = nmax(v[0], delta);
        v[1] = __dadd_rn(v[1], delta);
        v[2] = nmax(v[2], P_new);
        v[3] = nmin(v[3], P_new);
        v[4] = nmax(v[4], fabs(f0));
    }
    jac_tree<BS>(v, sh);
    if (threadIdx.x == 0) {
        for (int s = 0; s < KF_RED; ++s) partial[(long)blockIdx.x * KF_RED + s] = v[s];
        __threadfence();
        last = atomicAdd(&js->ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double w[KF_RED] = {0., 0., -INFINITY, INFINITY, 0.};
    for (int b = threadIdx.x; b < (int)gridDim.x; b += BS) {
        const double *p = partial + (long)b * KF_RED;
        w[0] = nmax(w[0], __ldcg(p));
        w[1] = __dadd_rn(w[1], __ldcg(p + 1));
        w[2] = nmax(w[2], __ldcg(p + 2));
        w[3] = nmin(w[3], __ldcg(p + 3));
        w[4] = nmax(w[4], __ldcg(p + 4));
    }
    __syncthreads();
    jac_tree<BS>(w, sh);
    if (threadIdx.x != 0) return;
    js->ticket = 0;
    const int iteration = js->iteration + 1;
    js->norm_sum_old = js->norm_sum;
    js->norm_max_old = js->norm_max;
    js->sup = w[2];
    js->inf = w[3];
    js->rlast = w[4];
    const double norm_max = w[0], norm_sum = w[1] / (double)N;
    bool nan = w[4] != w[4] || w[0] != w[0], done = nan, conv = false;
    // Carre's over-relaxation factor (:237-252)
    double om = .5;
    if (norm_max < js->norm_max_old && iteration > 1) {
        const double lambda = norm_sum / js->norm_sum_old;
        const double a = __dsub_rn(__dadd_rn(lambda, omega), 1.);
        om = 2. / __dadd_rn(1., sqrt(__dsub_rn(1., __dmul_rn(a, a) / __dmul_rn(lambda, __dmul_rn(omega, omega)))));
    }
    if (om != om) om = .5;
    if (!nan) {
        conv = S.resstop ? w[4] <= S.tol : norm_max < __dmul_rn(S.limit, __dsub_rn(w[2], w[3]));
        done = conv || iteration >= S.max_it;
    }
    js->norm_max = norm_max;
    js->norm_sum = nan ? w[1] : norm_sum;
    js->omega = om;
    js->iteration = iteration;
    js->converged = conv;
    js->nan = nan;
    js->done = done;
    if (cond) cudaGraphSetConditional(h, done ? 0u : 1u);
}

// phi <- tmp when the last sweep left the result there (an odd number of sweeps)
__global__ void __launch_bounds__(256) k_jacobi_out(double *__restrict__ phi, const double *__restrict__ tmp,
                                                    const JacState *__restrict__ js, long N) {
    if (!(js->iteration & 1)) return;
    const long i = (long)blockIdx.x * 256 + threadIdx.x;
    if (i < N) phi[i] = tmp[i];
}

}  // namespace kf
