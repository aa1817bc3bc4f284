// kf_jacobi.cuh -- the reference's nonlinear Jacobi relaxation
// (solver_poisson_jacobi_nlin.cpp:50-265) with its sweep loop on the device.
//
// A sweep is one kernel.  Its blocks leave their statistics (reduced in a fixed
// order) in memory; every block of the next sweep reduces them again and forms
// Carre's over-relaxation factor and the stop test from them, beside the update of
// its points, of which only the last step needs the factor.  So a sweep waits for
// no atomic, fence or last block: 6.8 -> 4 us at 32^3.  The loop is a conditional
// WHILE node whose body holds JC_UNROLL sweeps, which return at once when an
// earlier one has stopped; the host reads the record back once per solve.  A
// host-driven sweep (two launches, a copy and a synchronisation) took 27 us.
#pragma once

#include "kf_div.hpp"
#include "kf_poisson.cuh"

namespace kf {

// The relaxation's record (members of solver_poisson_jacobi_nlin.hpp:66-95):
// norm_max ... omega carry over between sweeps and solves.
struct JacState {
    double norm_max, norm_sum, norm_max_old, norm_sum_old, sup, inf, omega, rlast;
    int iteration, done, converged, nan;
    int fresh, pad;  // no sweep's statistics are to be taken in
};

struct JacStop {
    int max_it, resstop;
    double limit, tol;  // relative-update limit; residual target (resstop)
};

// The sum A of point_coeffs by divisions
__device__ __noinline__ double point_sum(const double *pm, const double *p, const double *pp, const Lev &L, int i, int j,
                                         int k) {
    const int n = L.n;
    double A = pp[j * n + k] / L.dp[i];
    A = __dadd_rn(A, pm[j * n + k] / L.dm[i]);
    A = __dadd_rn(A, p[wrapi(j + 1, n) * n + k] / L.dp[j]);
    A = __dadd_rn(A, p[wrapi(j - 1, n) * n + k] / L.dm[j]);
    A = __dadd_rn(A, p[j * n + wrapi(k + 1, n)] / L.dp[k]);
    return __dadd_rn(A, p[j * n + wrapi(k - 1, n)] / L.dm[k]);
}

// point_coeffs: the same quotients and sums, the divisors' reciprocals from
// tables; p: the plane i of the potential, pp and pm its neighbours
__device__ __forceinline__ void point_coeffs_div(const double *pm, const double *p, const double *pp, double rho,
                                                 const Lev &L, int i, int j, int k, double &A, double &D) {
    const int n = L.n;
    D = __dadd_rn(__dadd_rn(L.dd[i], L.dd[j]), L.dd[k]);
    A = div_by(pp[j * n + k], L.dp[i], L.rp[i]);
    A = __dadd_rn(A, div_by(pm[j * n + k], L.dm[i], L.rm[i]));
    A = __dadd_rn(A, div_by(p[wrapi(j + 1, n) * n + k], L.dp[j], L.rp[j]));
    A = __dadd_rn(A, div_by(p[wrapi(j - 1, n) * n + k], L.dm[j], L.rm[j]));
    A = __dadd_rn(A, div_by(p[j * n + wrapi(k + 1, n)], L.dp[k], L.rp[k]));
    A = __dadd_rn(A, div_by(p[j * n + wrapi(k - 1, n)], L.dm[k], L.rm[k]));
    if (A != A) A = point_sum(pm, p, pp, L, i, j, k);
    A = __dmul_rn(2., A);
    A = __dadd_rn(A, rho);
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

// Statistics of a sweep over some points: sum and maximum of |dP|, maximum of
// |f(P_old)|, extrema of P_new.  The sum's order is fixed: 256 values by a tree in
// which t takes t + w for w = 128, 64, ..., 1; the others do not depend on it.
struct JcStat {
    double sum;
    unsigned long long dmax, fmax;  // bit patterns (a NaN sorts above +inf)
    double pmax, pmin;
    __device__ __forceinline__ void join(const JcStat &o) {
        sum = __dadd_rn(sum, o.sum);
        dmax = max(dmax, o.dmax);
        fmax = max(fmax, o.fmax);
        pmax = ::fmax(pmax, o.pmax);
        pmin = ::fmin(pmin, o.pmin);
    }
    __device__ __forceinline__ void warp() {  // lane t takes t + 16, 8, ... 1: the result in lane 0
        for (int w = 16; w > 0; w >>= 1) {
            JcStat o;
            o.sum = __shfl_down_sync(0xffffffffu, sum, w);
            o.dmax = __shfl_down_sync(0xffffffffu, dmax, w);
            o.fmax = __shfl_down_sync(0xffffffffu, fmax, w);
            o.pmax = __shfl_down_sync(0xffffffffu, pmax, w);
            o.pmin = __shfl_down_sync(0xffffffffu, pmin, w);
            join(o);
        }
    }
};

// The tree over a block's 256 values, by its first warp (the result in lane 0).
__device__ __forceinline__ JcStat jac_tree(const JcStat &v, JcStat *sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    JcStat a[8];
    if (threadIdx.x < 32) {
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q] = sh[q * 32 + threadIdx.x];
#pragma unroll
        for (int w = 4; w > 0; w >>= 1)
#pragma unroll
            for (int q = 0; q < w; ++q) a[q].join(a[q + w]);
        a[0].warp();
    }
    return a[0];
}

// The record after a sweep with the statistics v.
__device__ __forceinline__ void jac_finish(JacState &st, const JcStat &v, long N, const JacStop &S) {
    const double w[5] = {__longlong_as_double((long long)v.dmax), v.sum, v.pmax, v.pmin,
                         __longlong_as_double((long long)v.fmax)};
    const int iteration = st.iteration + 1;
    const double omega = st.omega;
    st.norm_sum_old = st.norm_sum;
    st.norm_max_old = st.norm_max;
    st.sup = w[2];
    st.inf = w[3];
    st.rlast = w[4];
    const double norm_max = w[0], norm_sum = w[1] / (double)N;
    const bool nan = w[4] != w[4] || w[0] != w[0];
    // Carre's over-relaxation factor (:237-252)
    double om = .5;
    if (norm_max < st.norm_max_old && iteration > 1) {
        const double lambda = norm_sum / st.norm_sum_old;
        const double a = __dsub_rn(__dadd_rn(lambda, omega), 1.);
        om = 2. / __dadd_rn(1., sqrt(__dsub_rn(1., __dmul_rn(a, a) / __dmul_rn(lambda, __dmul_rn(omega, omega)))));
    }
    if (om != om) om = .5;
    bool conv = false, done = nan;
    if (!nan) {
        conv = S.resstop ? w[4] <= S.tol : norm_max < __dmul_rn(S.limit, __dsub_rn(w[2], w[3]));
        done = conv || iteration >= S.max_it;
    }
    st.norm_max = norm_max;
    st.norm_sum = nan ? w[1] : norm_sum;
    st.omega = om;
    st.iteration = iteration;
    st.converged = conv;
    st.nan = nan;
    st.done = done;
}

// The record with the last sweep's block statistics q[0 .. nq - 1] taken in, in
// every thread: the loads (jac_load) are issued before, the result needs the block.
__device__ __forceinline__ JcStat jac_load(const JcStat *q, int nq) {
    JcStat v{0., 0ull, 0ull, -INFINITY, INFINITY};
    for (int b = threadIdx.x; b < nq; b += 256) v.join(q[b]);
    return v;
}
__device__ __forceinline__ void jac_record(const JcStat &v, const JacState *in, long N, const JacStop &S, JcStat *sh,
                                           JacState *st) {
    const JcStat w = jac_tree(v, sh);
    if (threadIdx.x == 0) {
        JacState s = *in;
        if (!s.done && !s.fresh) jac_finish(s, w, N, S);
        *st = s;
    }
    __syncthreads();
}

// One sweep in -> out; q, sin: the last sweep's statistics and the record before
// it; p, sout: this one's statistics and the record before it.
__global__ void __launch_bounds__(256) k_jacobi(const double *__restrict__ in, double *__restrict__ out,
                                                const double *__restrict__ rho, Lev L, JacStop S,
                                                const JcStat *__restrict__ q, JcStat *__restrict__ p,
                                                const JacState *__restrict__ sin, JacState *__restrict__ sout) {
    __shared__ JcStat sh[256];
    __shared__ JacState st;
    const int n = L.n, nn = n * n, t = threadIdx.x;
    const long N = (long)nn * n;
    const JcStat prev = jac_load(q, gridDim.x);
    JcStat v{0., 0ull, 0ull, -INFINITY, INFINITY};
    double omega = 1.;
    bool have = false;
    for (long id = (long)blockIdx.x * 256 + t; id < N || !have; id += (long)gridDim.x * 256) {
        double P_old = 0., P_new = 0., f0 = 0.;
        if (id < N) {
            const unsigned u = (unsigned)id;
            const int k = (int)(u % (unsigned)n);
            const unsigned r = u / (unsigned)n;
            const int j = (int)(r % (unsigned)n), i = (int)(r / (unsigned)n);
            double A, D;
            point_coeffs_div(in + wrapi(i - 1, n) * nn, in + i * nn, in + wrapi(i + 1, n) * nn, rho[id], L, i, j, k, A, D);
            P_old = in[id];
            P_new = newton_point(P_old, A, D, f0);
        }
        if (!have) {  // the factor, once the first point has come this far
            have = true;
            jac_record(prev, sin, N, S, sh, &st);
            if (blockIdx.x == 0 && t == 0) {
                JacState s = st;
                s.fresh = 0;
                *sout = s;
            }
            if (st.done) return;
            omega = st.omega;
            __syncthreads();  // sh is used again below
        }
        if (id >= N) break;
        const double delta = fabs(__dsub_rn(P_new, P_old));
        out[id] = __dadd_rn(__dmul_rn(1. - omega, P_old), __dmul_rn(omega, P_new));
        v.join(JcStat{delta, (unsigned long long)__double_as_longlong(delta),
                      (unsigned long long)__double_as_longlong(fabs(f0)), P_new, P_new});
        if (id == 0) {  // supremum = infinum = in.val[0] at the start (:158-159)
            v.pmax = fmax(v.pmax, P_old);
            v.pmin = fmin(v.pmin, P_old);
        }
    }
    v = jac_tree(v, sh);
    if (t == 0) p[blockIdx.x] = v;
}

// After the body's sweeps: their last statistics into the record, the WHILE
// condition h from it (loop == 0: not in a loop).  One block.
__global__ void __launch_bounds__(256) k_jacobi_test(const JcStat *__restrict__ q, int nq, JacState *js, long N,
                                                     JacStop S, int loop, cudaGraphConditionalHandle h) {
    __shared__ JcStat sh[256];
    __shared__ JacState st;
    jac_record(jac_load(q, nq), js, N, S, sh, &st);
    if (threadIdx.x) return;
    JacState s = st;
    s.fresh = 1;
    *js = s;
    if (loop) cudaGraphSetConditional(h, s.done ? 0u : 1u);
}

// phi <- tmp when the last sweep left the result there (an odd number of sweeps)
__global__ void __launch_bounds__(256) k_jacobi_out(double *__restrict__ phi, const double *__restrict__ tmp,
                                                    const JacState *__restrict__ js, long N) {
    if (!(js->iteration & 1)) return;
    const long i = (long)blockIdx.x * 256 + threadIdx.x;
    if (i < N) phi[i] = tmp[i];
}

}  // namespace kf
