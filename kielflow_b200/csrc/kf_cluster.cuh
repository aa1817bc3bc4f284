// kf_cluster.cuh -- the coarse levels of a V-cycle in one thread-block cluster.
//
// Levels of at most 32^3 points are latency: launched one by one, each kernel of
// the cycle there lasts about its launch (2-3 us, 14 kernels a level), and the
// coarsest level's relaxation, a chain of 10-20 sweeps, ran in one block on one
// SM (84-150 us a visit).  k_cc holds all of these levels in the shared memory of
// one cluster: CTA c owns the planes i of its slab on every level (the cluster
// size divides the coarsest n), keeps the two neighbouring planes beside them
// and, when it updates a point of its first or last plane, writes it into the
// neighbour's copy as well (distributed shared memory); a cluster barrier (0.2
// us) ends each phase.  Points, operations and their order are those of the
// level-by-level kernels (k_fas_rhs, k_rbgs_t, k_residual, k_restrict,
// k_coarse_solve, k_correction, k_prolong_add), so the potentials are the same
// bit for bit.
//
// Planes are stored by colour, colour (i + j + k) & 1 at element j h + k / 2 (h =
// n / 2), and thread t owns the column pair (j, k2) = (t / h, t % h) of every
// plane: its loads are conflict-free (in natural order the stride of two doubles
// made the half sweep shared-memory bound, 2.1 us at 32^3 on 16 SMs) and its j
// and k table entries stay in registers.
#pragma once

#include <cooperative_groups.h>

#include "kf_poisson.cuh"

namespace kf {

constexpr int CC_LEVELS = 4, CC_THREADS = 512, CC_MAX_CTAS = 16, CC_MAX_N = 32;
constexpr int CC_SMEM_MAX = 200 * 1024;

struct ClusterCycle {
    int nl;  // levels held: 0 = the entry level, nl - 1 = the coarsest; n even, at most CC_MAX_N
    int n[CC_LEVELS];
    const double *dd[CC_LEVELS], *ip[CC_LEVELS], *im[CC_LEVELS];
    const double *gam[CC_LEVELS];  // fine-axis gammas of level m (prolongation from m + 1)
    const double *cc[CC_LEVELS];   // linear form: e^phi on the level (natural order)
};

// Doubles of one CTA's part of a level: pp own planes of 2 W = n^2 points.  P
// holds planes -1 .. pp, R and C (linear form) the own ones, F planes -1 .. pp - 1
// (on the coarsest level instead the second red buffer X, planes -1 .. pp), P0
// planes 0 .. pp (not on the entry level), then the axis tables.
__host__ __device__ inline int cc_slab_doubles(int n, int cl, bool entry, bool last, bool lin) {
    const int pp = n / cl, S = n * n;
    return (pp + 2) * S + pp * S + (last ? (pp + 2) * S / 2 : (pp + 1) * S) + (entry ? 0 : (pp + 1) * S) +
           (lin ? pp * S : 0) + 4 * n;
}
inline size_t cc_smem(const ClusterCycle &C, int cl, bool lin) {
    size_t d = 0;
    for (int m = 0; m < C.nl; ++m) d += cc_slab_doubles(C.n[m], cl, m == 0, m + 1 == C.nl, lin);
    return d * sizeof(double);
}

struct CcSlab {
    int n, h, W, pp, i0;
    double *P, *R, *F, *P0, *C, *dd, *ip, *im, *gam;
    // plane pl of a colour
    __device__ __forceinline__ int p(int pl, int c) const { return ((pl + 1) * 2 + c) * W; }
    __device__ __forceinline__ int r(int pl, int c) const { return (pl * 2 + c) * W; }
};

__device__ __forceinline__ CcSlab cc_slab(const ClusterCycle &C, double *sm, int m, int cl, int rank, bool lin) {
    for (int l = 0; l < m; ++l) sm += cc_slab_doubles(C.n[l], cl, l == 0, l + 1 == C.nl, lin);
    CcSlab V;
    V.n = C.n[m];
    V.h = V.n >> 1;
    V.W = V.n * V.h;
    V.pp = V.n / cl;
    V.i0 = rank * V.pp;
    const int S = V.n * V.n;
    V.P = sm;
    V.R = V.P + (V.pp + 2) * S;
    V.F = V.R + V.pp * S;
    V.P0 = V.F + (m + 1 == C.nl ? (V.pp + 2) * V.W : (V.pp + 1) * S);
    V.C = V.P0 + (m == 0 ? 0 : (V.pp + 1) * S);
    V.dd = V.C + (lin ? V.pp * S : 0);
    V.ip = V.dd + V.n;
    V.im = V.ip + V.n;
    V.gam = V.im + V.n;
    return V;
}

// Thread t's column pair on a level: element offsets of its neighbours and its
// table entries (k = 2 k2 + par).
struct CcLane {
    bool on;
    int t, j, ojp, ojm, okp, okm;
    double ddj, ipj, imj, ddk[2], ipk[2], imk[2];
};
__device__ __forceinline__ CcLane cc_lane(const CcSlab &V) {
    CcLane L;
    L.t = threadIdx.x;
    L.on = L.t < V.W;
    const int t = L.on ? L.t : 0, j = t / V.h, k2 = t - j * V.h;
    L.j = j;
    L.ojp = j == V.n - 1 ? -j * V.h : V.h;
    L.ojm = j == 0 ? (V.n - 1) * V.h : -V.h;
    L.okp = k2 == V.h - 1 ? -k2 : 1;  // k + 1 of an odd k
    L.okm = k2 == 0 ? V.h - 1 : -1;   // k - 1 of an even k
    L.ddj = V.dd[j];
    L.ipj = V.ip[j];
    L.imj = V.im[j];
#pragma unroll
    for (int par = 0; par < 2; ++par) {
        L.ddk[par] = V.dd[2 * k2 + par];
        L.ipk[par] = V.ip[2 * k2 + par];
        L.imk[par] = V.im[2 * k2 + par];
    }
    return L;
}

template <bool LIN> struct ClusterCore {
    cooperative_groups::cluster_group cg = cooperative_groups::this_cluster();
    double *lo, *hi;  // the neighbours' shared memory (ranks - 1 and + 1), same layout
    const double *base;

    // The sum A (with rho) and diagonal D (point_coeffs_fast's operations) of the
    // point of colour c in own plane pl; q: the other colour's planes pl - 1, pl,
    // pl + 1 at the thread's element.
    __device__ __forceinline__ void coeffs(const CcSlab &V, const CcLane &L, int pl, int par, const double *qm,
                                           const double *q, const double *qp, double rho, bool with_rho, double &A,
                                           double &D) const {
        const int i = V.i0 + pl;
        D = __dadd_rn(__dadd_rn(V.dd[i], L.ddj), par ? L.ddk[1] : L.ddk[0]);
        A = __dmul_rn(*qp, V.ip[i]);
        A = __dadd_rn(A, __dmul_rn(*qm, V.im[i]));
        A = __dadd_rn(A, __dmul_rn(q[L.ojp], L.ipj));
        A = __dadd_rn(A, __dmul_rn(q[L.ojm], L.imj));
        A = __dadd_rn(A, __dmul_rn(q[par ? L.okp : 0], par ? L.ipk[1] : L.ipk[0]));
        A = __dadd_rn(A, __dmul_rn(q[par ? 0 : L.okm], par ? L.imk[1] : L.imk[0]));
        if (with_rho) A = __dadd_rn(A, rho);
    }
    __device__ __forceinline__ void coeffs(const CcSlab &V, const CcLane &L, int pl, int c, bool with_rho, double &A,
                                           double &D) const {
        const int par = (V.i0 + pl + L.j + c) & 1;
        const double *q = V.P + V.p(pl, c ^ 1) + L.t;
        coeffs(V, L, pl, par, q - 2 * V.W, q, q + 2 * V.W, V.R[V.r(pl, c) + L.t], with_rho, A, D);
    }
    __device__ __forceinline__ double resid(double A, double D, double x, double c) const {
        if constexpr (LIN) return __dsub_rn(A, __dmul_rn(__dadd_rn(D, c), x));
        return f_point(A, D, x);
    }
    __device__ __forceinline__ double update(double A, double D, double x, double c, double w) const {
        if constexpr (LIN) {
            const double y = A / __dadd_rn(D, c);
            return w == 1. ? y : __dadd_rn(x, __dmul_rn(w, __dsub_rn(y, x)));
        }
        return newton_step(x, A, D, w);
    }
    // element e of colour c in own plane pl of P <- v, and the neighbours' copies
    __device__ __forceinline__ void put(const CcSlab &V, int pl, int c, int e, double v) const {
        V.P[V.p(pl, c) + e] = v;
        const long o = V.P - base;
        if (pl == 0) lo[o + V.p(V.pp, c) + e] = v;
        if (pl == V.pp - 1) hi[o + V.p(-1, c) + e] = v;
    }

    __device__ __forceinline__ void half_sweep(const CcSlab &V, const CcLane &L, int c, double w) const {
        if (L.on)
            for (int pl = 0; pl < V.pp; ++pl) {
                double A, D;
                coeffs(V, L, pl, c, true, A, D);
                put(V, pl, c, L.t,
                    update(A, D, V.P[V.p(pl, c) + L.t], LIN ? V.C[V.r(pl, c) + L.t] : 0., w));
            }
        cg.sync();
    }

    // rho = N(phi) + r in place of r (k_fas_rhs, k_fas_rhs_lin); the smoother that
    // follows writes into the neighbours' end planes, which this reads
    __device__ __forceinline__ void fas_rhs(const CcSlab &V, const CcLane &L) const {
        if (L.on)
            for (int pl = 0; pl < V.pp; ++pl)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    double A, D;
                    coeffs(V, L, pl, c, false, A, D);
                    const double x = V.P[V.p(pl, c) + L.t];
                    double *R = V.R + V.r(pl, c) + L.t;
                    const double N = LIN ? __dsub_rn(__dmul_rn(__dadd_rn(D, V.C[V.r(pl, c) + L.t]), x), A)
                                         : __dsub_rn(0., f_point(A, D, x));
                    *R = __dadd_rn(N, *R);
                }
        cg.sync();
    }

    // F = residual of the level, its last plane also in the next CTA's copy
    __device__ __forceinline__ void residual(const CcSlab &V, const CcLane &L) const {
        if (L.on)
            for (int pl = 0; pl < V.pp; ++pl)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    double A, D;
                    coeffs(V, L, pl, c, true, A, D);
                    const double f =
                        resid(A, D, V.P[V.p(pl, c) + L.t], LIN ? V.C[V.r(pl, c) + L.t] : 0.);
                    V.F[V.p(pl, c) + L.t] = f;
                    if (pl == V.pp - 1) hi[(V.F - base) + V.p(-1, c) + L.t] = f;
                }
        cg.sync();
    }

    // level V -> W: full weighting of F into W.R, injection of P into W.P and W.P0;
    // thread t < nc^2 takes the coarse column (J, K)
    __device__ __forceinline__ void restrict_to(const CcSlab &V, const CcSlab &W) const {
        const int nc = W.n, J = threadIdx.x / nc, K = threadIdx.x - J * nc;
        if (J < nc)
            for (int pl = 0; pl < W.pp; ++pl) {
                const double w[3] = {0.25, 0.5, 0.25};
                const int Km = K == 0 ? V.h - 1 : K - 1;
                double s = 0.;
#pragma unroll
                for (int a = -1; a <= 1; ++a) {
                    double sy = 0.;
#pragma unroll
                    for (int b = -1; b <= 1; ++b) {
                        const int j = b < 0 && J == 0 ? V.n - 1 : 2 * J + b, ev = (a + b) & 1;
                        const double *even = V.F + V.p(2 * pl + a, ev) + j * V.h;
                        const double *odd = V.F + V.p(2 * pl + a, ev ^ 1) + j * V.h;
                        double sz = __dadd_rn(0., __dmul_rn(w[0], odd[Km]));
                        sz = __dadd_rn(sz, __dmul_rn(w[1], even[K]));
                        sz = __dadd_rn(sz, __dmul_rn(w[2], odd[K]));
                        sy = __dadd_rn(sy, __dmul_rn(w[b + 1], sz));
                    }
                    s = __dadd_rn(s, __dmul_rn(w[a + 1], sy));
                }
                const int c = (W.i0 + pl + J + K) & 1, e = J * W.h + (K >> 1);
                const double p = V.P[V.p(2 * pl, 0) + 2 * J * V.h + K];
                W.R[W.r(pl, c) + e] = s;
                put(W, pl, c, e, p);
                W.P0[W.r(pl, c) + e] = p;
                if (pl == 0) lo[(W.P0 - base) + W.r(W.pp, c) + e] = p;
            }
        cg.sync();
    }

    // V.P += prolongation of W.P - W.P0 (prolong_cell's operations)
    __device__ __forceinline__ void prolong_from(const CcSlab &V, const CcSlab &W) const {
        const int nc = W.n, J = threadIdx.x / nc, K = threadIdx.x - J * nc;
        if (J < nc) {
            const int J1 = J + 1 == nc ? 0 : J + 1, K1 = K + 1 == nc ? 0 : K + 1;
            for (int pl = 0; pl < W.pp; ++pl) {
                const int I = W.i0 + pl;
                double zc[2][2][2], yc[2][2][2];
                const double gz = V.gam[2 * K + 1], gy = V.gam[2 * J + 1], gx = V.gam[2 * I + 1];
#pragma unroll
                for (int di = 0; di < 2; ++di)
#pragma unroll
                    for (int dj = 0; dj < 2; ++dj) {
                        double e[2];
#pragma unroll
                        for (int dk = 0; dk < 2; ++dk) {
                            // an index that wraps changes by the even nc: the colour is that of I + di, ...
                            const int c = (I + di + J + dj + K + dk) & 1;
                            const int o = (dj ? J1 : J) * W.h + ((dk ? K1 : K) >> 1);
                            e[dk] = __dsub_rn(W.P[W.p(pl + di, c) + o], W.P0[W.r(pl + di, c) + o]);
                        }
                        zc[di][dj][0] = e[0];
                        zc[di][dj][1] = __dadd_rn(__dmul_rn(1. - gz, e[0]), __dmul_rn(gz, e[1]));
                    }
#pragma unroll
                for (int di = 0; di < 2; ++di)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        yc[di][0][q] = zc[di][0][q];
                        yc[di][1][q] = __dadd_rn(__dmul_rn(1. - gy, zc[di][0][q]), __dmul_rn(gy, zc[di][1][q]));
                    }
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const double v =
                                a == 0 ? yc[0][b][q]
                                       : __dadd_rn(__dmul_rn(1. - gx, yc[0][b][q]), __dmul_rn(gx, yc[1][b][q]));
                            const int f = 2 * pl + a, c = (a + b + q) & 1, e = (2 * J + b) * V.h + K;
                            put(V, f, c, e, __dadd_rn(V.P[V.p(f, c) + e], v));
                        }
            }
        }
        cg.sync();
    }

    // max over the cluster of each CTA's m >= 0, as bit patterns (a NaN sorts above
    // +inf); slots [2][CC_MAX_CTAS] in every CTA, one row per parity so that a row is
    // rewritten two barriers later
    __device__ __forceinline__ double cluster_max(double m, unsigned long long *sh,
                                                  unsigned long long (*slots)[CC_MAX_CTAS], int par) const {
        unsigned long long u = (unsigned long long)__double_as_longlong(m);
        for (int o = 16; o > 0; o >>= 1) u = max(u, __shfl_xor_sync(0xffffffffu, u, o));
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = u;
        __syncthreads();
        const int cl = (int)cg.num_blocks();
        if (threadIdx.x < 32) {
            u = threadIdx.x < CC_THREADS / 32 ? sh[threadIdx.x] : 0ull;
            for (int o = CC_THREADS / 64; o > 0; o >>= 1) u = max(u, __shfl_xor_sync(0xffffffffu, u, o));
            if ((int)threadIdx.x < cl) *cg.map_shared_rank(&slots[par][cg.block_rank()], threadIdx.x) = u;
        }
        cg.sync();
        u = (threadIdx.x & 15) < cl ? slots[par][threadIdx.x & 15] : 0ull;
        for (int o = 8; o > 0; o >>= 1) u = max(u, __shfl_xor_sync(0xffffffffu, u, o));
        return __longlong_as_double((long long)u);
    }

    // block_coarse_relax: red-black sweeps until max |f| <= max(tol, rtol max |f|
    // at entry), tested before every `every` sweeps.  The test's residual at a red
    // point is the one its update starts from, so a test also forms the red half of
    // the sweep after it, into the second red buffer (the neighbours' copies
    // included); the sweep is entered by exchanging the buffers.  Returns the sweeps
    // done; red: the buffer that holds the result (planes from -1).
    __device__ __forceinline__ int relax(const CcSlab &V, const CcLane &L, double tol, double rtol, int max_sweeps,
                                         int every, double w, unsigned long long *sh,
                                         unsigned long long (*slots)[CC_MAX_CTAS]) const {
        double r0 = 0.;
        int s = 0, par = 0;
        const int W = V.W;
        // red planes: P's (stride 2 W) or X's (stride W)
        double *cur = V.P, *alt = V.F;
        int cs = 2 * W, as = W;
        for (;;) {
            double m = 0.;
            if (L.on)
                for (int pl = 0; pl < V.pp; ++pl) {
                    double A, D;
                    {  // red, from the black planes
                        const double *q = V.P + V.p(pl, 1) + L.t;
                        coeffs(V, L, pl, (V.i0 + pl + L.j) & 1, q - 2 * W, q, q + 2 * W, V.R[V.r(pl, 0) + L.t], true, A,
                               D);
                        const double x = cur[(pl + 1) * cs + L.t];
                        double f, y;
                        if constexpr (LIN) {
                            const double c = V.C[V.r(pl, 0) + L.t];
                            f = resid(A, D, x, c);
                            y = update(A, D, x, c, w);
                        } else {
                            const double ex = exp(x);
                            f = __dsub_rn(__dsub_rn(A, __dmul_rn(D, x)), ex);
                            y = __dsub_rn(x, __dmul_rn(w, f / __dsub_rn(-D, ex)));
                        }
                        m = nmax(m, fabs(f));
                        alt[(pl + 1) * as + L.t] = y;
                        const long o = alt - base;
                        if (pl == 0) lo[o + (V.pp + 1) * as + L.t] = y;
                        if (pl == V.pp - 1) hi[o + L.t] = y;
                    }
                    {  // black, from the red planes
                        const double *q = cur + (pl + 1) * cs + L.t;
                        coeffs(V, L, pl, (V.i0 + pl + L.j + 1) & 1, q - cs, q, q + cs, V.R[V.r(pl, 1) + L.t], true, A, D);
                        m = nmax(m, fabs(resid(A, D, V.P[V.p(pl, 1) + L.t], LIN ? V.C[V.r(pl, 1) + L.t] : 0.)));
                    }
                }
            const double res = cluster_max(m, sh, slots, par);
            par ^= 1;
            if (s == 0) r0 = res;
            if (!(res > fmax(tol, rtol * r0)) || s >= max_sweeps) break;  // reached, NaN or capped
            double *tp = cur;
            cur = alt;
            alt = tp;
            const int ts = cs;
            cs = as;
            as = ts;
            for (int t = 0; t < every; ++t) {
                if (t > 0) {  // red, in place
                    if (L.on)
                        for (int pl = 0; pl < V.pp; ++pl) {
                            double A, D;
                            const double *q = V.P + V.p(pl, 1) + L.t;
                            coeffs(V, L, pl, (V.i0 + pl + L.j) & 1, q - 2 * W, q, q + 2 * W, V.R[V.r(pl, 0) + L.t],
                                   true, A, D);
                            const double y = update(A, D, cur[(pl + 1) * cs + L.t],
                                                    LIN ? V.C[V.r(pl, 0) + L.t] : 0., w);
                            cur[(pl + 1) * cs + L.t] = y;
                            const long o = cur - base;
                            if (pl == 0) lo[o + (V.pp + 1) * cs + L.t] = y;
                            if (pl == V.pp - 1) hi[o + L.t] = y;
                        }
                    cg.sync();
                }
                if (L.on)
                    for (int pl = 0; pl < V.pp; ++pl) {
                        double A, D;
                        const double *q = cur + (pl + 1) * cs + L.t;
                        coeffs(V, L, pl, (V.i0 + pl + L.j + 1) & 1, q - cs, q, q + cs, V.R[V.r(pl, 1) + L.t], true, A, D);
                        put(V, pl, 1, L.t,
                            update(A, D, V.P[V.p(pl, 1) + L.t], LIN ? V.C[V.r(pl, 1) + L.t] : 0., w));
                    }
                cg.sync();
            }
            s += every;
        }
        if (cur != V.P) {  // the result's red planes (neighbours' copies included) into P
            if (L.on)
                for (int pl = -1; pl <= V.pp; ++pl) V.P[V.p(pl, 0) + L.t] = cur[(pl + 1) * cs + L.t];
            __syncthreads();
        }
        return s;
    }
};

// phi: the entry level's injected potential, phi0 its copy, r the restricted
// residual (k_restrict), in natural order; leaves the level's phi and its
// correction phi - phi0 (in phi0).  LIN: the adjoint's linear system.
template <bool LIN>
__global__ void __launch_bounds__(CC_THREADS) k_cc(double *__restrict__ phi, double *__restrict__ phi0,
                                                   const double *__restrict__ r, const __grid_constant__ ClusterCycle C,
                                                   int pre, int post, double tol, double rtol, int max_sweeps,
                                                   int every, double om, double om_coarse,
                                                   int *__restrict__ sweeps_out) {
    extern __shared__ __align__(16) double cc_sm[];
    __shared__ unsigned long long sh[CC_THREADS / 32];
    __shared__ unsigned long long slots[2][CC_MAX_CTAS];
    ClusterCore<LIN> K;
    const int cl = (int)K.cg.num_blocks(), rank = (int)K.cg.block_rank();
    K.base = cc_sm;
    K.lo = K.cg.map_shared_rank(cc_sm, rank == 0 ? cl - 1 : rank - 1);
    K.hi = K.cg.map_shared_rank(cc_sm, rank == cl - 1 ? 0 : rank + 1);
    for (int m = 0; m < C.nl; ++m) {
        const CcSlab V = cc_slab(C, cc_sm, m, cl, rank, LIN);
        const int t = threadIdx.x;
        if (t < V.n) {
            V.dd[t] = C.dd[m][t];
            V.ip[t] = C.ip[m][t];
            V.im[t] = C.im[m][t];
            V.gam[t] = C.gam[m] ? C.gam[m][t] : 0.;
        }
        if (LIN && t < V.W) {
            const int j = t / V.h;
            for (int pl = 0; pl < V.pp; ++pl) {
                const double2 v = reinterpret_cast<const double2 *>(C.cc[m])[(V.i0 + pl) * V.W + t];
                const int c = (V.i0 + pl + j) & 1;
                V.C[V.r(pl, c) + t] = v.x;
                V.C[V.r(pl, c ^ 1) + t] = v.y;
            }
        }
    }
    const CcSlab V0 = cc_slab(C, cc_sm, 0, cl, rank, LIN);
    const int t = threadIdx.x, j = t / V0.h;
    if (t < V0.W)
        for (int pl = -1; pl <= V0.pp; ++pl) {
            const int i = V0.i0 + pl, iw = i < 0 ? i + V0.n : i >= V0.n ? i - V0.n : i, c = (iw + j) & 1;
            const double2 v = reinterpret_cast<const double2 *>(phi)[iw * V0.W + t];
            V0.P[V0.p(pl, c) + t] = v.x;
            V0.P[V0.p(pl, c ^ 1) + t] = v.y;
            if (pl >= 0 && pl < V0.pp) {
                const double2 f = reinterpret_cast<const double2 *>(r)[iw * V0.W + t];
                V0.R[V0.r(pl, c) + t] = f.x;
                V0.R[V0.r(pl, c ^ 1) + t] = f.y;
            }
        }
    K.cg.sync();  // every CTA runs and has loaded before a neighbour writes into it
    for (int m = 0;; ++m) {
        const CcSlab V = cc_slab(C, cc_sm, m, cl, rank, LIN);
        const CcLane L = cc_lane(V);
        K.fas_rhs(V, L);
        if (m + 1 == C.nl) break;
        for (int s = 0; s < pre; ++s) {
            K.half_sweep(V, L, 0, om);
            K.half_sweep(V, L, 1, om);
        }
        K.residual(V, L);
        K.restrict_to(V, cc_slab(C, cc_sm, m + 1, cl, rank, LIN));
    }
    const CcSlab Vc = cc_slab(C, cc_sm, C.nl - 1, cl, rank, LIN);
    const int s = K.relax(Vc, cc_lane(Vc), tol, rtol, max_sweeps, every, om_coarse, sh, slots);
    for (int m = C.nl - 2; m >= 0; --m) {
        const CcSlab V = cc_slab(C, cc_sm, m, cl, rank, LIN);
        const CcLane L = cc_lane(V);
        K.prolong_from(V, cc_slab(C, cc_sm, m + 1, cl, rank, LIN));
        for (int q = 0; q < post; ++q) {
            K.half_sweep(V, L, 0, om);
            K.half_sweep(V, L, 1, om);
        }
    }
    if (t < V0.W)
        for (int pl = 0; pl < V0.pp; ++pl) {
            const int i = V0.i0 + pl, c = (i + j) & 1, g = i * V0.W + t;
            const double2 p = make_double2(V0.P[V0.p(pl, c) + t], V0.P[V0.p(pl, c ^ 1) + t]);
            const double2 o = reinterpret_cast<const double2 *>(phi0)[g];
            reinterpret_cast<double2 *>(phi)[g] = p;
            reinterpret_cast<double2 *>(phi0)[g] = make_double2(__dsub_rn(p.x, o.x), __dsub_rn(p.y, o.y));
        }
    if (rank == 0 && t == 0 && sweeps_out) *sweeps_out = s;
    K.cg.sync();
}

}  // namespace kf
