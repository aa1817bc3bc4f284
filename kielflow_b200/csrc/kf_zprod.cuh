// kf_zprod.cuh -- the z-local middle of the right-hand side in one kernel: the
// inverse z transforms of u', s and their derivatives, the physical-space
// products and the forward z transform of the four results,
//   prod_c = u.grad u_c, prod_3 = u.grad s                     (rhs_standard.cpp:323-436)
//   g_q = -prod_q                                             (no penalization)
//   g_q = (1-H) (rl_q - prod_q) + H eta (q_d - q_fix)          (penalization)
// with rl_q = c2r(-lin_q).  Without penalization the right-hand side is
// -lin_q + r2c(g_q), with it r2c(g_q).  There the linear terms go the way of the
// reference, through physical space, in FP32 (RL: two more packed lines a row),
// where each way has rounding errors of its own, 1e-7 of the result apart; in FP64
// they stay in k-space (-lin_q + r2c(g_q - rl_q)) and rl_q is formed only on the
// rows where H is not zero, which saves 7 % of a 256^3 step, 3 % at 128^3.
//
// Everything between the y passes is local to a z line (i, j), so the 16 real
// fields of round D never go to memory.  A block of 8 (RL: 10) groups of P threads (a
// group carries one packed complex line) takes ZP_ROWS rows in turn: per row the
// real lines are packed c2r lines,
//   lines 0-2: U_c + i d_z U_c        lines 3-5: d_y U_c + i d_x U_c
//   line  6  : d_y s + i d_x s        line  7  : d_z s
//   RL: lines 8, 9: rl_0 + i rl_1, rl_2 + i rl_3
// whose groups transform them at once; the products of the row's z points
// give 4 real lines = 2 packed lines, kept in shared memory for one forward
// transform of all rows' results at the end.  s_d, which only the penalization
// takes, comes from the pass that forms the Poisson source.
//
// 256^3 FP32, one right-hand side: the three passes it replaces (k_z_c2r 491 us,
// the products 305 us, k_z_r2c 74 us) wrote and read 40 real fields on the way; here
// 404 us with 8 lines a row, 560 us with 10.
//
// The sums' roundings are written out (fma, mul_rn), so that a result does not
// depend on which products a compiler contracts: an FP32 right-hand side has the
// same bits whatever kernel holds the operation.
#pragma once

#include "kf_passes.cuh"
#include "kf_types.cuh"

namespace kf {

// Two rows at a time leave half of the groups idle in the forward transform but
// fit 8 blocks per SM where 4 rows fit 6 (256^3 FP32: 497 us against 553 us).
constexpr int ZP_ROWS = 2;
template <bool RL> struct ZProdLines { static constexpr int value = RL ? 10 : 8; };

// Resident blocks per SM asked of the register allocator: 64 registers a thread
// in FP32, 128 in FP64, what the shared memory of a 256-point block allows as
// well.  The kernel is bound by latency (a third of the issue slots used without
// the request), so residency is time.  256^3, products without penalization:
// FP32 861 us with 159 registers and 3 blocks, 497 us with 64 and 8; FP64 1657 us
// with 226 and 2, 1031 us with 128 and 4.
template <typename T, int N, int V, bool RL> struct ZProdMinBlocks {
    static constexpr int by_regs = (sizeof(T) == 4 ? 1024 : 512) / (ZProdLines<RL>::value * PlanV<N, V>::P);
    static constexpr int value = by_regs < 12 ? by_regs : 12;
};

template <typename T> struct ZProdArgs {
    typedef typename C2<T>::type T2;
    const T2 *s0, *sy, *sx;             // y-passed spectra of P s, d_y s, d_x s
    const T2 *u[3], *uy[3], *ux[3];     // of U_c, d_y U_c, d_x U_c
    T2 *out[4];                         // z-transformed results, half spectra
    // penalization: the mask, the window of rows on which it is not zero (RowBox), s_d,
    // and c2r(-lin_q) on that window's rows (RL: the y-passed spectra of -lin_q, of
    // every row)
    const T *H, *sd;
    const int *box;
    const T *rl[4];
    const T2 *lin[4];
    T M, eta, scale;                    // scale: the 1/N of the c2r
    int terms;
    int nkz, ip;  // the inputs are zero from kz = nkz on; elements per row
    int nko, op;  // outputs are needed for kz < nko; elements per row
};

template <typename T, int N, bool RL> struct ZProdSmem {
    typedef typename C2<T>::type T2;
    static constexpr int LS = PadLen<N>::value;
    // exchange / line buffers, and the packed results of ZP_ROWS rows
    static constexpr size_t bytes = (size_t)(ZProdLines<RL>::value * LS + 2 * ZP_ROWS * N) * sizeof(T2);
};

// u.d of two vectors: the first product is added to the rounded second one
template <typename T> __device__ __forceinline__ T dot3(T ux, T dx, T uy, T dy, T uz, T dz) {
    return fma(uz, dz, fma(ux, dx, mul_rn(uy, dy)));
}

template <typename T, int N, int V, bool RL>
__global__ void __launch_bounds__(ZProdLines<RL>::value * PlanV<N, V>::P, ZProdMinBlocks<T, N, V, RL>::value)
k_zprod(const __grid_constant__ ZProdArgs<T> a, const T *__restrict__ kv,
        const typename C2<T>::type *__restrict__ tw) {
    typedef typename C2<T>::type T2;
    constexpr int P = PlanV<N, V>::P, E = N / P, NZC = N / 2 + 1, LS = PadLen<N>::value;
    constexpr int LINES = ZProdLines<RL>::value, NT = LINES * P;
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *xch = reinterpret_cast<T2 *>(kf_smem);  // [LINES][LS]
    T2 *res = xch + LINES * LS;                 // [2 ZP_ROWS][N]
    const int p = threadIdx.x % P, l = threadIdx.x / P;
    const int r0 = blockIdx.x * ZP_ROWS;
    // this group's line: half spectra A and B (B == nullptr: i kz A, line 7: i kz A alone),
    // zero from kz = nkz on, rows of `ip` elements
    const bool linear = RL && l >= 8, sz = l == 7;
    const T2 *__restrict__ inA = l < 3 ? a.u[l] : l < 6 ? a.uy[l - 3] : l == 6 ? a.sy : sz ? a.s0 : a.lin[2 * (l - 8)];
    const T2 *__restrict__ inB = l < 3 || sz ? nullptr : l < 6 ? a.ux[l - 3] : l == 6 ? a.sx : a.lin[2 * (l - 8) + 1];
    const int nkz = linear ? NZC : a.nkz, ip = linear ? NZC : a.ip;
    T2 *line = xch + l * LS;
    const PadAddr pa;
    const bool adv = a.terms & T_ADVECTION, cont = a.terms & T_CONTINUITY;
    const RowBox box(a.box);
#pragma unroll 1
    for (int rr = 0; rr < ZP_ROWS; ++rr) {
        const long off = (long)(r0 + rr) * ip;
        // the half spectra into the line's own buffer (A from 0, B from NZC), then
        // the packed Hermitian line from there: element k and N - k share a load
        for (int k = p; k < nkz; k += P) {
            line[k] = __ldg(inA + off + k);
            if (inB) line[NZC + k] = __ldg(inB + off + k);
        }
        __syncwarp();
        T2 v[E];
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int k = reg_row<N, P, PlanV<N, V>::R1>(p, q);
            const int kk = k < NZC ? k : N - k;
            T2 x = mk<T2>((T)0, (T)0), y = x;
            if (kk < nkz) {
                x = line[kk];
                y = inB ? line[NZC + kk] : mk<T2>(mul_rn(-kv[kk], x.y), mul_rn(kv[kk], x.x));
                if (sz) {
                    x = y;
                    y = mk<T2>((T)0, (T)0);
                }
            }
            if (kk == 0 || 2 * kk == N) x.y = y.y = (T)0;  // as a c2r transform does
            if (k >= NZC) {
                x.y = -x.y;
                y.y = -y.y;
            }
            v[q] = mk<T2>(x.x - y.y, x.y + y.x);  // A + iB
        }
        __syncwarp();
        PlanV<N, V>::template fft<T2, +1>(v, line, pa, p, tw);  // its last exchange ends with a warp barrier
#pragma unroll
        for (int q = 0; q < E; ++q)
            line[reg_row<N, P, PlanV<N, V>::RL>(p, q)] = mk<T2>(v[q].x * a.scale, v[q].y * a.scale);
        __syncthreads();
        const bool inbox = box.has((r0 + rr) / N, (r0 + rr) % N);
        const int brow = box.row((r0 + rr) / N, (r0 + rr) % N);
        for (int z = threadIdx.x; z < N; z += NT) {
            const T2 U0 = xch[z], U1 = xch[LS + z], U2 = xch[2 * LS + z];  // (U_c, d_z U_c)
            const T ux = U0.x, uy = U1.x, uz = U2.x;
            const T2 S = xch[6 * LS + z];  // (d_y s, d_x s)
            const T sz_ = xch[7 * LS + z].x;
            T pr[4];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                pr[c] = (T)0;
                if (adv) {
                    const T2 d = xch[(3 + c) * LS + z];  // (d_y U_c, d_x U_c)
                    pr[c] = dot3(ux, d.y, uy, d.x, uz, c == 0 ? U0.y : c == 1 ? U1.y : U2.y);
                }
            }
            pr[3] = cont ? dot3(ux, S.y, uy, S.x, uz, sz_) : (T)0;
            T rl[4];
            if constexpr (RL) {
                const T2 l0 = xch[8 * LS + z], l1 = xch[9 * LS + z];
                rl[0] = l0.x;
                rl[1] = l0.y;
                rl[2] = l1.x;
                rl[3] = l1.y;
            }
            const T h = inbox ? a.H[(long)(r0 + rr) * N + z] : (T)0;
            if (h != (T)0) {
                const T qd[4] = {ux, uy, uz, a.sd[(long)(r0 + rr) * N + z]};
                const T qfix[4] = {-a.M, (T)0, (T)0, (T)-10};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if constexpr (!RL) rl[q] = a.rl[q][(long)brow * N + z];
                    const T f = fma((T)1 - h, rl[q] - pr[q], mul_rn(mul_rn(h, a.eta), qd[q] - qfix[q]));
                    pr[q] = RL ? f : f - rl[q];
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) pr[q] = RL ? rl[q] - pr[q] : -pr[q];
            }
            res[(2 * rr) * N + z] = mk<T2>(pr[0], pr[1]);
            res[(2 * rr + 1) * N + z] = mk<T2>(pr[2], pr[3]);
        }
        __syncthreads();
    }
    // forward: group l < 2 ZP_ROWS carries the packed line l & 1 of row l / 2
    T2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) v[q] = res[(l % (2 * ZP_ROWS)) * N + reg_row<N, P, PlanV<N, V>::R1>(p, q)];
    PlanV<N, V>::template fft<T2, -1>(v, line, pa, p, tw);
#pragma unroll
    for (int q = 0; q < E; ++q) line[pa(reg_row<N, P, PlanV<N, V>::RL>(p, q))] = v[q];
    __syncwarp();
    if (l >= 2 * ZP_ROWS) return;
    const long off = (long)(r0 + l / 2) * a.op;
    T2 *oA = a.out[2 * (l & 1)] + off, *oB = a.out[2 * (l & 1) + 1] + off;
    for (int k = p; k < a.nko; k += P) {
        const T2 zk = line[pa(k)];
        const T2 zm = line[pa(k == 0 ? 0 : N - k)];
        const T cr = zm.x, ci = -zm.y;  // conj(Z[N-k])
        oA[k] = mk<T2>((T)0.5 * (zk.x + cr), (T)0.5 * (zk.y + ci));
        oB[k] = mk<T2>((T)0.5 * (zk.y - ci), (T)-0.5 * (zk.x - cr));
    }
}

// z pass of one field, ZLine<T>::ROWS of its rows to a complex line; ZTile<T>::LZ
// lines per block.  In FP64 two rows (2 m, 2 m + 1) make the real and the
// imaginary part of a line.  In FP32 a row has a line of its own with a zero
// imaginary part: the rounding errors of a shared line would mix its rows, and
// these two passes are bound by memory, not by the transforms.
template <typename T> struct ZLine { static constexpr int ROWS = sizeof(T) == 8 ? 2 : 1; };
template <typename T, int N> inline int zline_blocks() {
    constexpr int per = ZTile<T>::LZ * ZLine<T>::ROWS;
    return (N * N + per - 1) / per;
}

// Inverse, with the Poisson source as the epilogue: s_d = c2r(P s^) and
// rho = e^{s_d} + n_d in FP64 (rhs_standard.cpp:108-111), into rho and its
// colour-split copy rcs (k_split's layout), each when given; and s_d into sd on the
// rows of the window.
template <typename T, int N, int V>
__global__ void __launch_bounds__(ZTile<T>::LZ * PlanV<N, V>::P)
k_z_rho(const typename C2<T>::type *__restrict__ in, T *__restrict__ sd, const int *__restrict__ window, const double *__restrict__ nd,
        double *__restrict__ rho, double *__restrict__ rcs, const typename C2<T>::type *__restrict__ tw, T scale,
        int nkz, int pitch) {
    typedef typename C2<T>::type T2;
    constexpr int LZ = ZTile<T>::LZ, P = PlanV<N, V>::P, E = N / P, NZC = N / 2 + 1, LS = PadLen<N>::value;
    constexpr int ROWS = ZLine<T>::ROWS;
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *xch = reinterpret_cast<T2 *>(kf_smem);  // [LZ][LS]
    const int p = threadIdx.x % P, l = threadIdx.x / P;
    const int r = ROWS * (blockIdx.x * LZ + l);
    const long off = (long)r * pitch;
    T2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int k = reg_row<N, P, PlanV<N, V>::R1>(p, q);
        const int kk = k < NZC ? k : N - k;
        T2 x = mk<T2>((T)0, (T)0), y = x;
        if (kk < nkz && r < N * N) {
            x = __ldg(in + off + kk);
            if (ROWS == 2) y = __ldg(in + off + pitch + kk);
        }
        if (kk == 0 || 2 * kk == N) x.y = y.y = (T)0;
        if (k >= NZC) {
            x.y = -x.y;
            y.y = -y.y;
        }
        v[q] = mk<T2>(x.x - y.y, x.y + y.x);
    }
    PlanV<N, V>::template fft<T2, +1>(v, xch + l * LS, PadAddr{}, p, tw);
    if (r >= N * N) return;
    const RowBox box(window);
    constexpr long half = (long)N * N * (N / 2);
    auto put = [&](int row, int z, T s) {
        const long i = (long)row * N + z;
        const double e = exp((double)s) + nd[i];
        if (box.has(row / N, row % N)) sd[i] = s;
        if (rho) rho[i] = e;
        if (rcs) rcs[((row / N + row % N + z) & 1) * half + (i >> 1)] = e;
    };
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int z = reg_row<N, P, PlanV<N, V>::RL>(p, q);
        put(r, z, v[q].x * scale);
        if (ROWS == 2) put(r + 1, z, v[q].y * scale);
    }
}

// Forward, of the FP64 potential in the bulk precision: out = the half spectra
// of phi's rows, kz < nko, rows of `pitch` elements.  SP: phi in split order.
template <typename T, int N, int V, bool SP>
__global__ void __launch_bounds__(ZTile<T>::LZ * PlanV<N, V>::P)
k_z_phi(const double *__restrict__ phi, typename C2<T>::type *__restrict__ out,
        const typename C2<T>::type *__restrict__ tw, int nko, int pitch) {
    typedef typename C2<T>::type T2;
    constexpr int LZ = ZTile<T>::LZ, P = PlanV<N, V>::P, E = N / P, LS = PadLen<N>::value;
    constexpr int ROWS = ZLine<T>::ROWS;
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *xch = reinterpret_cast<T2 *>(kf_smem);  // [LZ][LS]
    const int p = threadIdx.x % P, l = threadIdx.x / P;
    const int r = ROWS * (blockIdx.x * LZ + l);
    T2 *line = xch + l * LS;
    const PadAddr pa;
    // a lone row's imaginary part, not known to the compiler: the transform's
    // operations are those of any line
    T zero = (T)0;
    if constexpr (ROWS == 1) asm volatile("" : "+f"(zero));
    T2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int z = reg_row<N, P, PlanV<N, V>::R1>(p, q);
        auto get = [&](int row) {
            const long i = (long)row * N + z;
            constexpr long half = (long)N * N * (N / 2);
            return (T)(SP ? phi[((row / N + row % N + z) & 1) * half + (i >> 1)] : phi[i]);
        };
        v[q] = r < N * N ? mk<T2>(get(r), ROWS == 2 ? get(r + 1) : zero) : mk<T2>((T)0, (T)0);
    }
    PlanV<N, V>::template fft<T2, -1>(v, line, pa, p, tw);
#pragma unroll
    for (int q = 0; q < E; ++q) line[pa(reg_row<N, P, PlanV<N, V>::RL>(p, q))] = v[q];
    __syncwarp();
    if (r >= N * N) return;
    T2 *oA = out + (long)r * pitch, *oB = oA + pitch;
    for (int k = p; k < nko; k += P) {
        const T2 zk = line[pa(k)];
        const T2 zm = line[pa(k == 0 ? 0 : N - k)];
        const T cr = zm.x, ci = -zm.y;
        oA[k] = mk<T2>((T)0.5 * (zk.x + cr), (T)0.5 * (zk.y + ci));
        if (ROWS == 2) oB[k] = mk<T2>((T)0.5 * (zk.y - ci), (T)-0.5 * (zk.x - cr));
    }
}

}  // namespace kf
