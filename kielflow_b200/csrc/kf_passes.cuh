// kf_passes.cuh -- the transform passes of the spectral right-hand side.
//
// A 3-D real transform of the reference's layout (real n^3, half spectrum
// n x n x (n/2+1), z fastest; field_base.hpp:23-24, field_imag.cpp:16) is done
// in three passes, each one read and one write of HBM:
//   inverse : x pass (complex) -> y pass (complex) -> z pass (c2r, x 1/N)
//   forward : z pass (r2c)     -> y pass (complex) -> x pass (complex)
// The x and y passes load a tile of TC contiguous columns by the whole line
// (coalesced 128-byte row segments), transform it with the Stockham engine and
// store it back in place of the same tile of another buffer.  The z passes
// pack two real rows into one complex line (z = a + i b).  Loads apply the
// spectral multipliers of the right-hand side (2/3 mask, i k) so derivative
// fields are generated on the fly instead of being written out.
#pragma once

#include "kf_fft.cuh"
#include "kf_types.cuh"

namespace kf {

// Columns per x/y-pass tile: one 128-byte row segment per line by default.
#ifndef KF_TC64
#define KF_TC64 8
#endif
#ifndef KF_TC32
#define KF_TC32 16
#endif
template <typename T> struct Tile { static constexpr int TC = sizeof(T) == 8 ? KF_TC64 : KF_TC32; };


template <typename T2>
__device__ __forceinline__ T2 mul_ik(T2 a, decltype(T2::x) k) {  // i k a
    return mk<T2>(-k * a.y, k * a.x);
}

// --------------------------------------------------------------- x / y pass
// axis 0: columns are the flattened (j, kz) plane, line index i, stride n*nzc.
// axis 1: columns are kz within an x-plane, line index j, stride nzc.
// gridDim.x = njobs * ntiles (job fastest so that jobs sharing an input run
// together and hit L2).
template <typename T, int N, int SIGN>
__global__ void __launch_bounds__(Tile<T>::TC * Plan<N>::P)
k_axis_pass(const AxisJob *__restrict__ jobs, int njobs, int axis, Geo<T> g,
            const typename C2<T>::type *__restrict__ tw) {
    typedef typename C2<T>::type T2;
    constexpr int TC = Tile<T>::TC, P = Plan<N>::P, E = N / P;
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *sm = reinterpret_cast<T2 *>(kf_smem);
    const int job = blockIdx.x % njobs, tile = blockIdx.x / njobs;
    const AxisJob J = jobs[job];
    const T2 *__restrict__ in = static_cast<const T2 *>(J.in);
    T2 *__restrict__ out = static_cast<T2 *>(J.out);
    const int c = threadIdx.x % TC, p = threadIdx.x / TC;
    const int n = g.n, nzc = g.nzc;
    long base;
    long rstride;
    int jj = 0, kk = 0;
    bool valid;
    if (axis == 0) {
        const int col = tile * TC + c;
        valid = col < n * nzc;
        base = col;
        rstride = (long)n * nzc;
        jj = col / nzc;
        kk = col - jj * nzc;
    } else {
        const int tpp = (nzc + TC - 1) / TC;
        const int plane = tile / tpp;
        kk = (tile - plane * tpp) * TC + c;
        valid = kk < nzc;
        base = (long)plane * n * nzc + kk;
        rstride = nzc;
    }
    const int pbnd = valid && (J.mul == MUL_P || J.mul == MUL_P_IK) ? dealias_bound(g.pb, jj, kk, g.nzc) : -2;
    T2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int row = reg_row<N, P, Plan<N>::R1>(p, q);
        T2 x = valid ? in[base + row * rstride] : mk<T2>((T)0, (T)0);
        if (J.mul == MUL_P || J.mul == MUL_P_IK) {
            if (!dealias_keep_b(g.q2, g.thr, pbnd, g.n, row, jj, kk)) x = mk<T2>((T)0, (T)0);
        }
        if (J.mul == MUL_P_IK || J.mul == MUL_IK) x = mul_ik(x, g.kv[row]);
        v[q] = x;
    }
    Plan<N>::template fft<T2, SIGN>(v, sm + c, StrideAddr{TC}, p, tw);
    if (valid) {
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int row = reg_row<N, P, Plan<N>::RL>(p, q);
            out[base + row * rstride] = v[q];
        }
    }
}

// ------------------------------------------------- pipelined x / y pass
// The x / y pass as a persistent kernel: each block walks tiles t, t + grid,
// ... and while tile t is transformed in registers, the loads of the next
// tile are in flight as cp.async copies into a staging buffer (shared memory
// beside the exchange buffer).  Every thread stages exactly the elements it
// later reads, so the staging buffer needs no barrier; the exchange buffer
// keeps the FFT's own.  Same tiles, multipliers, transforms and stores as
// k_axis_pass, so the same results.  The 2/3 rule (MUL_P, MUL_P_IK) is applied
// by the bounds of AX_XM, the mode of every masked launch.
__device__ __forceinline__ void cp_async_copy(void *smem, const float2 *g) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_copy(void *smem, const double2 *g) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING) : "memory");
}

template <typename T> struct AxisTile {
    typedef typename C2<T>::type T2;
    const T2 *in;
    T2 *out;
    int base, rstride;   // element indices: n * n * (n/2 + 1) < 2^31 for every supported n
    int obase, ostride;  // of the output
    int mul;
    int lb, sb;  // rows r with min(r, N - r) <= lb are loaded (the others are zero), <= sb stored
    bool valid;
};

// min(r, N - r), the |frequency| of row r
template <int N> __device__ __forceinline__ int row_freq(int r) { return r <= N / 2 ? r : N - r; }

// Tile `tile` of job `job` (global tile index tile * njobs + job), column c.
template <typename T, int N>
__device__ __forceinline__ AxisTile<T> axis_tile(const AxisJob *__restrict__ jobs, int job, int tile, int axis,
                                                 int c, const AxTrunc &A, const Geo<T> &g) {
    typedef typename C2<T>::type T2;
    constexpr int TC = Tile<T>::TC, n = N, nzc = N / 2 + 1;
    AxisTile<T> G;
    const AxisJob J = jobs[job];
    G.in = static_cast<const T2 *>(J.in);
    G.out = static_cast<T2 *>(J.out);
    G.mul = J.mul;
    G.lb = G.sb = N / 2;
    if (axis == 0) {
        G.rstride = n * A.ip;
        G.ostride = n * A.op;
        if (A.mode == AX_XM) {
            const int w = A.tl[tile], j = w >> 16, kk = (w & 0xffff) + c;
            G.base = j * A.ip + kk;
            G.obase = j * A.op + kk;
            G.lb = kk < A.nkz ? g.pb[j * nzc + kk] : -1;
            G.valid = G.lb >= 0;
        } else if (A.mode == AX_XF) {
            const int w = A.tl[tile], j = w >> 16, kk = (w & 0xffff) + c;
            G.base = j * A.ip + kk;
            G.obase = j * A.op + kk;
            G.valid = kk < A.nkz && row_freq<N>(j) <= A.jb[kk];
        } else {
            G.base = tile * TC + c;
            G.valid = G.base < n * nzc;
            G.obase = A.mode == AX_XB ? G.base - __ldg(A.win) * n * nzc : G.base;
        }
    } else {
        constexpr int tpp = (nzc + TC - 1) / TC;
        int plane, kk;
        if (A.mode == AX_FULL || A.mode == AX_YB) {
            plane = tile / tpp;
            kk = (tile - plane * tpp) * TC + c;
            G.valid = kk < nzc;
        } else {
            const int tq = (A.nkz + TC - 1) / TC;
            plane = __float2int_rd(((float)tile + 0.5f) * A.itpp);  // tile / tq (exact: tile < 2^13)
            kk = (tile - plane * tq) * TC + c;
            G.valid = kk < A.nkz;
            const int b = G.valid ? A.jb[kk] : -1;
            if (A.mode == AX_YI)
                G.lb = b;
            else
                G.sb = b;
        }
        G.base = plane * n * A.ip + kk;
        G.rstride = A.ip;
        G.ostride = A.op;
        G.obase = plane * n * A.op + kk;
        if (A.mode == AX_YB) {
            const RowBox w(A.win);
            G.obase = (plane * w.bj - w.j0) * nzc + kk;
        }
    }
    return G;
}

// Resident blocks per SM that the transform kernels ask the register
// allocator for: as many as their shared memory allows (TILES tiles of
// N x TC elements per block), at most CAP, and no more than leave FLOOR
// registers per thread.  Without this bound the allocator spends 128-224
// registers per thread on the 256-point transforms and two blocks fit; with
// it the same code fits 64-85 registers (FP32) without spilling (k_x_filter with the
// first plan, two transforms in one kernel, spills 60 bytes at 64 registers).
template <typename T, int N, int V, int TILES, int CAP, int FLOOR> struct PipeMinBlocks {
    static constexpr long threads = (long)Tile<T>::TC * PlanV<N, V>::P;
    static constexpr long smem = (long)TILES * N * Tile<T>::TC * sizeof(typename C2<T>::type);
    static constexpr long by_smem = (227L * 1024) / smem;
    static constexpr long by_regs = 65536L / (threads * FLOOR);
    static constexpr long lim = by_smem < by_regs ? by_smem : by_regs;
    static constexpr int value = lim < 1 ? 1 : (lim < CAP ? (int)lim : CAP);
};

// Staging slots per k_axis_pipe block: the tile being transformed was loaded
// into one slot while the next KF_PIPE_DEPTH - 1 tiles load into the others.
// (Two slots, 96 KB per block at 256^3, measured slower: 13.5 against 12.2 ms
// for the 48 inverse launches of a 20-step run; the shared memory they take
// from the L1 cache is what the twiddle and table loads hit.)
#ifndef KF_PIPE_DEPTH
#define KF_PIPE_DEPTH 1
#endif

// Shared memory of a k_axis_pipe launch: the exchange tile and KF_PIPE_DEPTH
// staging tiles.  (Held to fewer registers for three resident blocks, or with
// its twiddles, k values and job descriptors staged in shared memory, the
// one-slot pass measured no faster: 12.5 and 13.8 ms against 12.4 ms for 48
// launches.)
template <typename T, int N> inline size_t axis_pipe_smem(int) {
    return (1 + KF_PIPE_DEPTH) * (size_t)N * Tile<T>::TC * sizeof(typename C2<T>::type);
}

// Resident blocks per SM asked of the register allocator for k_axis_pipe
// (0: no request; 3 fits the FP32 256-point pass in 80 registers without
// spilling: its 48 inverse launches of 20 steps took 12.0-12.1 ms against
// 13.7 ms with 125 registers and 2 blocks), and for the FP32 k_z_c2r (12
// blocks, 40 registers with spills: 8.0 against 7.5 ms; not used).
#ifndef KF_PIPE_MINB
#define KF_PIPE_MINB 3
#endif
#ifndef KF_ZC2R_MINB
#define KF_ZC2R_MINB 0
#endif

template <typename T, int N, int SIGN, int V = 0>
__global__ void __launch_bounds__(Tile<T>::TC * PlanV<N, V>::P,
                                  (KF_PIPE_MINB ? PipeMinBlocks<T, N, V, 1 + KF_PIPE_DEPTH, (KF_PIPE_MINB > 0 ? KF_PIPE_MINB : 1), 64>::value : 1))
k_axis_pipe(const AxisJob *__restrict__ jobs, int njobs, int axis, Geo<T> g,
            const typename C2<T>::type *__restrict__ tw, int total, AxTrunc A) {
    typedef typename C2<T>::type T2;
    constexpr int TC = Tile<T>::TC, P = PlanV<N, V>::P, E = N / P, NZC = N / 2 + 1;
    constexpr int D = KF_PIPE_DEPTH;
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *sm = reinterpret_cast<T2 *>(kf_smem);  // exchange [N][TC]
    T2 *stg0 = sm + N * TC;                     // staging  [D][N][TC]
    const int c = threadIdx.x % TC, p = threadIdx.x / TC;
    int t = blockIdx.x;
    // the rows that the window modes store
    const bool win = A.mode == AX_XB || A.mode == AX_YB;
    int w0 = 0, wn = N;
    if (win) {
        const RowBox w(A.win);
        w0 = A.mode == AX_XB ? w.i0 : w.j0;
        wn = A.mode == AX_XB ? w.bi : w.bj;
        if (A.mode == AX_YB || w.bi == 0) total = njobs * w.bi * ((NZC + TC - 1) / TC);
    }
    if (t >= total) return;
    // (job, tile) of global tile t = tile * njobs + job, advanced by the grid
    // stride without a division per tile: for the tile being transformed (c*)
    // and for the next one to stage (p*)
    const int GS = gridDim.x, Gq = GS / njobs, Gr = GS - Gq * njobs;
    auto adv = [&](int &j, int &tl) {
        j += Gr;
        tl += Gq;
        if (j >= njobs) {
            j -= njobs;
            ++tl;
        }
    };
    int cj = t % njobs, ct = t / njobs;
    int pj = cj, pt = ct, ptt = t;
    // Each thread stages exactly the elements it reads back, so the slots need
    // no barrier.  One commit group per tile (empty past the end), so that
    // cp.async.wait_group D - 1 always leaves the current tile complete.
    auto prefetch = [&](int slot) {
        if (ptt < total) {
            const AxisTile<T> G = axis_tile<T, N>(jobs, pj, pt, axis, c, A, g);
            T2 *st = stg0 + slot * (N * TC);
#pragma unroll
            for (int q = 0; q < E; ++q) {
                const int row = reg_row<N, P, PlanV<N, V>::R1>(p, q);
                T2 *dst = st + row * TC + c;
                if (G.valid && row_freq<N>(row) <= G.lb)
                    cp_async_copy(dst, G.in + G.base + row * G.rstride);
                else
                    *dst = mk<T2>((T)0, (T)0);
            }
        }
        cp_async_commit();
        ptt += GS;
        adv(pj, pt);
    };
#pragma unroll
    for (int d = 0; d < D; ++d) prefetch(d);
    for (int it = 0; t < total; t += GS, ++it) {
        const int slot = it % D;
        const AxisTile<T> cur = axis_tile<T, N>(jobs, cj, ct, axis, c, A, g);
        adv(cj, ct);
        cp_async_wait<D - 1>();
        const T2 *stg = stg0 + slot * (N * TC);
        T2 v[E];
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int row = reg_row<N, P, PlanV<N, V>::R1>(p, q);
            T2 x = stg[row * TC + c];  // AX_XM: zeros staged outside the 2/3 rule
            if (cur.mul == MUL_P_IK || cur.mul == MUL_IK) x = mul_ik(x, g.kv[row]);
            v[q] = x;
        }
        prefetch(slot);
        PlanV<N, V>::template fft<T2, SIGN>(v, sm + c, StrideAddr{TC}, p, tw);
        if (cur.valid) {
#pragma unroll
            for (int q = 0; q < E; ++q) {
                const int row = reg_row<N, P, PlanV<N, V>::RL>(p, q);
                if (win ? (unsigned)(row - w0) < (unsigned)wn : row_freq<N>(row) <= cur.sb) cur.out[cur.obase + row * cur.ostride] = v[q];
            }
        }
    }
}

// --------------------------------------------------------------- z c2r pass
// LZ line pairs per block; thread = p + P*l.  Half rows are staged in shared
// memory, multiplied, extended by Hermitian symmetry (the imaginary parts of
// the kz = 0 and kz = n/2 bins are dropped, as a c2r transform does), packed
// as A + iB, transformed backwards and written as two real rows scaled by
// `scale` (the 1/N of OP_iFFT.cpp:59-61).
// Line pairs per z-pass block (4 and 16 measured no faster than 8 at 256^3:
// the c2r launches took 7.36 and 8.01 ms against 7.33 ms over 20 steps).
#ifndef KF_ZLZ
#define KF_ZLZ 8
#endif
template <typename T> struct ZTile { static constexpr int LZ = KF_ZLZ; };

// Shared memory of a z pass: its line buffers (the c2r staging of two half
// spectra per line pair, reused by the transform).
template <typename T, int N, bool C2R> struct ZSmem {
    typedef typename C2<T>::type T2;
    static constexpr int LZ = ZTile<T>::LZ, NZC = N / 2 + 1, LS = PadLen<N>::value;
    static constexpr int lines = C2R ? (2 * LZ * NZC > LZ * LS ? 2 * LZ * NZC : LZ * LS) : LZ * LS;
    static constexpr size_t bytes = (size_t)lines * sizeof(T2);
};

template <typename T, int N, int V = 0>
__global__ void __launch_bounds__(ZTile<T>::LZ * PlanV<N, V>::P, (sizeof(T) == 4 && KF_ZC2R_MINB > 0 ? KF_ZC2R_MINB : 1))
k_z_c2r(const ZJob *__restrict__ jobs, int njobs, int nrows, Geo<T> g,
        const typename C2<T>::type *__restrict__ tw, T scale, int nkz, int pitch, const int *__restrict__ win) {
    typedef typename C2<T>::type T2;
    constexpr int LZ = ZTile<T>::LZ, P = PlanV<N, V>::P, E = N / P, NZC = N / 2 + 1;
    constexpr int LS = PadLen<N>::value;  // padded line of the exchange buffer
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *half = reinterpret_cast<T2 *>(kf_smem);  // [2][LZ][NZC], staging of the half spectra
    T2 *xch = half;                              // [LZ][LS], reused by the transform once staged
    const int job = blockIdx.x % njobs, tile = blockIdx.x / njobs;
    const int r0 = tile * LZ;
    if (win) {  // the window's rows, packed
        const RowBox w(win);
        nrows = w.bi * w.bj;
        if (r0 >= nrows) return;
    }
    const ZJob J = jobs[job];
    const T2 *inA = static_cast<const T2 *>(J.inA);
    const T2 *inB = static_cast<const T2 *>(J.inB);
    const int p = threadIdx.x % P, l = threadIdx.x / P;
    // raw half spectra -> shared memory with asynchronous copies (all of a
    // thread's loads in flight at once); the multipliers are applied below.
    const int lim = (nrows - r0) * NZC;  // elements of the run inside the field
    const long off = (long)r0 * NZC;
    if (nkz == NZC) {
        // the tile's LZ rows of a half spectrum are one contiguous run of
        // LZ * NZC elements from row r0
        for (int e = threadIdx.x; e < LZ * NZC; e += blockDim.x) {
            if (e < lim) {
                cp_async_copy(half + e, inA + off + e);
                if (inB)
                    cp_async_copy(half + LZ * NZC + e, inB + off + e);
                else
                    half[LZ * NZC + e] = mk<T2>((T)0, (T)0);
            } else {
                half[e] = mk<T2>((T)0, (T)0);
                half[LZ * NZC + e] = mk<T2>((T)0, (T)0);
            }
        }
    } else {
        // spectra that are zero from kz = nkz on, rows of `pitch` elements
        const long ro = (long)(r0 + l) * pitch;
        for (int k = p; k < nkz; k += P) {
            const int e = l * NZC + k;
            if (r0 + l < nrows) {
                cp_async_copy(half + e, inA + ro + k);
                if (inB)
                    cp_async_copy(half + LZ * NZC + e, inB + ro + k);
                else
                    half[LZ * NZC + e] = mk<T2>((T)0, (T)0);
            } else {
                half[e] = mk<T2>((T)0, (T)0);
                half[LZ * NZC + e] = mk<T2>((T)0, (T)0);
            }
        }
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    const T2 *hA = half + l * NZC;
    const T2 *hB = half + LZ * NZC + l * NZC;
    // staged element kk (0 <= kk < NZC) times its job's multiplier, with the
    // imaginary parts of the kz = 0 and kz = n/2 bins dropped
    auto staged = [&](const T2 *h, int kk, int mul) {
        if (kk >= nkz) return mk<T2>((T)0, (T)0);
        T2 x = h[kk];
        if (mul == MUL_IK) x = mul_ik(x, g.kv[kk]);
        if (mul == MUL_HALF && kk > 0 && 2 * kk < N) x = mk<T2>((T)0.5 * x.x, (T)0.5 * x.y);
        if (kk == 0 || 2 * kk == N) x.y = (T)0;
        return x;
    };
    T2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int k = reg_row<N, P, PlanV<N, V>::R1>(p, q);
        T2 a, b;
        if (k < NZC) {
            a = staged(hA, k, J.mulA);
            b = staged(hB, k, J.mulB);
        } else {
            a = staged(hA, N - k, J.mulA);
            b = staged(hB, N - k, J.mulB);
            a.y = -a.y;
            b.y = -b.y;
        }
        v[q] = mk<T2>(a.x - b.y, a.y + b.x);  // A + iB
    }
    __syncthreads();  // staging consumed: the exchange buffer may overwrite it
    PlanV<N, V>::template fft<T2, +1>(v, xch + l * LS, PadAddr{}, p, tw);
    const int r = r0 + l;
    if (r < nrows) {
        T *oA = static_cast<T *>(J.outA) + (long)r * N;
        T *oB = J.outB ? static_cast<T *>(J.outB) + (long)r * N : nullptr;
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int z = reg_row<N, P, PlanV<N, V>::RL>(p, q);
            oA[z] = v[q].x * scale;
            if (oB) oB[z] = v[q].y * scale;
        }
    }
}

// --------------------------------------------------------------- z r2c pass
template <typename T, int N, int V = 0>
__global__ void __launch_bounds__(ZTile<T>::LZ * PlanV<N, V>::P)
k_z_r2c(const ZJob *__restrict__ jobs, int njobs, int nrows,
        const typename C2<T>::type *__restrict__ tw, int pitch) {
    typedef typename C2<T>::type T2;
    constexpr int LZ = ZTile<T>::LZ, P = PlanV<N, V>::P, E = N / P;
    constexpr int LS = PadLen<N>::value;
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *xch = reinterpret_cast<T2 *>(kf_smem);  // [LZ][LS], padded lines
    const int job = blockIdx.x % njobs, tile = blockIdx.x / njobs;
    const ZJob J = jobs[job];
    const int r0 = tile * LZ;
    const int p = threadIdx.x % P, l = threadIdx.x / P;
    const int r = r0 + l;
    const T *iA = static_cast<const T *>(J.inA);
    const T *iB = static_cast<const T *>(J.inB);
    T2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int z = reg_row<N, P, PlanV<N, V>::R1>(p, q);
        T a = (T)0, b = (T)0;
        if (r < nrows) {
            a = iA[(long)r * N + z];
            if (iB) b = iB[(long)r * N + z];
        }
        v[q] = mk<T2>(a, b);
    }
    T2 *line = xch + l * LS;
    const PadAddr pa;
    PlanV<N, V>::template fft<T2, -1>(v, line, pa, p, tw);
#pragma unroll
    for (int q = 0; q < E; ++q) line[pa(reg_row<N, P, PlanV<N, V>::RL>(p, q))] = v[q];
    __syncthreads();
    const int lim = (nrows - r0) * pitch;
    T2 *oA = static_cast<T2 *>(J.outA) + (long)r0 * pitch;
    T2 *oB = J.outB ? static_cast<T2 *>(J.outB) + (long)r0 * pitch : nullptr;
    // the tile's LZ output rows of `pitch` elements (of NZC) are one contiguous run
    // from row r0
    for (int idx = threadIdx.x; idx < LZ * pitch && idx < lim; idx += blockDim.x) {
        const int ll = idx / pitch, k = idx - ll * pitch;
        const T2 zk = xch[ll * LS + pa(k)];
        const T2 zm = xch[ll * LS + pa(k == 0 ? 0 : N - k)];
        const T cr = zm.x, ci = -zm.y;  // conj(Z[N-k])
        oA[idx] = mk<T2>((T)0.5 * (zk.x + cr), (T)0.5 * (zk.y + ci));
        if (oB) oB[idx] = mk<T2>((T)0.5 * (zk.y - ci), (T)-0.5 * (zk.x - cr));
    }
}

// ------------------------------ forward x pass + assembly + RK4 stage update
// One block transforms one column tile of one of the four fields and finishes
// the right-hand side there,
//   K_q = -lin_q + F_q                             (rhs_standard.cpp:538-560)
// with -lin_q from k_lin and F_q the transform of the physical part (k_zprod; lin[q]
// == nullptr: that holds the linear terms, too);
// with penalization F_q and -lin_q are needed inside the 2/3 rule only (the
// filter after the physical-space penalization, rhs_standard.cpp:491-532): the
// active columns (A.mode AX_XM), the rows within their bounds, K being zero
// elsewhere.  What the RK4 stage does with K (RKO4.cpp:140-238) follows in
// place, so K is neither written nor read back:
//   mode 0: acc = K,      ys = y + c K
//   mode 1: acc += 2 K,   ys = y + c K
//   mode 2: y += c (acc + K), ys = y
//   mode 3: K itself (a right-hand side on its own)
// Outside the 2/3 rule K = 0, hence ys = y, which holds from the stage's start.
template <typename T> struct StageArgs {
    typedef typename C2<T>::type T2;
    const T2 *in[4], *lin[4];
    T2 *y[4], *acc[4], *ys[4], *K[4];
    T c;
    int mode;
};

template <typename T, int N, int V = 0>
__global__ void __launch_bounds__(Tile<T>::TC * PlanV<N, V>::P,
                                  PipeMinBlocks<T, N, V, 1, sizeof(T) == 4 ? 4 : 2, 64>::value)
k_xfwd_stage(const __grid_constant__ StageArgs<T> a, Geo<T> g, const typename C2<T>::type *__restrict__ tw, AxTrunc A) {
    typedef typename C2<T>::type T2;
    constexpr int TC = Tile<T>::TC, P = PlanV<N, V>::P, E = N / P, NZC = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char kf_smem[];
    T2 *sm = reinterpret_cast<T2 *>(kf_smem);
    const int q = blockIdx.x & 3, tile = blockIdx.x >> 2;
    const int c = threadIdx.x % TC, p = threadIdx.x / TC;
    constexpr int rstride = N * NZC;
    int col = tile * TC + c, icol = col, b = N / 2;
    bool valid = col < N * NZC;
    if (A.mode == AX_XM) {
        const int w = A.tl[tile];
        const int kk = (w & 0xffff) + c;
        col = (w >> 16) * NZC + kk;
        icol = (w >> 16) * A.ip + kk;
        b = kk < A.nkz ? g.pb[col] : -1;
        valid = b >= 0;
    }
    const int istride = N * A.ip;
    const T2 *__restrict__ in = a.in[q];
    T2 v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int row = reg_row<N, P, PlanV<N, V>::R1>(p, e);
        v[e] = valid ? in[icol + row * istride] : mk<T2>((T)0, (T)0);
    }
    PlanV<N, V>::template fft<T2, -1>(v, sm + c, StrideAddr{TC}, p, tw);
    if (!valid) return;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = reg_row<N, P, PlanV<N, V>::RL>(p, e);
        if (row_freq<N>(i) > b) continue;
        const int idx = col + i * rstride;
        T2 k = v[e];
        if (a.lin[q]) {
            const T2 l = a.lin[q][idx];
            k = mk<T2>(l.x + v[e].x, l.y + v[e].y);
        }
        if (a.mode == 3) {
            a.K[q][idx] = k;
            continue;
        }
        const T2 y = a.y[q][idx];
        if (a.mode == 2) {
            const T2 s = a.acc[q][idx];
            const T2 r = mk<T2>(y.x + a.c * (s.x + k.x), y.y + a.c * (s.y + k.y));
            a.y[q][idx] = r;
            a.ys[q][idx] = r;
        } else {
            T2 s = k;
            if (a.mode == 1) {
                s = a.acc[q][idx];
                s = mk<T2>(s.x + (T)2 * k.x, s.y + (T)2 * k.y);
            }
            a.acc[q][idx] = s;
            a.ys[q][idx] = mk<T2>(y.x + a.c * k.x, y.y + a.c * k.y);
        }
    }
}

}  // namespace kf
