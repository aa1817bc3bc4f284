// kf_split.cuh -- the FAS cycle on colour-split levels.
//
// A level's points are stored by colour: element (i, j, k) of colour c = (i + j +
// k) & 1 at c n^3/2 + (i n + j) n/2 + k/2.  A red-black half sweep then reads its
// own colour and the other one as whole rows: in the natural order a warp's
// k = 2 k2 + parity loads used every second element of what they fetched, and the
// half sweep was bound by L1 (87 % busy, 3.75 TB/s from DRAM at 256^3).  The
// restriction's even and odd k and the injection (colour 0) are contiguous, too.
// Every point's operations and their order are those of the natural-order
// kernels (kf_poisson.cuh), so the potentials are the same bit for bit.
#pragma once

#include "kf_graph.cuh"
#include "kf_poisson.cuh"

namespace kf {

// One colour-split level: n even, h = n / 2, H = n h n elements per colour.
// Axis tables as in Lev; *k hold an axis by parity (even entries, then odd).
struct SLev {
    int n;
    const double *dd, *ip, *im;     // by index
    const double *ddk, *ipk, *imk;  // [parity * h + k / 2]
};

// Split order -> natural (k_split's inverse).
__global__ void __launch_bounds__(256) k_unsplit(const double *__restrict__ s, double *__restrict__ x, int n) {
    const int k2 = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (2 * k2 >= n || j >= n) return;
    const int row = (i * n + j) * (n / 2) + k2, half = n * n * (n / 2), c0 = (i + j) & 1;
    *reinterpret_cast<double2 *>(x + 2 * row) = make_double2(s[c0 * half + row], s[(c0 ^ 1) * half + row]);
}

// k_guess with the start of the solve in split order, from phi or (phi == nullptr)
// from the last solution in s: blocks as k_split.
__global__ void __launch_bounds__(256) k_guess_s(const double *__restrict__ phi, double *__restrict__ phi_a,
                                                 double *__restrict__ s, const DevTime *__restrict__ d, double xt,
                                                 int n) {
    const int k2 = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (2 * k2 >= n || j >= n) return;
    const double t = d->t + xt, ta = d->tau_a, tb = d->tau_b;
    const int nh = d->nhist;
    const int row = (i * n + j) * (n / 2) + k2, half = n * n * (n / 2), c0 = (i + j) & 1;
    double2 b = phi ? *reinterpret_cast<const double2 *>(phi + 2 * row)
                    : make_double2(s[c0 * half + row], s[(c0 ^ 1) * half + row]);
    const bool newtime = nh != 0 && t != tb;
    if (!phi && !newtime) return;
    if (newtime) {
        double2 *pa = reinterpret_cast<double2 *>(phi_a + 2 * row);
        const double2 o = b;
        if (nh >= 2) {
            const double w = (t - tb) / (tb - ta);
            const double2 a = *pa;
            b.x = __dadd_rn(b.x, __dmul_rn(w, __dsub_rn(b.x, a.x)));
            b.y = __dadd_rn(b.y, __dmul_rn(w, __dsub_rn(b.y, a.y)));
        }
        *pa = o;
    }
    s[c0 * half + row] = b.x;
    s[(c0 ^ 1) * half + row] = b.y;
}

// One colour of a level, two points of a row per thread (elements k2 = 2 t and
// 2 t + 1: 16-byte loads, two independent chains of Newton steps or residuals).
// Block (n / 4, rows), grid (1, ceil(n / rows), n).  256^3: 51 us for the half
// sweep, 5.2 TB/s, in blocks of 64 threads as of 128 (51.3 and 50.7 us; natural
// order: 72 us); threads that march 2-16 planes with the i-neighbours in registers
// and the next plane prefetched took 68-88 us, for their 93-128 registers leave
// fewer warps.  Up to 128^3, in L2, blocks of 128 threads are faster (128^3: 8.3 us
// against 9.3 in blocks of 64; a 96^3 step 1.71 ms against 1.76).
template <typename F>
__device__ __forceinline__ void split_pair(const double *__restrict__ phi, const double *__restrict__ rho,
                                           const SLev &L, const AxTab &T, int color, int i, int j, F f) {
    const int n = L.n, h = n >> 1, H = n * n * h, k2 = 2 * threadIdx.x, st = n * h;
    const int q = (i * n + j) * h + k2, par = (i + j + color) & 1;
    const double *own = phi + color * H, *oth = phi + (color ^ 1) * H;
    auto ld = [](const double *p) { return *reinterpret_cast<const double2 *>(p); };
    const double2 im = ld(oth + (i == 0 ? q + (n - 1) * st : q - st));
    const double2 ip = ld(oth + (i == n - 1 ? q - (n - 1) * st : q + st));
    const double2 jp = ld(oth + (j == n - 1 ? q - (n - 1) * h : q + h));
    const double2 jm = ld(oth + (j == 0 ? q + (n - 1) * h : q - h));
    const double2 kc = ld(oth + q), x = ld(own + q), r = ld(rho + color * H + q);
    // the k-neighbour outside the pair
    const double ke = oth[q + (par ? (k2 + 2 == h ? 2 - h : 2) : (k2 == 0 ? h - 1 : -1))];
    const double2 kp = par ? make_double2(kc.y, ke) : kc;
    const double2 km = par ? kc : make_double2(ke, kc.x);
    const int kt = par * h + k2;
    const double2 dk = ld(L.ddk + kt), ipk = ld(L.ipk + kt), imk = ld(L.imk + kt);
    const double dij = __dadd_rn(T.dd[i], T.dd[j]);
    auto point = [&](double a, double b, double c, double d, double e, double g, double rr, double wp, double wm) {
        double A = __dmul_rn(a, T.ip[i]);
        A = __dadd_rn(A, __dmul_rn(b, T.im[i]));
        A = __dadd_rn(A, __dmul_rn(c, T.ip[j]));
        A = __dadd_rn(A, __dmul_rn(d, T.im[j]));
        A = __dadd_rn(A, __dmul_rn(e, wp));
        A = __dadd_rn(A, __dmul_rn(g, wm));
        return __dadd_rn(A, rr);
    };
    const double A0 = point(ip.x, im.x, jp.x, jm.x, kp.x, km.x, r.x, ipk.x, imk.x);
    const double A1 = point(ip.y, im.y, jp.y, jm.y, kp.y, km.y, r.y, ipk.y, imk.y);
    f(color * H + q, x, A0, A1, __dadd_rn(dij, dk.x), __dadd_rn(dij, dk.y));
}

// One red-black half sweep (k_rbgs_t's point update).
__global__ void __launch_bounds__(128) k_rbgs_s(double *phi, const double *__restrict__ rho, SLev L, int color,
                                                double om, const __grid_constant__ AxTab T) {
    const int j = blockIdx.y * blockDim.y + threadIdx.y, i = blockIdx.z;
    if (j >= L.n) return;
    split_pair(phi, rho, L, T, color, i, j, [&](int q, double2 x, double A0, double A1, double D0, double D1) {
        *reinterpret_cast<double2 *>(phi + q) = make_double2(newton_step(x.x, A0, D0, om), newton_step(x.y, A1, D1, om));
    });
}

// The residual r = f(phi) of the level (k_residual<true>); MAX: max |r| into the
// slots as well.  A block takes Z consecutive (plane, colour) pairs, grid (1,
// ceil(n / rows), 2 n / Z): with one pair per block the warps' atomics on the slots
// cost a third of the time (256^3: 117 us; Z = 4 91 us, without the maximum 80 us;
// more pairs leave too few blocks).
template <bool MAX>
__global__ void __launch_bounds__(128) k_residual_s(const double *__restrict__ phi, const double *__restrict__ rho,
                                                    SLev L, double *__restrict__ r,
                                                    unsigned long long *__restrict__ slots, int Z,
                                                    const __grid_constant__ AxTab T) {
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    unsigned long long af = 0;  // |r| as bit patterns: a NaN sorts above +inf
    if (j < L.n)
#pragma unroll 1
        for (int z = blockIdx.z * Z; z < (int)(blockIdx.z + 1) * Z; ++z)
            split_pair(phi, rho, L, T, z & 1, z >> 1, j,
                       [&](int q, double2 x, double A0, double A1, double D0, double D1) {
                           const double2 v = make_double2(f_point(A0, D0, x.x), f_point(A1, D1, x.y));
                           *reinterpret_cast<double2 *>(r + q) = v;
                           if (MAX)
                               af = max(af, max((unsigned long long)__double_as_longlong(fabs(v.x)),
                                                (unsigned long long)__double_as_longlong(fabs(v.y))));
                       });
    if constexpr (MAX) {
        // per warp, by 32-bit halves; the lanes past the last row hold 0.  Which lanes
        // there are follows from the block's size: after the branch above a warp need
        // not be together, and a part of it without lane 0 would not post its maximum
        const int t = threadIdx.y * blockDim.x + threadIdx.x, left = (int)(blockDim.x * blockDim.y) - (t & ~31);
        const unsigned lanes = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
        __syncwarp(lanes);
        const unsigned hi = (unsigned)(af >> 32), mh = __reduce_max_sync(lanes, hi);
        const unsigned ml = __reduce_max_sync(lanes, hi == mh ? (unsigned)af : 0u);
        if ((t & 31) == 0)
            atomicMax(slots + ((blockIdx.y + blockIdx.z * gridDim.y + (t >> 5)) & 63),
                      ((unsigned long long)mh << 32) | ml);
    }
}

// Level n (split) -> the coarse level: full weighting of r, injection of phi into
// phic and phi0 (fw_point's and k_restrict's operations) and, with RHS, the FAS
// source N_c(phic) + rc (k_fas_rhs) in rc's place, the neighbours of phic taken
// from phi.  CS: the coarse arrays are split.  Block (32, 8), one coarse point per thread.
template <bool CS, bool RHS>
__global__ void __launch_bounds__(256) k_restrict_s(const double *__restrict__ r, const double *__restrict__ phi, int n,
                                                    Lev Lc, double *__restrict__ rc, double *__restrict__ phic,
                                                    double *__restrict__ phi0) {
    const int nc = n >> 1, h = nc, H = n * n * h;
    const int K = blockIdx.x * 32 + threadIdx.x, J = blockIdx.y * 8 + threadIdx.y, I = blockIdx.z;
    if (K >= nc || J >= nc) return;
    const int Km = K == 0 ? h - 1 : K - 1;  // k = 2 K - 1
    const double w[3] = {0.25, 0.5, 0.25};
    double s = 0.;
#pragma unroll
    for (int a = -1; a <= 1; ++a) {
        const int i = a < 0 && I == 0 ? n - 1 : 2 * I + a;
        double sy = 0.;
#pragma unroll
        for (int b = -1; b <= 1; ++b) {
            const int j = b < 0 && J == 0 ? n - 1 : 2 * J + b;
            const int row = (i * n + j) * h, p = (a + b) & 1;  // colour of the row's even k
            const double *odd = r + (p ^ 1) * H + row;
            double sz = __dadd_rn(0., __dmul_rn(w[0], odd[Km]));
            sz = __dadd_rn(sz, __dmul_rn(w[1], r[p * H + row + K]));
            sz = __dadd_rn(sz, __dmul_rn(w[2], odd[K]));
            sy = __dadd_rn(sy, __dmul_rn(w[b + 1], sz));
        }
        s = __dadd_rn(s, __dmul_rn(w[a + 1], sy));
    }
    auto inj = [&](int ii, int jj, int kk) { return phi[(2 * ii * n + 2 * jj) * h + kk]; };  // colour 0
    const double p = inj(I, J, K);
    if constexpr (RHS) {
        const double D = __dadd_rn(__dadd_rn(Lc.dd[I], Lc.dd[J]), Lc.dd[K]);
        double A = __dmul_rn(inj(I + 1 == nc ? 0 : I + 1, J, K), Lc.ip[I]);
        A = __dadd_rn(A, __dmul_rn(inj(I == 0 ? nc - 1 : I - 1, J, K), Lc.im[I]));
        A = __dadd_rn(A, __dmul_rn(inj(I, J + 1 == nc ? 0 : J + 1, K), Lc.ip[J]));
        A = __dadd_rn(A, __dmul_rn(inj(I, J == 0 ? nc - 1 : J - 1, K), Lc.im[J]));
        A = __dadd_rn(A, __dmul_rn(inj(I, J, K + 1 == nc ? 0 : K + 1), Lc.ip[K]));
        A = __dadd_rn(A, __dmul_rn(inj(I, J, Km), Lc.im[K]));
        s = __dadd_rn(__dsub_rn(0., f_point(A, D, p)), s);
    }
    const int hc = nc >> 1;
    const int id = CS ? ((I + J + K) & 1) * nc * nc * hc + (I * nc + J) * hc + (K >> 1) : (I * nc + J) * nc + K;
    rc[id] = s;
    phic[id] = p;
    phi0[id] = p;
}

// phi (split, n) += P e with e = phic - phi0 on the coarse level (prolong_cell's
// operations on k_correction's differences), one thread per coarse cell.  CS: the
// coarse arrays are split; E: phi0 already holds e.
template <bool CS, bool E>
__global__ void __launch_bounds__(256) k_prolong_s(double *__restrict__ phi, const double *__restrict__ phic,
                                                   const double *__restrict__ phi0, const double *__restrict__ gam,
                                                   int n) {
    const int nc = n >> 1, h = nc, H = n * n * h, hc = nc >> 1;
    const int K = blockIdx.x * 32 + threadIdx.x, J = blockIdx.y * 8 + threadIdx.y, I = blockIdx.z;
    if (K >= nc || J >= nc) return;
    const int I1 = I + 1 == nc ? 0 : I + 1, J1 = J + 1 == nc ? 0 : J + 1, K1 = K + 1 == nc ? 0 : K + 1;
    auto e = [&](int ii, int jj, int kk) {
        const int id = CS ? ((ii + jj + kk) & 1) * nc * nc * hc + (ii * nc + jj) * hc + (kk >> 1) : (ii * nc + jj) * nc + kk;
        return E ? phi0[id] : __dsub_rn(phic[id], phi0[id]);
    };
    const double gz = gam[2 * K + 1], gy = gam[2 * J + 1], gx = gam[2 * I + 1];
    double zc[2][2][2], yc[2][2][2];
#pragma unroll
    for (int di = 0; di < 2; ++di)
#pragma unroll
        for (int dj = 0; dj < 2; ++dj) {
            const double c0 = e(di ? I1 : I, dj ? J1 : J, K), c1 = e(di ? I1 : I, dj ? J1 : J, K1);
            zc[di][dj][0] = c0;
            zc[di][dj][1] = __dadd_rn(__dmul_rn(1. - gz, c0), __dmul_rn(gz, c1));
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
                const double v = a == 0 ? yc[0][b][q]
                                        : __dadd_rn(__dmul_rn(1. - gx, yc[0][b][q]), __dmul_rn(gx, yc[1][b][q]));
                double *f = phi + ((a + b + q) & 1) * H + ((2 * I + a) * n + 2 * J + b) * h + K;
                *f = __dadd_rn(*f, v);
            }
}

}  // namespace kf
