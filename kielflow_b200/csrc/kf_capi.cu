// kf_capi.cu -- host driver and C ABI (include/kielflow_b200.h).
//
// The right-hand side of rhs_standard::solve (rhs_standard.cpp:89-566) is run as
// six rounds of kernels on device-resident buffers:
//   A  inverse x/y passes of s^ (P s^, i k_x P s^, i k_y P s^) and the z pass of
//      P s^  ->  s_d;  rho = exp(s_d) + n_d;  Poisson solve -> phi
//   B  phi^ = r2c(phi)                                    (E-force, :218-226)
//   C  -lin_q in k-space (k_lin); with penalization also the inverse x and y
//      passes of -lin_q (FP32) or c2r(-lin_q) on the window of rows on which the
//      mask is not zero (FP64)
//   D  inverse x / y passes generating U_c, d_d U_c, d_d s
//   E  k_zprod: their inverse z pass, the physical-space products (advection,
//      u.grad s) [+ penalization] and the forward z pass of the results
//   F  forward y pass, then the forward x pass fused with the assembly
//      K_q = -lin_q + F_q (inside the 2/3 rule with penalization) and with the
//      RK4 stage update (RKO4.cpp:50-241) that uses it
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <memory>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "../../include/kielflow_b200.h"
#include "kf_adjoint.cuh"
#include "kf_cluster.cuh"
#include "kf_graph.cuh"
#include "kf_hostpipe.hpp"
#include "kf_jacobi.cuh"
#include "kf_march.cuh"
#include "kf_passes.cuh"
#include "kf_pointwise.cuh"
#include "kf_poisson.cuh"
#include "kf_split.cuh"
#include "kf_stretch.cuh"
#include "kf_zprod.cuh"

using namespace kf;

namespace {

struct KfError {
    int code;
    std::string msg;
};

#define CK(x)                                                                                  \
    do {                                                                                       \
        cudaError_t e_ = (x);                                                                  \
        if (e_ != cudaSuccess) throw KfError{KF_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)}; \
    } while (0)

struct LevelBuf {
    int n = 0;
    double *dd = nullptr, *dp = nullptr, *dm = nullptr, *ip = nullptr, *im = nullptr, *gam = nullptr;
    double *rp = nullptr, *rm = nullptr;
    double *phi = nullptr, *rho = nullptr, *r = nullptr, *phi0 = nullptr;
    double *t = nullptr;  // second potential of the streaming smoother (k_rbgs_march), n >= MT_TK
    // colour-split form (kf_split.cuh): sp says that the half-sweep cycle keeps the
    // level's phi, rho, r and phi0 in split order; ph, rh are phi and rho so kept
    // (the finest level's are buffers of their own)
    bool sp = false;
    double *ddk = nullptr, *ipk = nullptr, *imk = nullptr;
    double *ph = nullptr, *rh = nullptr;
    SLev slev() const { return SLev{n, dd, ip, im, ddk, ipk, imk}; }
    std::shared_ptr<AxTab> tab;  // host copy of dd, ip, im (kernel parameter of the half sweeps)
    Lev lev() const { return Lev{n, dd, dp, dm, ip, im, rp, rm}; }
};

constexpr int RBS = 256;  // reduction block size

// Sweeps in the body of the Jacobi loop's WHILE node (even: they alternate
// between the two potentials).
constexpr int JC_UNROLL = 16;

// The sweep loop of one level and stop rule, captured on first use.
struct JacGraph {
    const double *phi, *tmp, *rho;
    JacStop stop;
    cudaGraphExec_t exec;
};

struct AdjState;  // discrete-adjoint buffers (allocated by the first kf_adjoint_run)
struct OutState;  // output buffers of kf_run / kf_get_output (allocated on first use)

}  // namespace

struct kf_ctx {
    kf_config cfg;
    int n = 0, nzc = 0;
    long N = 0, Nc = 0;
    bool fp32 = false;
    size_t es = 8, cs = 16;
    cudaStream_t st = nullptr;
    bool own_stream = false;
    std::string err;
    long long launches = 0;
    std::vector<void *> allocs;
    HostPipe pipe;  // pageable host arrays (put_host, get_host)

    void *Y[4] = {}, *Ys[4] = {}, *ACC[4] = {}, *K[4] = {};
    void *CX[12] = {}, *CY[16] = {}, *R[24] = {}, *phihat = nullptr, *LIN[4] = {};
    double *phi = nullptr, *rho = nullptr, *nd = nullptr;
    double *rho_cs = nullptr, *phi_cs = nullptr;  // the finest rho and phi in split order
    void *H = nullptr;
    void *kv = nullptr, *SV = nullptr, *PF = nullptr;
    void *tw[2] = {};  // twiddles of the two radix plans (plan_twiddles)
    double *q2 = nullptr;
    int *pb = nullptr;  // x-pass 2/3-rule bounds per (j, kz) column (dealias_bounds)
    // active columns of a half spectrum (AxTrunc): the 2/3 rule's, and those on which
    // the phi filter table is not 0
    struct Cols {
        int nkz = 0, nt = 0, mp = 0;  // mp: elements per row of the intermediates
        int *jb = nullptr, *tl = nullptr;
        double cols = 0.;  // elements of the active columns
    };
    Cols tr, pf;
    double tr_ball = 0.;  // elements the 2/3 rule keeps
    double *stage64 = nullptr;
    std::vector<LevelBuf> lv;
    double *partial = nullptr;
    int npartial = 0;
    double *red = nullptr;
    double *h_red = nullptr;
    int *d_sweeps = nullptr;
    unsigned long long *d_max = nullptr, *h_max = nullptr;
    int *d_err = nullptr, *h_err = nullptr;  // kernel error word (bit 0: a bounded copy wait gave up)
    // RK4 time (Runge_kutta_O4::t_) and the phi history for extrapolated starts
    double t = 0., t_stage = 0.;
    double *phi_a = nullptr;
    double tau_a = 0., tau_b = 0.;
    int nhist = 0;
    AxisJob *dj = nullptr;
    ZJob *dz = nullptr;
    // job-list offsets (into dj / dz) and counts
    int jA_x = 0, jA_y = 0, zA = 0, jB_y = 0, jB_x = 0, jD_x = 0, jD_y = 0;
    int zD = 0, zF = 0, jF_y = 0, jT_x = 0, jT_y = 0, zT = 0, jTf_y = 0, jTf_x = 0;
    int jG_x = 0, jG_y = 0, zG = 0;
    // sine-stretched axes: the chain-rule right-hand side's buffers, metric
    // tables and job lists (allocated only when cfg.stretch_m != 0)
    bool stretched = false;
    void *SX[12] = {};
    void *met = nullptr;    // filtered 1/dS per index (bulk precision)
    double *vol = nullptr;  // dS per index (cell widths / h) for the diagnostics
    int jS_Dx = 0, jS_Dy = 0, zS_D = 0, zS_F = 0, jS_Fy = 0, jS_Gx = 0, jS_Gy = 0, zS_G = 0;
    // Jacobi state carried between solves (solver_poisson_jacobi_nlin.hpp:66-95)
    double norm_max = 0., norm_sum = 0.;
    JacState *d_js = nullptr, *h_js = nullptr;  // two on the device, taken in turn by the sweeps
    JcStat *jc_part[2] = {};
    std::vector<JacGraph> jac;
    kf_diag_out diag{};
    // kernel profiling (CUDA events around each launch, when enabled)
    bool prof = false;
    struct ProfRec { int cls; cudaEvent_t a, b; double bytes; };
    std::vector<ProfRec> recs;
    std::vector<cudaEvent_t> evfree;
    double prof_ms[32] = {}, prof_bytes[32] = {};
    long long prof_n[32] = {};
    std::vector<AxisJob> hj;
    std::vector<ZJob> hz;
    // the FAS V-cycle captured once as a CUDA graph (replayed every cycle)
    cudaGraphExec_t vgraph = nullptr;
    long long vgraph_kernels = 0;
    // an adaptive solve for the host-driven callers (fas_solve)
    long long host_solves = 0;  // adaptive FAS solves that the host drove
    cudaGraphExec_t solve_graph = nullptr;
    long long solve_kernels = 0, solve_cycle_kernels = 0;
    DevPois *h_pois = nullptr;
    // per-(precision, n) entry points
    void (*rhs_fn)(kf_ctx *) = nullptr;
    void (*r2c_fn)(kf_ctx *) = nullptr;
    void (*c2r_fn)(kf_ctx *) = nullptr;
    void (*inv_state_fn)(kf_ctx *) = nullptr;
    void (*adj_fn)(kf_ctx *, int) = nullptr;
    // discrete adjoint: buffers, job-list offsets, and the "phi given" switch
    // under which a right-hand side uses c->phi as it stands (no solve)
    AdjState *adj = nullptr;
    OutState *out = nullptr;
    bool phi_given = false;
    int fftv = 0;     // radix-plan variant of the transform kernels (kf_autotune)
    int rbgs_by = 8;  // smoother variant (kf_autotune): half-sweep block size, or 0 for k_rbgs_march
    bool march_maps = false;  // the driver's tensor-map encoder is available
    bool coarse_block = true;  // the coarse levels of a V-cycle in one k_cc cluster (kf_set_coarse_block)
    int cc_level = -1;         // entry level of k_cc, or -1 (cc_setup)
    int cc_ctas = 0;           // its cluster size
    ClusterCycle ccyc{};
    // window of rows (i, j) on which the penalization mask is not zero (RowBox), and
    // its size
    int *d_box = nullptr;
    int bx_i = 0, bx_j = 0;
    // what the end of the right-hand side does with K (k_xfwd_stage; 3: store it)
    int rk_mode = 3;
    double rk_c = 0.;
    double stage_x = 0.;  // its time minus the step's (captured step)
    int stage_idx = 0;  // RK stage of the right-hand side being evaluated (0..3)
    // one RK4 step captured as a CUDA graph (FAS or no Poisson, profile off):
    // time / warm-start history and solve statistics live on the device
    bool capturing = false;
    cudaStream_t st_body = nullptr;  // stream on which conditional bodies are captured
    // round D's transforms of u' and s, which do not depend on phi, run in a
    // captured step on st_side beside the Poisson solve (kf_set_overlap)
    bool overlap_d = true;
    cudaStream_t st_side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    DevTime *dtime = nullptr;
    DevPois *dpois = nullptr;
    DevPois hpois{};  // last values read back
    cudaGraphExec_t step_graph = nullptr;
    // the same step whose stage 1 waits for ev_u (the u' upload of kf_step_host)
    // after its Poisson solve, before the first use of u'
    cudaGraphExec_t step_graph_wait = nullptr;
    bool capture_wait_u = false;
    cudaStream_t st_copy = nullptr;
    cudaEvent_t ev_u = nullptr;
    double *stage64b = nullptr;  // FP32-bulk staging of the copy stream
    double step_dt = 0.;
    long long step_kernels = 0, cycle_kernels = 0;
    int jV_x = 0, jV_y = 0, zV = 0, zW = 0, nWz = 0, nWf = 0, jW_y = 0, jW_x = 0, zS = 0, jS_y = 0, jS_x = 0;
    int jP_x = 0, jP_y = 0, zP = 0, jQ_x = 0, jQ_y = 0, zQ = 0;
};

namespace {

// Host-side NVTX range (profiler timelines and ncu --nvtx filters): each RK4
// stage, each Poisson solve, each replay of a captured step.  Header-only NVTX:
// without a profiler attached the calls return at once.
struct NvtxRange {
    explicit NvtxRange(const char *s) { nvtxRangePushA(s); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

template <typename P> P *dalloc(kf_ctx *c, size_t bytes) {
    void *p = nullptr;
    CK(cudaMalloc(&p, bytes ? bytes : 16));
    c->allocs.push_back(p);
    return static_cast<P *>(p);
}

inline int nblk(long work, int bs) { return (int)((work + bs - 1) / bs); }

// Kernel classes for the profile (kf_profile_read); names in kf_profile_class_name.
enum KCls { KC_AXIS_INV, KC_AXIS_FWD, KC_Z_C2R, KC_Z_R2C, KC_XASM, KC_PROD, KC_LIN, KC_RHO, KC_RK,
            KC_JACOBI, KC_RBGS, KC_RESID, KC_TRANSFER, KC_COARSE, KC_REDUCE, KC_MISC, KC_ADJ_PW, KC_ADJ_MG,
            KC_MG_COARSE, KC_MARCH, KC_MARCH_RES,
            KC_N };
const char *const kKClsName[KC_N] = {"k_axis_pass(inverse)", "k_axis_pass(forward)", "k_z_c2r", "k_z_r2c",
                                     "k_xfwd_stage", "k_zprod/k_sl_products", "k_lin", "k_rho", "-", "k_jacobi",
                                     "k_rbgs", "k_residual", "k_restrict/k_fas_rhs/k_prolong/k_inject",
                                     "k_coarse_solve/k_cc", "-", "conversion/diagnostics",
                                     "adjoint pointwise (k_prod_vjp/k_vjp_assemble/k_adj_stage/...)",
                                     "adjoint Poisson (linear multigrid)",
                                     "FAS levels below the finest (k_rbgs/k_residual/transfers)",
                                     "k_rbgs_march(sweep)", "k_rbgs_march(sweep+residual)"};

void prof_flush(kf_ctx *c) {
    if (c->recs.empty()) return;
    CK(cudaStreamSynchronize(c->st));
    for (auto &r : c->recs) {
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, r.a, r.b));
        c->prof_ms[r.cls] += ms;
        c->prof_n[r.cls] += 1;
        c->prof_bytes[r.cls] += r.bytes;
        c->evfree.push_back(r.a);
        c->evfree.push_back(r.b);
    }
    c->recs.clear();
}

cudaEvent_t prof_event(kf_ctx *c) {
    if (c->evfree.empty()) {
        cudaEvent_t e;
        CK(cudaEventCreate(&e));
        return e;
    }
    cudaEvent_t e = c->evfree.back();
    c->evfree.pop_back();
    return e;
}

// One kernel launch: counts it and, when profiling, brackets it with events
// on the context's stream and records its algorithmic bytes.
struct Launch {
    kf_ctx *c;
    int cls;
    double bytes;
    cudaEvent_t a = nullptr;
    Launch(kf_ctx *c_, int cls_, double bytes_) : c(c_), cls(cls_), bytes(bytes_) {
        c->launches++;
        if (c->prof) {
            if (c->recs.size() > 16384) prof_flush(c);
            a = prof_event(c);
            CK(cudaEventRecord(a, c->st));
        }
    }
    ~Launch() noexcept(false) {
        if (c->prof) {
            cudaEvent_t b = prof_event(c);
            CK(cudaEventRecord(b, c->st));
            c->recs.push_back(kf_ctx::ProfRec{cls, a, b, bytes});
        }
    }
};

// Whether everything is launched kernel by kernel: for the per-launch profile, and
// with KIELFLOW_B200_NO_GRAPH=1, for tools that do not see into captured graphs.
bool host_driven(const kf_ctx *c) {
    static const bool off = [] {
        const char *e = std::getenv("KIELFLOW_B200_NO_GRAPH");
        return e && e[0] == '1';
    }();
    return c->prof || off;
}

// ------------------------------------------------------------------ host tables
double k_val_at(int i, int n, double L) {  // axis_EqSt.cpp:57-61
    double pi = acos(-1.);
    return ((i <= n / 2) ? (2. * pi * i / L) : (2. * pi * (i - n) / L));
}
// Position of index i (-1 <= i <= n) on the box axis [-L/2, L/2):
// axis_CoEqSt for m == 0 (axis_EqSt.cpp:52-55), else axis_CoSiSt with the
// periodic extension of its val_at (axis_SiSt.cpp:93-116) and
// S(x) = x - m sin(2 pi x / L) (:153-157).
double val_at(int i, int n, double L, double m = 0.) {
    if (m == 0.) return -0.5 * L + i * (L / n);
    int shift = 0;
    if (i < 0) {
        do {
            shift += 1;
        } while (i + shift * n < 0);
    }
    if (i >= n) {
        do {
            shift -= 1;
        } while (i + shift * n >= n - 1);
    }
    const double pi = acos(-1.);
    const double x = -0.5 * L + L * double(i + shift * n) / (n);
    return (x - m * sin(2. * pi * x / L)) - shift * L;
}
// dS/dx of the stretched axis at index i (axis_SiSt.cpp:158-164)
double dS_at(int i, int n, double L, double m) {
    const double pi = acos(-1.);
    const double x = -0.5 * L + (L / n) * i;
    return 1. - (2. * pi * m / L) * cos(2. * pi * x / L);
}
// 1/dS of each index after the 2/3 filter: OP_partial_derivative.cpp:60-80
// forms it on the whole grid (FFT, OP_dealiasing, inverse FFT); the field
// depends on one index only, so that is one 1-D DFT pair along the axis with
// the filter of the (k, 0, 0) line, done here in long double.
std::vector<double> metric_table(int n, double L, double m, double thr) {
    std::vector<double> f(n), q2(n), out(n);
    const double kmax = k_val_at(n / 2, n, L);
    for (int i = 0; i < n; ++i) {
        f[i] = 1. / dS_at(i, n, L, m);
        q2[i] = pow(k_val_at(i, n, L) / kmax, 2.);
    }
    const long double twopi = 6.283185307179586476925286766559005768L;
    std::vector<long double> acc(n, 0.L);
    for (int kk = 0; kk < n; ++kk) {
        if (!(q2[kk] + q2[0] + q2[0] < thr)) continue;
        long double Fr = 0.L, Fi = 0.L;
        for (int i = 0; i < n; ++i) {
            const long double a = twopi * (long double)((long)kk * i % n) / n;
            Fr += f[i] * cosl(a);
            Fi -= f[i] * sinl(a);
        }
        for (int i = 0; i < n; ++i) {
            const long double a = twopi * (long double)((long)kk * i % n) / n;
            acc[i] += Fr * cosl(a) - Fi * sinl(a);
        }
    }
    for (int i = 0; i < n; ++i) out[i] = (double)(acc[i] / n);
    return out;
}

// The 2/3 rule of OP_dealiasing.hpp:24-30 on one (j, kz) column of the x
// pass, (q2[i] + q2[j]) + q2[kz] < thr, as a bound b: keep(i) == (min(i, n - i)
// <= b).  The bound is the largest such m in [0, n/2] (-1: none), and the
// equivalence is checked on every i of the column with the same additions as
// the device; a column where it fails gets -2 (the kernels then test each
// element).
std::vector<int> dealias_bounds(const std::vector<double> &q2, int n, double thr) {
    const int nzc = n / 2 + 1;
    std::vector<int> pb((size_t)n * nzc);
    for (int j = 0; j < n; ++j)
        for (int k = 0; k < nzc; ++k) {
            int b = -1;
            for (int m = 0; m <= n / 2; ++m)
                if ((q2[m] + q2[j]) + q2[k] < thr) b = m;
            bool ok = true;
            for (int i = 0; i < n && ok; ++i) {
                const bool keep = (q2[i] + q2[j]) + q2[k] < thr;
                ok = keep == ((i <= n / 2 ? i : n - i) <= b);
            }
            pb[(size_t)j * nzc + k] = ok ? b : -2;
        }
    return pb;
}

// The kept part of a masked half spectrum from its x-pass bounds pb: nkz and
// jb[kz] such that the column (j, kz) has a kept element exactly when kz < nkz
// and min(j, n - j) <= jb[kz], and the x-pass tiles of tc columns that cover
// those columns.  (q2 grows with |frequency| and is the same for both signs, and
// rounded sums keep that order, so every column fits this form; a column that
// did not is an error.)
struct TruncTab {
    int nkz = 0;
    std::vector<int> jb, tl;
};
TruncTab trunc_table(const std::vector<int> &pb, int n, int tc) {
    const int nzc = n / 2 + 1;
    TruncTab t;
    std::vector<int> jb(nzc, -1);
    int nkz = 0;
    for (int k = 0; k < nzc; ++k) {
        for (int m = 0; m <= n / 2; ++m)
            if (pb[(size_t)m * nzc + k] >= 0) jb[k] = m;
        if (jb[k] >= 0) nkz = k + 1;
    }
    for (int j = 0; j < n; ++j)
        for (int k = 0; k < nzc; ++k) {
            const int b = pb[(size_t)j * nzc + k];
            if (b == -2 || (b >= 0) != ((j <= n / 2 ? j : n - j) <= jb[k]))
                throw KfError{KF_ERR_ARG, "the 2/3 rule has no index bounds on this grid"};
        }
    t.nkz = nkz;
    t.jb = jb;
    for (int j = 0; j < n; ++j) {
        int last = -1;
        for (int k = 0; k < nkz; ++k)
            if (pb[(size_t)j * nzc + k] >= 0) last = k;
        for (int k = 0; k <= last; k += tc) t.tl.push_back((j << 16) | k);
    }
    return t;
}

// ------------------------------------------------------------------ Poisson driver
int red_blocks(long N) {
    long nb = (N + RBS - 1) / RBS;
    return (int)(nb < 1184 ? nb : 1184);
}

// Levels on which the column form of the residual runs (whole warps along k,
// columns of COL_PI planes).  At 256^3 (one B200): 99.6 us against 155.9 us for
// k_residual<1, 1>; the column form of the half sweep measured slower (201-225
// us per sweep against 150 us: its per-thread chain of Newton steps is
// latency-bound), so the half sweep stays one point per thread.
constexpr int COL_PI = 16;
bool col_level(int n) { return n >= 64 && n % 64 == 0 && n % COL_PI == 0; }

// The kernel error word: queued for reading before a synchronisation
// (kerr_fetch) and checked after it (kerr_check, which clears it)
void kerr_fetch(kf_ctx *c) {
    CK(cudaMemcpyAsync(c->h_err, c->d_err, sizeof(int), cudaMemcpyDeviceToHost, c->st));
}
void kerr_check(kf_ctx *c) {
    if (*c->h_err) {
        *c->h_err = 0;
        CK(cudaMemsetAsync(c->d_err, 0, sizeof(int), c->st));
        throw KfError{KF_ERR_CUDA, "a shared-memory copy of the multigrid smoother did not land within its wait limit"};
    }
}

double max_residual(kf_ctx *c, const LevelBuf &L, const double *phi, const double *rho, bool fast) {
    const long N = (long)L.n * L.n * L.n;
    CK(cudaMemsetAsync(c->d_max, 0, 64 * sizeof(unsigned long long), c->st));
    {
        Launch L_(c, KC_RESID, 16. * N);
        dim3 g = mg_grid(L.n, L.n);
        g.z = L.n < 16 ? L.n : 16;  // each block strides over the i-planes
        if (fast && col_level(L.n))
            k_residual_col<8, COL_PI, true, false, false>
                <<<dim3(L.n / 64, L.n / 8, L.n / COL_PI), mg_block(), 0, c->st>>>(phi, rho, L.lev(), nullptr, c->d_max);
        else if (fast)
            k_resmax<true><<<g, mg_block(), 0, c->st>>>(phi, rho, L.lev(), c->d_max);
        else
            k_resmax<false><<<g, mg_block(), 0, c->st>>>(phi, rho, L.lev(), c->d_max);
    }
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(c->h_max, c->d_max, 64 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, c->st));
    kerr_fetch(c);
    CK(cudaStreamSynchronize(c->st));
    kerr_check(c);
    unsigned long long m = 0;
    for (int s = 0; s < 64; ++s) m = c->h_max[s] > m ? c->h_max[s] : m;
    double r;
    std::memcpy(&r, &m, sizeof(double));
    return r;
}

// Blocks of a sweep: every block reads all of them (k_jacobi), so as few as fill
// the chip; a thread takes several points from 64^3 on.
int jac_blocks(long N) { return (int)std::min<long>((N + 255) / 256, N >= (1 << 20) ? 592 : 296); }

// Sweep s of a run on level L (phi -> tmp for even s, back for odd).
void jacobi_sweep(kf_ctx *c, const LevelBuf &L, double *phi, double *tmp, const double *rho, const JacStop &S, int s) {
    const long N = (long)L.n * L.n * L.n;
    const int i = s & 1, o = i ^ 1;
    Launch L_(c, KC_JACOBI, 24. * N);
    k_jacobi<<<jac_blocks(N), 256, 0, c->st>>>(i ? tmp : phi, i ? phi : tmp, rho, L.lev(), S, c->jc_part[i],
                                              c->jc_part[o], c->d_js + i, c->d_js + o);
}
// The record of a run after an even number of sweeps brought up to date.
void jacobi_test(kf_ctx *c, const LevelBuf &L, const JacStop &S, int loop, cudaGraphConditionalHandle h) {
    const long N = (long)L.n * L.n * L.n;
    Launch L_(c, KC_JACOBI, 0.);
    k_jacobi_test<<<1, 256, 0, c->st>>>(c->jc_part[0], jac_blocks(N), c->d_js, N, S, loop, h);
}

// The captured sweep loop: WHILE { JC_UNROLL sweeps phi -> tmp -> phi ... }, then
// the result into phi.
cudaGraphExec_t jacobi_graph(kf_ctx *c, const LevelBuf &L, double *phi, double *tmp, const double *rho,
                             const JacStop &S) {
    for (const JacGraph &g : c->jac)
        if (g.phi == phi && g.tmp == tmp && g.rho == rho && g.stop.max_it == S.max_it &&
            g.stop.resstop == S.resstop && g.stop.limit == S.limit && g.stop.tol == S.tol)
            return g.exec;
    const long N = (long)L.n * L.n * L.n;
    const long long l0 = c->launches;
    cudaStream_t outer = c->st;
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(outer, cudaStreamCaptureModeThreadLocal));
    try {
        cudaStreamCaptureStatus cs;
        cudaGraph_t cg = nullptr;
        const cudaGraphNode_t *deps = nullptr;
        size_t ndeps = 0;
        CK(cudaStreamGetCaptureInfo(outer, &cs, nullptr, &cg, &deps, &ndeps));
        cudaGraphConditionalHandle h;
        CK(cudaGraphConditionalHandleCreate(&h, cg, 1, cudaGraphCondAssignDefault));
        cudaGraphNodeParams wp = {cudaGraphNodeTypeConditional};
        wp.conditional.handle = h;
        wp.conditional.type = cudaGraphCondTypeWhile;
        wp.conditional.size = 1;
        cudaGraphNode_t wnode;
        CK(cudaGraphAddNode(&wnode, cg, deps, ndeps, &wp));
        CK(cudaStreamUpdateCaptureDependencies(outer, &wnode, 1, cudaStreamSetCaptureDependencies));
        c->st = c->st_body;
        CK(cudaStreamBeginCaptureToGraph(c->st, wp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                         cudaStreamCaptureModeThreadLocal));
        cudaGraph_t body = nullptr;
        try {
            for (int s = 0; s < JC_UNROLL; ++s)
                jacobi_sweep(c, L, phi, tmp, rho, S, s);
            jacobi_test(c, L, S, 1, h);
        } catch (...) {
            cudaStreamEndCapture(c->st, &body);
            throw;
        }
        CK(cudaStreamEndCapture(c->st, &body));
        c->st = outer;
        Launch L_(c, KC_JACOBI, 0.);
        k_jacobi_out<<<nblk(N, 256), 256, 0, c->st>>>(phi, tmp, c->d_js, N);
    } catch (...) {
        c->st = outer;
        cudaStreamEndCapture(outer, &g);
        if (g) cudaGraphDestroy(g);
        c->launches = l0;
        throw;
    }
    CK(cudaStreamEndCapture(outer, &g));
    JacGraph J{phi, tmp, rho, S, nullptr};
    const cudaError_t e = cudaGraphInstantiate(&J.exec, g, 0);
    cudaGraphDestroy(g);
    CK(e);
    c->launches = l0;
    c->jac.push_back(J);
    return J.exec;
}

// solver_poisson_jacobi_nlin::solve (:50-108) on one level; phi, tmp: level-sized.
int jacobi_solve(kf_ctx *c, const LevelBuf &L, double *phi, double *tmp, const double *rho, int max_it,
                 double limit_max, bool resstop, double tol) {
    const long N = (long)L.n * L.n * L.n;
    const JacStop S{max_it < 0 ? 1000 : max_it, resstop, limit_max, tol};
    JacState &js = *c->h_js;
    js = JacState{};
    js.norm_max = c->norm_max;
    js.norm_sum = c->norm_sum;
    js.omega = 1.;
    if (S.max_it > 0) {
        cudaGraphExec_t exec = host_driven(c) ? nullptr : jacobi_graph(c, L, phi, tmp, rho, S);
        js.fresh = 1;
        CK(cudaMemcpyAsync(c->d_js, &js, sizeof(JacState), cudaMemcpyHostToDevice, c->st));
        if (exec) {
            CK(cudaGraphLaunch(exec, c->st));
        } else {  // launched one by one
            while (!js.done) {
                for (int s = 0; s < 2; ++s) jacobi_sweep(c, L, phi, tmp, rho, S, s);
                jacobi_test(c, L, S, 0, 0);
                CK(cudaGetLastError());
                CK(cudaMemcpyAsync(&js, c->d_js, sizeof(JacState), cudaMemcpyDeviceToHost, c->st));
                CK(cudaStreamSynchronize(c->st));
            }
            Launch L_(c, KC_JACOBI, 0.);
            k_jacobi_out<<<nblk(N, 256), 256, 0, c->st>>>(phi, tmp, c->d_js, N);
        }
        CK(cudaMemcpyAsync(&js, c->d_js, sizeof(JacState), cudaMemcpyDeviceToHost, c->st));
        CK(cudaStreamSynchronize(c->st));
        if (exec) c->launches += js.iteration + 1;
    }
    c->norm_max = js.norm_max;
    c->norm_sum = js.norm_sum;
    if (js.nan) throw KfError{KF_ERR_NAN, "NaN in the Jacobi sweep"};
    c->diag.last_iterations = js.iteration;
    c->diag.total_iterations += js.iteration;
    c->diag.last_residual = js.rlast;
    if (!js.converged) c->diag.not_converged++;
    return js.converged ? 0 : 1;
}

// over-relaxation factor of the FAS smoother's Newton step (0 selects 1)
double mg_omega(const kf_config &cf) { return cf.mg_omega > 0. ? cf.mg_omega : 1.; }

// ------------------------------------------------------- streaming smoother
// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library)
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiledFn)p;
    }();
    return fn;
}

// Tensor map of an n^3 FP64 level whose copies are single rows of MT_PITCH
// doubles (x = k fastest, then j, then i)
bool row_map(CUtensorMap *m, const double *base, int n) {
    const EncodeTiledFn f = encode_tiled();
    if (!f) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)n, (cuuint64_t)n};
    const cuuint64_t strides[2] = {(cuuint64_t)n * 8, (cuuint64_t)n * n * 8};
    const cuuint32_t box[3] = {MT_PITCH, 1, 1};
    const cuuint32_t es[3] = {1, 1, 1};
    return f(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, (void *)base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// planes per CTA of the streaming smoother: at least three waves of CTAs at
// 256^3 (128 tiles x 8 chunks), the ghost planes (2 H per chunk) small
int march_ci(int n) { return n >= 256 ? 32 : (n >= 128 ? 16 : 8); }
constexpr int MT_TJ = 8;

bool march_level(const LevelBuf &L) { return L.n >= MT_TK && L.n % MT_TK == 0 && L.n % MT_TJ == 0; }

bool march_ok(const kf_ctx *c, const LevelBuf &L) { return c->rbgs_by == 0 && c->march_maps && L.t && march_level(L); }

void march_attrs() {
    CK(cudaFuncSetAttribute(k_rbgs_march<MM_RES, MT_TJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)march_smem<MM_RES, MT_TJ>(32)));
    CK(cudaFuncSetAttribute(k_rbgs_march<MM_SWEEP, MT_TJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)march_smem<MM_SWEEP, MT_TJ>(32)));
    CK(cudaFuncSetAttribute(k_rbgs_march<MM_SWEEP_RES, MT_TJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)march_smem<MM_SWEEP_RES, MT_TJ>(32)));
}

// One streaming pass on level L: src -> dst (a whole red-black sweep) and/or
// the residual r of the result, max |r| into `slots` when given.
template <int MODE>
void march(kf_ctx *c, const LevelBuf &L, const double *src, const double *rho, double *dst, double *r,
           unsigned long long *slots, int cls) {
    const int n = L.n, ci = march_ci(n);
    CUtensorMap mp, mr;
    if (!row_map(&mp, src, n) || !row_map(&mr, rho, n))
        throw KfError{KF_ERR_CUDA, "cuTensorMapEncodeTiled refused a multigrid level"};
    MarchArgs a{dst, r, src, rho, L.dd, L.ip, L.im, slots, c->d_err, n, ci, n / MT_TK, mg_omega(c->cfg)};
    const dim3 g((n / MT_TK) * (n / MT_TJ), n / ci);
    const long N = (long)n * n * n;
    Launch L_(c, cls, (MODE == MM_SWEEP_RES ? 32. : 24.) * N);
    k_rbgs_march<MODE, MT_TJ><<<g, MT_THREADS, march_smem<MODE, MT_TJ>(ci), c->st>>>(mp, mr, a);
}

// `sweeps` red-black Gauss-Seidel sweeps on level L (phi in place), two
// half-sweep launches each.  cc: the adjoint's e^phi (linear point solve) or
// nullptr (Newton step).
void smooth_plain(kf_ctx *c, LevelBuf &L, double *phi, const double *rho, const double *cc, int sweeps, int cls);

void smooth(kf_ctx *c, LevelBuf &L, double *phi, const double *rho, const double *cc, int sweeps, int cls) {
    if (!cc && march_ok(c, L) && phi != L.t) {
        // streaming passes phi -> t -> phi; an odd sweep first in place
        if (sweeps & 1) smooth_plain(c, L, phi, rho, nullptr, 1, cls);
        const int mc = cls == KC_RBGS ? KC_MARCH : cls;
        for (int s = 0; s + 1 < sweeps; s += 2) {
            march<MM_SWEEP>(c, L, phi, rho, L.t, nullptr, nullptr, mc);
            march<MM_SWEEP>(c, L, L.t, rho, phi, nullptr, nullptr, mc);
        }
        return;
    }
    smooth_plain(c, L, phi, rho, cc, sweeps, cls);
}

// `sweeps` red-black sweeps as two half-sweep launches each (k_rbgs_t, or
// k_rbgs_lin_t with the adjoint's e^phi).  (Sweeping a level larger than L2 in
// chunks of i-planes, black one plane behind red so that the black half finds
// its data in L2, gives the same potentials bit for bit but measured slower at
// 256^3: 156 / 169 / 181 / 214 us per sweep for 1 / 2 / 4 / 8 chunks.  So did
// threads that update one (j, k) on 2 or 4 planes two apart, sharing the axis
// tables and the planes between their points: 20.4 / 20.2 ms against 18.9 ms
// for 240 half sweeps; L1 use fell from 89 to 62 %, but occupancy halved and
// the DRAM throughput, 4.5 TB/s on 1.33x the algorithmic bytes, stayed.)
void smooth_plain(kf_ctx *c, LevelBuf &L, double *phi, const double *rho, const double *cc, int sweeps, int cls) {
    const int n = L.n;
    const long N = (long)n * n * n;
    const int by = c->rbgs_by ? c->rbgs_by : 8;
    const double om = mg_omega(c->cfg);
    const dim3 g((n / 2 + 31) / 32, (n + by - 1) / by, n), b(32, by);
    for (int s = 0; s < sweeps; ++s)
        for (int color = 0; color < 2; ++color) {
            Launch L_(c, cls, 16. * N);
            if (cc) {
                if (by == 4)
                    k_rbgs_lin_t<4><<<g, b, 0, c->st>>>(phi, rho, cc, L.lev(), color, om, *L.tab);
                else if (by == 16)
                    k_rbgs_lin_t<16><<<g, b, 0, c->st>>>(phi, rho, cc, L.lev(), color, om, *L.tab);
                else
                    k_rbgs_lin_t<8><<<g, b, 0, c->st>>>(phi, rho, cc, L.lev(), color, om, *L.tab);
            } else {
                if (by == 4)
                    k_rbgs_t<4><<<g, b, 0, c->st>>>(phi, rho, L.lev(), color, om, *L.tab);
                else if (by == 16)
                    k_rbgs_t<16><<<g, b, 0, c->st>>>(phi, rho, L.lev(), color, om, *L.tab);
                else
                    k_rbgs_t<8><<<g, b, 0, c->st>>>(phi, rho, L.lev(), color, om, *L.tab);
            }
        }
}

// The coarse levels' cycle (k_cc) from the injected potential, its copy and the
// restricted residual of the entry level.  LIN: the adjoint's linear system with
// e^phi in cc, its coarsest relaxation tested every 4 sweeps and not over-relaxed
// (k_coarse_solve_lin).
template <bool LIN>
void coarse_cluster(kf_ctx *c, double *phi, double *phi0, const double *r, const std::vector<double *> *cc,
                    double rtol, int max_sweeps, int cls) {
    const kf_config &cf = c->cfg;
    ClusterCycle C = c->ccyc;
    if (LIN)
        for (int m = 0; m < C.nl; ++m) C.cc[m] = (*cc)[c->cc_level + m];
    const long N = (long)C.n[0] * C.n[0] * C.n[0];
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(c->cc_ctas);
    lc.blockDim = dim3(CC_THREADS);
    lc.dynamicSmemBytes = cc_smem(C, c->cc_ctas, LIN);
    lc.stream = c->st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = c->cc_ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    lc.attrs = &at;
    lc.numAttrs = 1;
    Launch L_(c, cls, 40. * N);
    CK(cudaLaunchKernelEx(&lc, k_cc<LIN>, phi, phi0, r, C, cf.mg_pre, cf.mg_post, LIN ? 0. : cf.coarse_tol, rtol,
                          max_sweeps, LIN ? 4 : 1, mg_omega(cf), LIN ? 1. : mg_omega(cf), c->d_sweeps));
}

// Whether level l's cycle runs in split order (not with the streaming smoother)
bool split_on(const kf_ctx *c, int l) { return c->lv[l].sp && c->rbgs_by != 0; }

// Blocks of the split-order kernels: 128 threads where the level lies in L2, 64
// where it streams from memory and both serve (split_pair); halved, at least a row,
// by rbgs_rows 4 and doubled, at most 128, by 16.
dim3 split_block(const kf_ctx *c, int n) {
    const int want = std::min(128, (n >= 256 ? 8 : 16) * c->rbgs_by), tx = n / 4;
    return dim3(tx, std::max(1, want / tx));
}

// `sweeps` red-black sweeps in split order
void smooth_split(kf_ctx *c, const LevelBuf &L, double *ph, const double *rh, int sweeps, int cls) {
    const int n = L.n;
    const dim3 b = split_block(c, n), g(1, (n + b.y - 1) / b.y, n);
    for (int s = 0; s < sweeps; ++s)
        for (int color = 0; color < 2; ++color) {
            Launch L_(c, cls, 16. * n * n * n);
            k_rbgs_s<<<g, b, 0, c->st>>>(ph, rh, L.slev(), color, mg_omega(c->cfg), *L.tab);
        }
}

// r = residual in split order, its max |r| into the d_max slots with_max
void residual_split(kf_ctx *c, const LevelBuf &L, bool with_max, int cls, bool slots_zero = false) {
    const int n = L.n;
    const int Z = with_max ? (n >= 128 ? 4 : 2) : (n >= 128 ? 2 : 1);
    const dim3 b = split_block(c, n), g(1, (n + b.y - 1) / b.y, 2 * n / Z);
    if (with_max && !slots_zero) CK(cudaMemsetAsync(c->d_max, 0, 64 * sizeof(unsigned long long), c->st));
    Launch L_(c, cls, 24. * n * n * n);
    if (with_max)
        k_residual_s<true><<<g, b, 0, c->st>>>(L.ph, L.rh, L.slev(), L.r, c->d_max, Z, *L.tab);
    else
        k_residual_s<false><<<g, b, 0, c->st>>>(L.ph, L.rh, L.slev(), L.r, nullptr, Z, *L.tab);
}

void vcycle(kf_ctx *c, int l);

// First part of a V-cycle on level l (not the coarsest): pre-smoothing and the
// residual L.r; with_max also leaves max |L.r| in the d_max slots (slots_zero:
// they are zero already).
void vcycle_head(kf_ctx *c, int l, bool with_max, bool slots_zero = false) {
    LevelBuf &L = c->lv[l];
    const kf_config &cf = c->cfg;
    const int n = L.n;
    const long N = (long)n * n * n;
    if (split_on(c, l)) {
        smooth_split(c, L, L.ph, L.rh, cf.mg_pre, l == 0 ? KC_RBGS : KC_MG_COARSE);
        residual_split(c, L, with_max, l == 0 ? KC_RESID : KC_MG_COARSE, slots_zero);
        return;
    }
    if (march_ok(c, L) && cf.mg_pre >= 1) {
        // the last pre-smoothing sweep fused with the residual (and its max):
        // the sweeps before it leave the potential in L.t
        int s = cf.mg_pre - 1;
        const int cls = l == 0 ? KC_MARCH : KC_MG_COARSE;
        if (s > 0 && s % 2 == 0) {
            smooth_plain(c, L, L.phi, L.rho, nullptr, 1, l == 0 ? KC_RBGS : KC_MG_COARSE);
            --s;
        }
        if (s == 0) {
            CK(cudaMemcpyAsync(L.t, L.phi, 8 * (size_t)N, cudaMemcpyDeviceToDevice, c->st));
        } else {
            march<MM_SWEEP>(c, L, L.phi, L.rho, L.t, nullptr, nullptr, cls);
            for (; s > 1; s -= 2) {
                march<MM_SWEEP>(c, L, L.t, L.rho, L.phi, nullptr, nullptr, cls);
                march<MM_SWEEP>(c, L, L.phi, L.rho, L.t, nullptr, nullptr, cls);
            }
        }
        if (with_max) CK(cudaMemsetAsync(c->d_max, 0, 64 * sizeof(unsigned long long), c->st));
        march<MM_SWEEP_RES>(c, L, L.t, L.rho, L.phi, L.r, with_max ? c->d_max : nullptr,
                            l == 0 ? KC_MARCH_RES : KC_MG_COARSE);
        return;
    }
    smooth(c, L, L.phi, L.rho, nullptr, cf.mg_pre, l == 0 ? KC_RBGS : KC_MG_COARSE);
    if (with_max) CK(cudaMemsetAsync(c->d_max, 0, 64 * sizeof(unsigned long long), c->st));
    Launch L_(c, l == 0 ? KC_RESID : KC_MG_COARSE, 24. * N);
    if (col_level(n)) {
        const dim3 gc(n / 64, n / 8, n / COL_PI);
        if (with_max)
            k_residual_col<8, COL_PI, true><<<gc, mg_block(), 0, c->st>>>(L.phi, L.rho, L.lev(), L.r, c->d_max);
        else
            k_residual_col<8, COL_PI, false><<<gc, mg_block(), 0, c->st>>>(L.phi, L.rho, L.lev(), L.r, nullptr);
    } else if (with_max) {
        dim3 g = mg_grid(n, n);
        g.z = n < 16 ? n : 16;  // each block strides over n/16 i-planes (ncu, 256^3: 158 us; 64 groups 169 us)
        k_residual<true, true><<<g, mg_block(), 0, c->st>>>(L.phi, L.rho, L.lev(), L.r, c->d_max);
    } else {
        k_residual<true><<<mg_grid(n, n), mg_block(), 0, c->st>>>(L.phi, L.rho, L.lev(), L.r);
    }
}

// The rest of the V-cycle on level l: restriction, the coarse cycle, the
// correction and post-smoothing.
void vcycle_tail(kf_ctx *c, int l) {
    LevelBuf &L = c->lv[l];
    const kf_config &cf = c->cfg;
    const int n = L.n;
    const long N = (long)n * n * n;
    LevelBuf &Lc = c->lv[l + 1];
    const long Nc3 = (long)Lc.n * Lc.n * Lc.n;
    if (split_on(c, l)) {
        const int cls = l == 0 ? KC_TRANSFER : KC_MG_COARSE;
        const bool cs = split_on(c, l + 1), cl = l + 1 == c->cc_level;
        const dim3 g = mg_grid(Lc.n, Lc.n);
        {
            Launch L_(c, cls, 8. * N + 24. * Nc3);
            if (cl)
                k_restrict_s<false, false><<<g, mg_block(), 0, c->st>>>(L.r, L.ph, n, Lc.lev(), Lc.r, Lc.phi, Lc.phi0);
            else if (cs)
                k_restrict_s<true, true><<<g, mg_block(), 0, c->st>>>(L.r, L.ph, n, Lc.lev(), Lc.rho, Lc.phi, Lc.phi0);
            else
                k_restrict_s<false, true><<<g, mg_block(), 0, c->st>>>(L.r, L.ph, n, Lc.lev(), Lc.rho, Lc.phi, Lc.phi0);
        }
        if (cl)
            coarse_cluster<false>(c, Lc.phi, Lc.phi0, Lc.r, nullptr, 1e-4, 1000, KC_COARSE);
        else
            vcycle(c, l + 1);
        {
            Launch L_(c, cls, 16. * N + (cl ? 8. : 16.) * Nc3);
            if (cl)
                k_prolong_s<false, true><<<g, mg_block(), 0, c->st>>>(L.ph, Lc.phi, Lc.phi0, L.gam, n);
            else if (cs)
                k_prolong_s<true, false><<<g, mg_block(), 0, c->st>>>(L.ph, Lc.phi, Lc.phi0, L.gam, n);
            else
                k_prolong_s<false, false><<<g, mg_block(), 0, c->st>>>(L.ph, Lc.phi, Lc.phi0, L.gam, n);
        }
        smooth_split(c, L, L.ph, L.rh, cf.mg_post, l == 0 ? KC_RBGS : KC_MG_COARSE);
        CK(cudaGetLastError());
        return;
    }
    {
        Launch L_(c, l == 0 ? KC_TRANSFER : KC_MG_COARSE, 8. * N + 32. * Nc3);
        k_restrict<<<mg_grid(Lc.n, Lc.n), mg_block(), 0, c->st>>>(L.r, L.phi, n, Lc.r, Lc.phi, Lc.phi0);
    }
    if (l + 1 == c->cc_level) {
        // the levels from l + 1 down: FAS right-hand side, cycle, correction
        coarse_cluster<false>(c, Lc.phi, Lc.phi0, Lc.r, nullptr, 1e-4, 1000, KC_COARSE);
    } else {
        {
            Launch L_(c, l == 0 ? KC_TRANSFER : KC_MG_COARSE, 24. * Nc3);
            k_fas_rhs<<<mg_grid(Lc.n, Lc.n), mg_block(), 0, c->st>>>(Lc.phi, Lc.r, Lc.lev(), Lc.rho);
        }
        vcycle(c, l + 1);
        {
            Launch L_(c, l == 0 ? KC_TRANSFER : KC_MG_COARSE, 24. * Nc3);
            k_correction<<<mg_grid(Lc.n, Lc.n), mg_block(), 0, c->st>>>(Lc.phi, Lc.phi0, Lc.n);
        }
    }
    {
        Launch L_(c, l == 0 ? KC_TRANSFER : KC_MG_COARSE, 16. * N + 8. * Nc3);
        k_prolong_add<<<mg_grid(Lc.n, Lc.n), mg_block(), 0, c->st>>>(L.phi, Lc.phi0, nullptr, L.gam, n);
    }
    smooth(c, L, L.phi, L.rho, nullptr, cf.mg_post, l == 0 ? KC_RBGS : KC_MG_COARSE);
    CK(cudaGetLastError());
}

void vcycle(kf_ctx *c, int l) {
    LevelBuf &L = c->lv[l];
    const kf_config &cf = c->cfg;
    const int n = L.n;
    const long N = (long)n * n * n;
    if (l == (int)c->lv.size() - 1) {
        Launch L_(c, KC_COARSE, 16. * N);
        const int bs = N >= 1024 ? 1024 : (int)((N + 31) / 32 * 32);
        k_coarse_solve<<<1, bs, (size_t)(16 * N + 24 * n), c->st>>>(L.phi, L.rho, L.lev(), cf.coarse_tol, 1000,
                                                                   c->d_sweeps, mg_omega(cf));
        return;
    }
    vcycle_head(c, l, false);
    vcycle_tail(c, l);
}

// One FAS V-cycle on the finest level: replayed from a CUDA graph captured on
// first use (one launch instead of ~70), or launched kernel by kernel
// (host_driven).
void run_vcycle(kf_ctx *c) {
    if (host_driven(c)) {
        vcycle(c, 0);
        return;
    }
    if (!c->vgraph) {
        const long long l0 = c->launches;
        CK(cudaStreamBeginCapture(c->st, cudaStreamCaptureModeThreadLocal));
        vcycle(c, 0);
        cudaGraph_t g = nullptr;
        CK(cudaStreamEndCapture(c->st, &g));
        cudaError_t e = cudaGraphInstantiate(&c->vgraph, g, 0);
        cudaGraphDestroy(g);
        CK(e);
        c->vgraph_kernels = c->launches - l0;
        c->launches = l0;
    }
    CK(cudaGraphLaunch(c->vgraph, c->st));
    c->launches += c->vgraph_kernels;
}

// max over the 64 d_max slots (IEEE bit patterns of non-negative doubles)
double read_max_slots(kf_ctx *c) {
    CK(cudaMemcpyAsync(c->h_max, c->d_max, 64 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, c->st));
    kerr_fetch(c);
    CK(cudaStreamSynchronize(c->st));
    kerr_check(c);
    unsigned long long m = 0;
    for (int s = 0; s < 64; ++s) m = c->h_max[s] > m ? c->h_max[s] : m;
    double r;
    std::memcpy(&r, &m, sizeof(double));
    return r;
}

// The finest level in and out of split order around a solve.  rho: unless the
// pass that wrote c->rho (k_z_rho) wrote its split copy as well.
void split_field(kf_ctx *c, const double *x, double *s) {
    Launch L_(c, KC_RHO, 16. * c->N);
    k_split<<<mg_grid(c->n / 2, c->n), mg_block(), 0, c->st>>>(x, s, c->n);
    CK(cudaGetLastError());
}
void solve_begin(kf_ctx *c, bool rho_done) {
    if (!split_on(c, 0)) return;
    if (!rho_done) split_field(c, c->rho, c->rho_cs);
    split_field(c, c->phi, c->phi_cs);
}
void unsplit_field(kf_ctx *c, const double *s, double *x) {
    Launch L_(c, KC_RHO, 16. * c->N);
    k_unsplit<<<mg_grid(c->n / 2, c->n), mg_block(), 0, c->st>>>(s, x, c->n);
    CK(cudaGetLastError());
}
void solve_end(kf_ctx *c) {
    if (split_on(c, 0)) unsplit_field(c, c->phi_cs, c->phi);
}

// The adaptive FAS loop inside a capture on c->st: head of the cycle
// (pre-smoothing, residual with its max); k_fas_check; WHILE { rest of the cycle;
// head; k_fas_check }: as many passes as V-cycles.  (WHILE { head; check; IF { rest
// } } took one pass more and an IF node in each; a pass costs about 7 us beside its
// kernels.)  Returns the kernels of a pass.
long long fas_loop(kf_ctx *c) {
    const kf_config &cf = c->cfg;
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    CK(cudaStreamGetCaptureInfo(c->st, &cs, nullptr, &g, nullptr, nullptr));
    cudaGraphConditionalHandle hw;
    CK(cudaGraphConditionalHandleCreate(&hw, g, 0, 0));
    auto head = [&](int first) {
        vcycle_head(c, 0, true, !first);  // k_fas_check leaves the slots zero
        Launch L_(c, KC_MISC, 0.);
        k_fas_check<<<1, 32, 0, c->st>>>(c->d_max, c->dpois, cf.res_tol, cf.max_cycles, first, false, c->stage_idx, hw);
    };
    head(1);
    const cudaGraphNode_t *deps = nullptr;
    size_t ndeps = 0;
    CK(cudaStreamGetCaptureInfo(c->st, &cs, nullptr, &g, &deps, &ndeps));
    cudaGraphNodeParams wp = {cudaGraphNodeTypeConditional};
    wp.conditional.handle = hw;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    cudaGraphNode_t wnode;
    CK(cudaGraphAddNode(&wnode, g, deps, ndeps, &wp));
    CK(cudaStreamUpdateCaptureDependencies(c->st, &wnode, 1, cudaStreamSetCaptureDependencies));
    const long long l1 = c->launches;
    cudaStream_t outer = c->st;
    c->st = c->st_body;
    cudaError_t e = cudaStreamBeginCaptureToGraph(c->st, wp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                  cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        cudaGraph_t body_out = nullptr;
        try {
            vcycle_tail(c, 0);
            head(0);
            e = cudaStreamEndCapture(c->st, &body_out);
        } catch (...) {
            cudaStreamEndCapture(c->st, &body_out);
            c->st = outer;
            throw;
        }
    }
    c->st = outer;
    CK(e);
    return c->launches - l1;
}

// A whole adaptive solve of the finest level from its own graph (fas_loop and the
// way back from split order), for the host-driven callers: one launch and one
// synchronisation.  Returns as poisson().
int fas_solve(kf_ctx *c) {
    const long long l0 = c->launches;
    if (!c->solve_graph) {
        CK(cudaStreamBeginCapture(c->st, cudaStreamCaptureModeThreadLocal));
        cudaGraph_t g = nullptr;
        try {
            c->solve_cycle_kernels = fas_loop(c);
            solve_end(c);
        } catch (...) {
            cudaStreamEndCapture(c->st, &g);
            if (g) cudaGraphDestroy(g);
            c->launches = l0;
            throw;
        }
        CK(cudaStreamEndCapture(c->st, &g));
        const cudaError_t e = cudaGraphInstantiate(&c->solve_graph, g, 0);
        cudaGraphDestroy(g);
        CK(e);
        c->solve_kernels = c->launches - l0 - c->solve_cycle_kernels;
        c->launches = l0;
    }
    CK(cudaGraphLaunch(c->solve_graph, c->st));
    CK(cudaMemcpyAsync(c->h_pois, c->dpois, sizeof(DevPois), cudaMemcpyDeviceToHost, c->st));
    kerr_fetch(c);
    CK(cudaStreamSynchronize(c->st));
    kerr_check(c);
    const DevPois &hp = *c->h_pois;
    const int cyc = hp.last_cycles;
    const bool nc = hp.not_converged != c->hpois.not_converged;
    c->hpois = hp;
    c->launches += c->solve_kernels + cyc * c->solve_cycle_kernels;
    c->diag.last_iterations = cyc;
    c->diag.stage_cycles[c->stage_idx & 3] += cyc;
    c->diag.total_iterations += cyc;
    c->diag.last_residual = hp.last_residual;
    if (hp.last_residual != hp.last_residual) throw KfError{KF_ERR_NAN, "NaN in the multigrid solve"};
    if (nc) c->diag.not_converged++;
    return nc ? 1 : 0;
}

// Poisson solve on c->phi with source c->rho; split: whoever wrote c->rho wrote
// its colour-split copy too.  Returns KF_OK or KF_ERR_NOT_CONVERGED.
int poisson(kf_ctx *c, bool split = false) {
    NvtxRange nv("kf Poisson solve");
    const kf_config &cf = c->cfg;
    c->diag.solves++;
    LevelBuf &L0 = c->lv[0];
    int rc = 0;
    if (cf.poisson_mode == KF_PS_JACOBI_REF || cf.poisson_mode == KF_PS_JACOBI_RES) {
        rc = jacobi_solve(c, L0, c->phi, L0.r, c->rho, cf.nlj_max_it, cf.nlj_limit,
                          cf.poisson_mode == KF_PS_JACOBI_RES, cf.res_tol);
        if (cf.poisson_mode == KF_PS_JACOBI_REF) {
            c->diag.last_residual = max_residual(c, L0, c->phi, c->rho, false);
            rc = 0;  // the reference's plan has no failure on a sweep cap
        }
    } else if (cf.poisson_mode == KF_PS_CASCADIC) {
        // kielflow.cpp:207-217 through solver_poisson_multigrid.cpp:246-418
        const int steps[4] = {0, -1, -1, -1};
        const double tol[4] = {0.01, 0.0005, 0.0001, 0.0001};
        const int n = c->n;
        LevelBuf &L3 = c->lv[3];
        {
            Launch L_(c, KC_TRANSFER, 16. * L3.n * L3.n * L3.n);
            k_inject<<<mg_grid(L3.n, L3.n), mg_block(), 0, c->st>>>(c->phi, n, 8, L3.phi);
        }
        for (int cas = 0; cas < 4; ++cas) {
            const int l = 3 - cas;
            LevelBuf &L = c->lv[l];
            const long Nl = (long)L.n * L.n * L.n;
            if (cas > 0) {
                double *dst = l == 0 ? c->phi : L.phi;
                Launch L_(c, KC_TRANSFER, 9. * Nl);
                k_prolong_set<<<mg_grid(L.n, L.n), mg_block(), 0, c->st>>>(dst, c->lv[l + 1].phi, L.gam, L.n);
            }
            const double *rho_l = c->rho;
            if (l > 0) {
                {
                    Launch L_(c, KC_TRANSFER, 16. * Nl);
                    k_inject<<<mg_grid(L.n, L.n), mg_block(), 0, c->st>>>(c->rho, n, n / L.n, L.rho);
                }
                rho_l = L.rho;
            }
            double *phi_l = l == 0 ? c->phi : L.phi;
            jacobi_solve(c, L, phi_l, L.r, rho_l, steps[cas], tol[cas], false, 0.);
        }
        c->diag.last_residual = max_residual(c, L0, c->phi, c->rho, false);
        rc = 0;
    } else if (!(cf.res_tol > 0.)) {
        // fixed number of V-cycles: the result is a smooth function of rho
        // and of the initial guess (no data-dependent stopping)
        solve_begin(c, split);
        for (int cyc = 0; cyc < cf.max_cycles; ++cyc) run_vcycle(c);
        solve_end(c);
        const double r = max_residual(c, L0, c->phi, c->rho, true);
        c->diag.last_iterations = cf.max_cycles;
        c->diag.total_iterations += cf.max_cycles;
        c->diag.stage_cycles[c->stage_idx & 3] += cf.max_cycles;
        c->diag.last_residual = r;
        if (r != r) throw KfError{KF_ERR_NAN, "NaN in the multigrid solve"};
    } else if (c->lv.size() > 1) {
        // test after each cycle's pre-smoothing on the residual the cycle
        // computes anyway; the rest of the cycle only when it fails
        solve_begin(c, split);
        // a context's first solve from here: making the graph takes as long as the
        // launches and synchronisations that it saves in a few solves
        if (!host_driven(c) && c->host_solves++) return fas_solve(c);
        double r = 0.;
        int cyc = 0;
        for (;;) {
            vcycle_head(c, 0, true);
            CK(cudaGetLastError());
            r = read_max_slots(c);
            if (!(r > cf.res_tol) || cyc >= cf.max_cycles) break;
            vcycle_tail(c, 0);
            ++cyc;
        }
        solve_end(c);
        c->diag.last_iterations = cyc;
        c->diag.stage_cycles[c->stage_idx & 3] += cyc;
        c->diag.total_iterations += cyc;
        c->diag.last_residual = r;
        if (r != r) throw KfError{KF_ERR_NAN, "NaN in the multigrid solve"};
        if (r > cf.res_tol) {
            c->diag.not_converged++;
            rc = 1;
        }
    } else {
        solve_begin(c, split);
        double r = max_residual(c, L0, c->phi, c->rho, true);
        int cyc = 0;
        while (r > cf.res_tol && cyc < cf.max_cycles) {
            run_vcycle(c);
            ++cyc;
            r = max_residual(c, L0, c->phi, c->rho, true);
        }
        c->diag.last_iterations = cyc;
        c->diag.stage_cycles[c->stage_idx & 3] += cyc;
        c->diag.total_iterations += cyc;
        c->diag.last_residual = r;
        if (r != r) throw KfError{KF_ERR_NAN, "NaN in the multigrid solve"};
        if (r > cf.res_tol) {
            c->diag.not_converged++;
            rc = 1;
        }
    }
    if (c->diag.last_residual != c->diag.last_residual) throw KfError{KF_ERR_NAN, "NaN in phi"};
    return rc;
}

// Start of a solve at time t_stage: linear extrapolation of the last two
// solutions at distinct times (returns whether t_stage is a new time).
bool phi_guess(kf_ctx *c) {
    const double t = c->t_stage;
    const bool newtime = c->nhist == 0 || t != c->tau_b;
    if (!c->cfg.phi_extrap || !newtime || c->nhist == 0) return newtime;
    if (c->nhist >= 2) {
        const double w = (t - c->tau_b) / (c->tau_b - c->tau_a);
        Launch L_(c, KC_MISC, 24. * c->N);
        k_extrap<<<nblk(c->N, 256), 256, 0, c->st>>>(c->phi, c->phi_a, w, c->N);
    } else {
        CK(cudaMemcpyAsync(c->phi_a, c->phi, 8 * c->N, cudaMemcpyDeviceToDevice, c->st));
    }
    c->tau_a = c->tau_b;
    return newtime;
}

// Whether the right-hand side being formed solves by poisson_captured.
bool captured_solve(const kf_ctx *c) {
    return c->capturing && !c->phi_given && (c->cfg.terms & T_POISSON) && (c->cfg.terms & T_E_INT);
}

// The stage's Poisson solve inside the capture of a step graph: device-side
// warm start, then the FAS loop as a conditional WHILE node whose body (one
// V-cycle + the max-residual test) is captured on st_body.  On split levels phi
// stays in split order from the first stage's start to the last stage's end: the
// next stage's start and phi^ read it there.
void poisson_captured(kf_ctx *c) {
    const kf_config &cf = c->cfg;
    const bool extrap = cf.phi_extrap != 0;
    const bool sp = split_on(c, 0);
    if (extrap && sp) {
        Launch L_(c, KC_MISC, 32. * c->N);
        k_guess_s<<<mg_grid(c->n / 2, c->n), mg_block(), 0, c->st>>>(c->stage_idx ? nullptr : c->phi, c->phi_a,
                                                                     c->phi_cs, c->dtime, c->stage_x, c->n);
    } else if (extrap) {
        Launch L_(c, KC_MISC, 24. * c->N);
        k_guess<<<nblk(c->N, 256), 256, 0, c->st>>>(c->phi, c->phi_a, c->dtime, c->stage_x, c->N);
    } else if (sp && c->stage_idx == 0) {
        split_field(c, c->phi, c->phi_cs);
    }
    LevelBuf &L0 = c->lv[0];
    const bool fixed = !(cf.res_tol > 0.);
    if (!fixed && c->lv.size() > 1) {
        c->cycle_kernels = fas_loop(c);
        if (c->stage_idx == 3) solve_end(c);
        if (extrap) {
            Launch L_(c, KC_MISC, 0.);
            k_hist_post<<<1, 32, 0, c->st>>>(c->dtime, c->stage_x);
        }
        CK(cudaGetLastError());
        return;
    }
    auto resmax = [&](cudaStream_t st) {
        if (sp) {
            residual_split(c, L0, true, KC_RESID);
            return;
        }
        CK(cudaMemsetAsync(c->d_max, 0, 64 * sizeof(unsigned long long), st));
        Launch L_(c, KC_RESID, 16. * c->N);
        dim3 g = mg_grid(L0.n, L0.n);
        g.z = L0.n < 16 ? L0.n : 16;
        if (col_level(L0.n))
            k_residual_col<8, COL_PI, true, false, false>
                <<<dim3(L0.n / 64, L0.n / 8, L0.n / COL_PI), mg_block(), 0, st>>>(c->phi, c->rho, L0.lev(), nullptr,
                                                                                  c->d_max);
        else
            k_resmax<true><<<g, mg_block(), 0, st>>>(c->phi, c->rho, L0.lev(), c->d_max);
    };
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    CK(cudaStreamGetCaptureInfo(c->st, &cs, nullptr, &g, nullptr, nullptr));
    cudaGraphConditionalHandle h;
    CK(cudaGraphConditionalHandleCreate(&h, g, 0, 0));
    resmax(c->st);
    {
        Launch L_(c, KC_MISC, 0.);
        k_fas_check<<<1, 32, 0, c->st>>>(c->d_max, c->dpois, cf.res_tol, cf.max_cycles, 1, fixed, c->stage_idx, h);
    }
    const cudaGraphNode_t *deps = nullptr;
    size_t ndeps = 0;
    CK(cudaStreamGetCaptureInfo(c->st, &cs, nullptr, &g, &deps, &ndeps));
    cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    CK(cudaGraphAddNode(&node, g, deps, ndeps, &cp));
    CK(cudaStreamUpdateCaptureDependencies(c->st, &node, 1, cudaStreamSetCaptureDependencies));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    const long long l0 = c->launches;
    cudaStream_t outer = c->st;
    c->st = c->st_body;
    CK(cudaStreamBeginCaptureToGraph(c->st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    vcycle(c, 0);
    resmax(c->st);
    {
        Launch L_(c, KC_MISC, 0.);
        k_fas_check<<<1, 32, 0, c->st>>>(c->d_max, c->dpois, cf.res_tol, cf.max_cycles, 0, fixed, c->stage_idx, h);
    }
    cudaGraph_t body_out = nullptr;
    cudaError_t e = cudaStreamEndCapture(c->st, &body_out);
    c->st = outer;
    CK(e);
    c->cycle_kernels = c->launches - l0;
    if (c->stage_idx == 3) solve_end(c);
    if (extrap) {
        Launch L_(c, KC_MISC, 0.);
        k_hist_post<<<1, 32, 0, c->st>>>(c->dtime, c->stage_x);
    }
    CK(cudaGetLastError());
}

// ------------------------------------------------------------------ per-(T, N) implementation
template <typename T, int N> struct Impl {
    typedef typename C2<T>::type T2;
    static constexpr int TC = Tile<T>::TC, LZ = ZTile<T>::LZ, NZC = N / 2 + 1;
    template <int V> static constexpr int PV = PlanV<N, V>::P;
    // with penalization the linear terms go through physical space whole (k_zprod):
    // 256^3 FP32 bulk 14.2 ms a step against 13.1 with them in k-space
    static constexpr bool RLINES = sizeof(T) == 4;

    static const T2 *tw(kf_ctx *c) { return (const T2 *)c->tw[c->fftv]; }

    static Geo<T> geo(kf_ctx *c) {
        return Geo<T>{c->n, c->nzc, (const T *)c->kv, c->q2, dealias_threshold(), c->pb};
    }

    static void set_attrs() {
        static bool done = false;
        if (done) return;
        const int big = 200 * 1024;
        CK(cudaFuncSetAttribute(k_axis_pass<T, N, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_axis_pass<T, N, +1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        set_attrs_v<0>(big);
        set_attrs_v<1>(big);
        done = true;
    }

    template <int V> static void set_attrs_v(int big) {
        CK(cudaFuncSetAttribute(k_axis_pipe<T, N, -1, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_axis_pipe<T, N, +1, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_z_c2r<T, N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_z_r2c<T, N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_zprod<T, N, V, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        if constexpr (RLINES)
            CK(cudaFuncSetAttribute(k_zprod<T, N, V, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_z_rho<T, N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_z_phi<T, N, V, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_z_phi<T, N, V, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_xfwd_stage<T, N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
        CK(cudaFuncSetAttribute(k_x_filter<T, N, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    }

    // distinct inputs and outputs of a launch, each as far as the mode moves it
    static double job_bytes(kf_ctx *c, int off, int njobs, int mode, const kf_ctx::Cols &t) {
        std::vector<const void *> u;
        for (int j = 0; j < njobs; ++j) {
            const void *p = c->hj[off + j].in;
            bool seen = false;
            for (auto q : u) seen |= q == p;
            if (!seen) u.push_back(p);
        }
        double fin = (double)c->Nc, fout = fin;
        if (mode == AX_XM) fin = c->tr_ball, fout = t.cols;
        if (mode == AX_YI) fin = t.cols, fout = (double)N * N * t.nkz;
        if (mode == AX_XB) fout = (double)c->bx_i * N * NZC;
        if (mode == AX_YB) fin = (double)c->bx_i * N * NZC, fout = (double)c->bx_i * c->bx_j * NZC;
        if (mode == AX_XF) fin = fout = t.cols;
        if (mode == AX_YF) fin = (double)N * N * t.nkz, fout = t.cols;
        return (u.size() * fin + njobs * fout) * sizeof(T2);
    }
    // resident blocks per SM x SMs of the pipelined pass (its grid)
    template <int V> static int pipe_grid(int sign) {
        static int g[2] = {0, 0};
        int &v = g[sign > 0];
        if (!v) {
            int dev = 0, sms = 0, per = 0;
            CK(cudaGetDevice(&dev));
            CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            const size_t smem = axis_pipe_smem<T, N>(32);
            if (sign < 0)
                CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_axis_pipe<T, N, -1, V>, TC * PV<V>, smem));
            else
                CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_axis_pipe<T, N, +1, V>, TC * PV<V>, smem));
            v = (per > 0 ? per : 1) * sms;
        }
        return v;
    }
    // inv: an inverse x pass reads a state field, the forward one a masked intermediate
    static AxTrunc trunc(kf_ctx *c, int mode, bool inv = true, const kf_ctx::Cols *cols = nullptr) {
        const kf_ctx::Cols &t = cols ? *cols : c->tr;
        AxTrunc A{AX_FULL, NZC, 0.f, nullptr, nullptr, nullptr, NZC, NZC};
        if (mode == AX_XB || mode == AX_YB) {
            A.mode = mode;
            A.win = c->d_box;
            return A;
        }
        if (mode == AX_FULL) return A;
        A.mode = mode;
        A.nkz = t.nkz;
        A.itpp = 1.f / (float)((t.nkz + TC - 1) / TC);
        A.jb = t.jb;
        A.tl = t.tl;
        A.ip = mode == AX_XM && inv ? NZC : t.mp;
        A.op = mode == AX_XF ? NZC : t.mp;
        return A;
    }
    // kz extent of a z pass over masked fields
    static int nkz(kf_ctx *c, bool masked) { return masked ? c->tr.nkz : NZC; }
    template <int V>
    static void axis_v(kf_ctx *c, int off, int njobs, int ax, int sign, int mode, const kf_ctx::Cols *cols) {
        const AxTrunc A = trunc(c, mode, true, cols);
        const int ntiles = A.mode == AX_XM || A.mode == AX_XF ? (cols ? cols->nt : c->tr.nt)
                           : ax == 0       ? (N * NZC + TC - 1) / TC
                                           : N * ((A.nkz + TC - 1) / TC);
        const int total = njobs * ntiles, grid = std::min(total, pipe_grid<V>(sign));
        const size_t smem = axis_pipe_smem<T, N>(njobs);
        if (sign < 0)
            k_axis_pipe<T, N, -1, V><<<grid, TC * PV<V>, smem, c->st>>>(c->dj + off, njobs, ax, geo(c),
                                                                      tw(c), total, A);
        else
            k_axis_pipe<T, N, +1, V><<<grid, TC * PV<V>, smem, c->st>>>(c->dj + off, njobs, ax, geo(c),
                                                                      tw(c), total, A);
    }
    // cols: the active columns of a truncated mode (nullptr: the 2/3 rule's)
    static void axis(kf_ctx *c, int off, int njobs, int ax, int sign, int mode = AX_FULL,
                     const kf_ctx::Cols *cols = nullptr) {
        Launch L_(c, sign > 0 ? KC_AXIS_INV : KC_AXIS_FWD, job_bytes(c, off, njobs, mode, cols ? *cols : c->tr));
        if (c->fftv)
            axis_v<1>(c, off, njobs, ax, sign, mode, cols);
        else
            axis_v<0>(c, off, njobs, ax, sign, mode, cols);
    }
    static double z_bytes(kf_ctx *c, int off, int njobs, bool c2r, bool masked, int nrows = N * N) {
        std::vector<const void *> u;
        int outs = 0;
        for (int j = 0; j < njobs; ++j) {
            const ZJob &z = c->hz[off + j];
            for (const void *p : {z.inA, z.inB}) {
                if (!p) continue;
                bool seen = false;
                for (auto q : u) seen |= q == p;
                if (!seen) u.push_back(p);
            }
            outs += (z.outA ? 1 : 0) + (z.outB ? 1 : 0);
        }
        const double cb = (double)nrows * nkz(c, masked) * sizeof(T2), rb = (double)nrows * N * sizeof(T);
        return c2r ? u.size() * cb + outs * rb : u.size() * rb + outs * cb;
    }
    // scale < 0: the 1/N of c2r; otherwise the given factor (1 for transposes)
    // masked: the half spectra come from masked x / y passes (zero from kz = nkz on)
    // window: rows of the mask's window, packed
    static void zc2r(kf_ctx *c, int off, int njobs, bool masked = false, double scale = -1., bool window = false) {
        const int nrows = N * N, ntiles = (nrows + LZ - 1) / LZ;
        const int *win = window ? c->d_box : nullptr;
        const size_t smem = ZSmem<T, N, true>::bytes;
        Launch L_(c, KC_Z_C2R, z_bytes(c, off, njobs, true, masked, window ? c->bx_i * c->bx_j : nrows));
        const T sc = (T)(scale < 0. ? 1. / ((double)N * N * N) : scale);
        if (c->fftv)
            k_z_c2r<T, N, 1><<<njobs * ntiles, LZ * PV<1>, smem, c->st>>>(c->dz + off, njobs, nrows, geo(c),
                                                                        tw(c), sc, nkz(c, masked), masked ? c->tr.mp : NZC, win);
        else
            k_z_c2r<T, N, 0><<<njobs * ntiles, LZ * PV<0>, smem, c->st>>>(c->dz + off, njobs, nrows, geo(c),
                                                                        tw(c), sc, nkz(c, masked), masked ? c->tr.mp : NZC, win);
    }
    // masked: only the rows' kept part, in rows of whole tiles
    static void zr2c(kf_ctx *c, int off, int njobs, bool masked = false) {
        const int pitch = masked ? c->tr.mp : NZC;
        const int nrows = N * N;
        const int ntiles = (nrows + LZ - 1) / LZ;
        const size_t smem = ZSmem<T, N, false>::bytes;
        Launch L_(c, KC_Z_R2C, z_bytes(c, off, njobs, false, masked));
        if (c->fftv)
            k_z_r2c<T, N, 1><<<njobs * ntiles, LZ * PV<1>, smem, c->st>>>(c->dz + off, njobs, nrows, tw(c), pitch);
        else
            k_z_r2c<T, N, 0><<<njobs * ntiles, LZ * PV<0>, smem, c->st>>>(c->dz + off, njobs, nrows, tw(c), pitch);
    }
    static RhsArgs<T> rargs(kf_ctx *c) {
        RhsArgs<T> a;
        for (int q = 0; q < 4; ++q) a.Y[q] = (const T2 *)c->Ys[q];
        a.phihat = (const T2 *)c->phihat;
        a.SV = (const T *)c->SV;
        a.PF = (const T *)c->PF;
        a.tau = (T)c->cfg.tau;
        a.theta = (T)c->cfg.theta;
        a.M = (T)c->cfg.M;
        a.D = (T)c->cfg.diff_D;
        a.terms = c->cfg.terms;
        return a;
    }

    // Round D's passes on u' (the first 6 x and 9 y jobs of its lists): every
    // input is the stage state.
    static void round_D_us(kf_ctx *c) {
        axis(c, c->jD_x, 6, 0, +1, AX_XM);
        axis(c, c->jD_y, 9, 1, +1, AX_YI);
    }

    // rho = exp(c2r(P s)) + n_d (and its colour-split copy) from round A's P s
    // in CY[0]; s_d itself into R[0] on the rows of the window
    static void rho_pass(kf_ctx *c, const int *window) {
        const int nb = zline_blocks<T, N>();
        const size_t smem = (size_t)LZ * PadLen<N>::value * sizeof(T2);
        const T sc = (T)(1. / ((double)N * N * N));
        double *rho = captured_solve(c) && split_on(c, 0) ? nullptr : c->rho;  // then only the split copy is read
        Launch L_(c, KC_RHO, (double)N * N * nkz(c, true) * sizeof(T2) + (double)c->N * (8 + (rho ? 8 : 0) + (c->rho_cs ? 8 : 0)));
        if (c->fftv)
            k_z_rho<T, N, 1><<<nb, LZ * PV<1>, smem, c->st>>>((const T2 *)c->CY[0], (T *)c->R[0], window, c->nd, rho, c->rho_cs,
                                                              tw(c), sc, nkz(c, true), c->tr.mp);
        else
            k_z_rho<T, N, 0><<<nb, LZ * PV<0>, smem, c->st>>>((const T2 *)c->CY[0], (T *)c->R[0], window, c->nd, rho, c->rho_cs,
                                                              tw(c), sc, nkz(c, true), c->tr.mp);
        CK(cudaGetLastError());
    }

    // phi^ = r2c(phi) in the bulk precision.  With the pressure term phi^ is used
    // times the filter table PF alone, which underflows to 0 for the larger wave
    // numbers (kz above 0.4 n/2 in FP32): only the columns where it does not are
    // formed, and phi^ is not read where it does.  (Together with phi staying in split
    // order between the stages: 2-4 % of a 256^3 step.)
    static void phi_transform(kf_ctx *c) {
        const int nb = zline_blocks<T, N>();
        const size_t smem = (size_t)LZ * PadLen<N>::value * sizeof(T2);
        const bool pf = (c->cfg.terms & T_PRESSURE) && c->pf.nkz;
        const bool sp = captured_solve(c) && split_on(c, 0);  // (solve_end comes with the last stage)
        const int nko = pf ? c->pf.nkz : NZC, pitch = pf ? c->pf.mp : NZC;
        const double *phi = sp ? c->phi_cs : c->phi;
        const int mode = pf ? AX_YF : AX_FULL;
        {
            Launch L_(c, KC_Z_R2C, (double)c->N * 8 + (double)N * N * nko * sizeof(T2));
            auto go = [&](auto k, int threads) {
                k<<<nb, threads, smem, c->st>>>(phi, (T2 *)c->CX[8], tw(c), nko, pitch);
            };
            if (c->fftv)
                go(sp ? k_z_phi<T, N, 1, true> : k_z_phi<T, N, 1, false>, LZ * PV<1>);
            else
                go(sp ? k_z_phi<T, N, 0, true> : k_z_phi<T, N, 0, false>, LZ * PV<0>);
            CK(cudaGetLastError());
        }
        axis(c, c->jB_y, 1, 1, -1, mode, &c->pf);
        axis(c, c->jB_x, 1, 0, -1, pf ? AX_XF : AX_FULL, &c->pf);
    }

    // rounds D (z), E and the z part of F: k_zprod -> CX[0..3]
    // (RL: with the linear terms' lines)
    template <bool RL> static void zprod(kf_ctx *c, bool pen) {
        ZProdArgs<T> a{};
        a.s0 = (const T2 *)c->CY[0];
        a.sy = (const T2 *)c->CY[1];
        a.sx = (const T2 *)c->CY[2];
        for (int q = 0; q < 3; ++q) {
            a.u[q] = (const T2 *)c->CY[3 + 3 * q];
            a.uy[q] = (const T2 *)c->CY[4 + 3 * q];
            a.ux[q] = (const T2 *)c->CY[5 + 3 * q];
        }
        for (int q = 0; q < 4; ++q) {
            a.out[q] = (T2 *)c->CX[q];
            a.rl[q] = (const T *)c->R[16 + q];
            a.lin[q] = (const T2 *)c->CY[12 + q];
        }
        a.sd = (const T *)c->R[0];
        a.H = (const T *)c->H;
        a.box = pen ? c->d_box : nullptr;
        a.M = (T)c->cfg.M;
        a.eta = (T)c->cfg.pen_eta;
        a.scale = (T)(1. / ((double)N * N * N));
        a.terms = c->cfg.terms;
        a.nkz = nkz(c, true);
        a.ip = c->tr.mp;
        a.nko = nkz(c, pen);
        a.op = pen ? c->tr.mp : NZC;
        const size_t smem = ZProdSmem<T, N, RL>::bytes;
        Launch L_(c, KC_PROD, (double)N * N * sizeof(T2) * (12. * a.nkz + 4. * a.nko + (RL ? 4. * NZC : 0.)) + (pen ? (RL ? 2. : 6.) * c->bx_i * c->bx_j * N : 0.) * sizeof(T));
        if (c->fftv)
            k_zprod<T, N, 1, RL><<<N * N / ZP_ROWS, ZProdLines<RL>::value * PV<1>, smem, c->st>>>(a, (const T *)c->kv, tw(c));
        else
            k_zprod<T, N, 0, RL><<<N * N / ZP_ROWS, ZProdLines<RL>::value * PV<0>, smem, c->st>>>(a, (const T *)c->kv, tw(c));
        CK(cudaGetLastError());
    }

    // In a captured step, fork round_D_us onto st_side after round A; rhs
    // joins it before the products.  The branch writes CX[2..7] and CY[3..11],
    // which nothing between the fork and the join touches (the
    // Poisson solve, round B in CX[8] / CY[12], k_lin, round D's LIN part).
    // (Measured at 256^3 FP32 bulk: +1 to +2.4 % per step; the Poisson chain
    // at a higher stream priority than the branch was slower than equal
    // priorities, and the branch's transform passes on half the persistent
    // grid were no faster.)
    static bool fork_D(kf_ctx *c) {
        if (!(c->capturing && c->overlap_d)) return false;
        CK(cudaEventRecord(c->ev_fork, c->st));
        CK(cudaStreamWaitEvent(c->st_side, c->ev_fork, 0));
        if (c->capture_wait_u && c->stage_idx == 0)
            CK(cudaStreamWaitEvent(c->st_side, c->ev_u, cudaEventWaitExternal));
        cudaStream_t main = c->st;
        c->st = c->st_side;
        try {
            round_D_us(c);
        } catch (...) {
            c->st = main;
            throw;
        }
        c->st = main;
        CK(cudaEventRecord(c->ev_join, c->st_side));
        return true;
    }

    // rounds A (P s, d_x s, d_y s, the Poisson source and, with penalization, s_d
    // in R[0] where the mask is not zero), the Poisson solve and B (phi^ =
    // r2c(phi)), shared by both right-hand sides
    static bool rounds_AB(kf_ctx *c, bool fork) {
        const int Tm = c->cfg.terms;
        const bool pois = (Tm & T_POISSON) && (Tm & T_E_INT);
        // A
        axis(c, c->jA_x, 2, 0, +1, AX_XM);
        axis(c, c->jA_y, 3, 1, +1, AX_YI);
        const bool solve = pois && !c->phi_given;
        const bool pen = Tm & T_PENALIZATION;
        if (solve)
            rho_pass(c, pen ? c->d_box : nullptr);
        else if (pen)
            zc2r(c, c->zA, 1, true);
        const bool forked = fork && fork_D(c);
        if (solve) {
            if (c->capturing) {
                poisson_captured(c);
            } else {
                const bool newtime = phi_guess(c);
                int rc = poisson(c, true);
                if (rc) throw KfError{KF_ERR_NOT_CONVERGED, "Poisson solve did not reach its tolerance"};
                if (c->cfg.phi_extrap && newtime) {
                    c->nhist = c->nhist < 2 ? c->nhist + 1 : 2;
                    c->tau_b = c->t_stage;
                }
            }
        }
        // B
        if (c->capturing && c->capture_wait_u && c->stage_idx == 0)
            CK(cudaStreamWaitEvent(c->st, c->ev_u, cudaEventWaitExternal));
        if (Tm & T_E_INT) {
            phi_transform(c);
        }
        return forked;
    }

    // one right-hand-side evaluation: Ys -> K
    static void rhs(kf_ctx *c) {
        const int Tm = c->cfg.terms;
        const bool pen = Tm & T_PENALIZATION;
        const bool forked = rounds_AB(c, true);
        // C
        {
            Launch L_(c, KC_LIN, (double)c->Nc * (9 * sizeof(T2) + 2 * sizeof(T)));
            const auto k = pen && !RLINES ? k_lin<T, !RLINES> : k_lin<T, false>;
            k<<<mg_grid(NZC, N), mg_block(), 0, c->st>>>(rargs(c), geo(c), (T2 *)c->LIN[0], (T2 *)c->LIN[1],
                                                         (T2 *)c->LIN[2], (T2 *)c->LIN[3]);
        }
        const bool rl = RLINES && pen;
        if (rl) {  // the linear terms' inverse x and y passes, whole
            axis(c, c->jD_x + 6, 4, 0, +1);
            axis(c, c->jD_y + 9, 4, 1, +1);
        } else if (pen) {  // c2r(-lin_q) on the mask's window
            axis(c, c->jD_x + 6, 4, 0, +1, AX_XB);
            axis(c, c->jD_y + 9, 4, 1, +1, AX_YB);
            zc2r(c, c->zD + 8, 2, false, -1., true);
        }
        // D: the u', s part, unless forked
        if (!forked)
            round_D_us(c);
        else
            CK(cudaStreamWaitEvent(c->st, c->ev_join, 0));
        // z part of D, E, z part of F (with penalization only what the 2/3 rule keeps is formed)
        if constexpr (RLINES) {
            if (rl)
                zprod<true>(c, pen);
            else
                zprod<false>(c, pen);
        } else {
            zprod<false>(c, pen);
        }
        axis(c, c->jF_y, 4, 1, -1, pen ? AX_YF : AX_FULL);
        stage(c, pen, !rl);
    }

    // the end of F: the forward x pass, K and its use in the RK4 stage
    // (lin: with the linear terms of k_lin)
    static void stage(kf_ctx *c, bool pen, bool lin) {
        const AxTrunc A = trunc(c, pen ? AX_XM : AX_FULL, false);
        StageArgs<T> a;
        for (int q = 0; q < 4; ++q) {
            a.in[q] = (const T2 *)c->CY[q];
            a.lin[q] = lin ? (const T2 *)c->LIN[q] : nullptr;
            a.y[q] = (T2 *)c->Y[q];
            a.acc[q] = (T2 *)c->ACC[q];
            a.ys[q] = (T2 *)c->Ys[q];
            a.K[q] = (T2 *)c->K[q];
        }
        a.c = (T)c->rk_c;
        a.mode = c->rk_mode;
        const bool act = A.mode == AX_XM;
        const int ntiles = act ? c->tr.nt : (N * NZC + TC - 1) / TC;
        const double use = act ? c->tr_ball : (double)c->Nc;
        const size_t sm = (size_t)N * TC * sizeof(T2);
        Launch L_(c, KC_XASM, 4. * sizeof(T2) * ((act ? c->tr.cols : use) + use * (a.mode == 3 ? 2 : a.mode == 0 ? 4 : 5)));
        if (c->fftv)
            k_xfwd_stage<T, N, 1><<<4 * ntiles, TC * PV<1>, sm, c->st>>>(a, geo(c), tw(c), A);
        else
            k_xfwd_stage<T, N, 0><<<4 * ntiles, TC * PV<0>, sm, c->st>>>(a, geo(c), tw(c), A);
        CK(cudaGetLastError());
    }

    // The right-hand side on sine-stretched axes: every derivative takes the
    // chain-rule path D_d F = r2c(m_d c2r(P i k_d F)) of
    // OP_partial_derivative.cpp:104-136.  What the right-hand side adds of them as
    // they are it adds in physical space, to the products, and transforms once:
    //   C' linear parts, F1                 D' raw derivatives (15 c2r)
    //   E' times the metric; sums S_q       c2r(-lin_q) on the mask's window
    //   G' c2r(P D_d u'_c), c2r(P D_d s): 12 fields forward and back, filtered
    //   H' S_q + products (rhs_standard.cpp:323-436), penalization
    //   then the end of F, as rhs()
    // (15 + 4 forward transforms of derivatives and products, their assembly in
    // k-space and the penalization of the assembled right-hand side through
    // another 4 back and forth before.)
    static void rhs_stretched(kf_ctx *c) {
        const int Tm = c->cfg.terms;
        const bool pen = Tm & T_PENALIZATION;
        const long Nc = c->Nc, Nr = c->N;
        const double cb = (double)Nc * sizeof(T2), rb = (double)Nr * sizeof(T);
        rounds_AB(c, false);
        {  // C'
            Launch L_(c, KC_LIN, 4 * cb + 6 * cb + 2 * rb);
            k_sl_lin<T><<<nblk(Nc, 256), 256, 0, c->st>>>(rargs(c), geo(c), (T2 *)c->LIN[0], (T2 *)c->LIN[1],
                                                            (T2 *)c->LIN[2], (T2 *)c->LIN[3], (T2 *)c->CX[10], pen);
        }
        // D'
        axis(c, c->jS_Dx, 8, 0, +1, AX_XM);
        axis(c, c->jS_Dy, 12, 1, +1, AX_YI);
        zc2r(c, c->zS_D, 10, true);
        {  // E'
            ScaleArgs<T> sa;
            for (int j = 0; j < 12; ++j) sa.f[j] = (T *)c->R[4 + j];
            for (int j = 0; j < 3; ++j) sa.F1[j] = (const T *)c->R[16 + j];
            for (int j = 0; j < 4; ++j) sa.S[j] = (T *)c->R[20 + j];
            sa.met = (const T *)c->met;
            sa.M = (T)c->cfg.M;
            sa.terms = Tm;
            sa.n = c->n;
            sa.N = Nr;
            Launch L_(c, KC_PROD, 31. * rb);
            k_sl_scale<T><<<nblk(Nr, 256), 256, 0, c->st>>>(sa);
        }
        if (pen) {
            axis(c, c->jD_x + 6, 4, 0, +1, AX_XB);
            axis(c, c->jD_y + 9, 4, 1, +1, AX_YB);
            zc2r(c, c->zD + 8, 2, false, -1., true);
        }
        if (Tm & (T_ADVECTION | T_CONTINUITY)) {  // G'
            zr2c(c, c->zS_F, 6, true);
            axis(c, c->jS_Fy, 12, 1, -1, AX_YF);
            x_filter(c, c->jS_Gx, 12);
            axis(c, c->jS_Gy, 12, 1, +1, AX_YI);
            zc2r(c, c->zS_G, 6, true);
        }
        {  // H'
            SlProdArgs<T> pa{};
            for (int q = 0; q < 3; ++q) {
                pa.U[q] = (const T *)c->R[1 + q];
                pa.ds[q] = (const T *)c->R[13 + q];
                for (int d = 0; d < 3; ++d) pa.dU[q][d] = (const T *)c->R[4 + 3 * q + d];
            }
            for (int q = 0; q < 4; ++q) {
                pa.out[q] = (T *)c->R[20 + q];
                pa.rl[q] = (const T *)c->R[16 + q];
            }
            pa.sd = (const T *)c->R[0];
            pa.H = (const T *)c->H;
            pa.M = (T)c->cfg.M;
            pa.eta = (T)c->cfg.pen_eta;
            pa.box = pen ? c->d_box : nullptr;
            pa.terms = Tm;
            pa.n = c->n;
            pa.N = Nr;
            Launch L_(c, KC_PROD, 23. * rb);
            k_sl_products<T><<<nblk(Nr, 256), 256, 0, c->st>>>(pa);
        }
        zr2c(c, c->zF, 2, pen);
        axis(c, c->jF_y, 4, 1, -1, pen ? AX_YF : AX_FULL);
        stage(c, pen, true);
    }
    static void x_filter(kf_ctx *c, int off, int njobs) {
        const AxTrunc A = trunc(c, AX_XM, false);
        const size_t sm = (size_t)N * TC * sizeof(T2);
        Launch L_(c, KC_AXIS_INV, 2. * njobs * c->tr.cols * sizeof(T2));
        if (c->fftv)
            k_x_filter<T, N, 1><<<njobs * c->tr.nt, TC * PV<1>, sm, c->st>>>(c->dj + off, njobs, geo(c), tw(c), A);
        else
            k_x_filter<T, N, 0><<<njobs * c->tr.nt, TC * PV<0>, sm, c->st>>>(c->dj + off, njobs, geo(c), tw(c), A);
        CK(cudaGetLastError());
    }

    // standalone transforms on R[0] <-> CX[0] (through CY[0])
    static void r2c(kf_ctx *c) {
        zr2c(c, c->zT, 1);
        axis(c, c->jTf_y, 1, 1, -1);
        axis(c, c->jTf_x, 1, 0, -1);
        CK(cudaGetLastError());
    }
    static void c2r(kf_ctx *c) {
        axis(c, c->jT_x, 1, 0, +1);
        axis(c, c->jT_y, 1, 1, +1);
        zc2r(c, c->zT + 1, 1);
        CK(cudaGetLastError());
    }
    // transform passes of the discrete adjoint (job lists of build_adj_jobs)
    static void adj_pass(kf_ctx *c, int which) {
        switch (which) {
            case 0:  // forward intermediates s_d, U_c, d_d U_c, d_d s of the stage input in Ys
                axis(c, c->jA_x, 2, 0, +1, AX_XM);
                axis(c, c->jA_y, 3, 1, +1, AX_YI);
                zc2r(c, c->zA, 1, true);
                round_D_us(c);
                zc2r(c, c->zD, 8, true);
                break;
            case 1:  // f_bar = r2c^T(P Kbar) = c2r_unscaled(P Kbar / w)
            {
                const bool pen = c->cfg.terms & T_PENALIZATION;  // masked then (build_adj_jobs)
                axis(c, c->jV_x, 4, 0, +1, pen ? AX_XM : AX_FULL);
                axis(c, c->jV_y, 4, 1, +1, pen ? AX_YI : AX_FULL);
                zc2r(c, c->zV, 2, pen, 1.);
            }
                break;
            case 2:  // r2c of the physical cotangents
                zr2c(c, c->zW, c->nWz);
                axis(c, c->jW_y, c->nWf, 1, -1);
                axis(c, c->jW_x, c->nWf, 0, -1);
                break;
            case 3:  // phi_bar = r2c^T(phihat_bar)
                axis(c, c->jP_x, 1, 0, +1);
                axis(c, c->jP_y, 1, 1, +1);
                zc2r(c, c->zP, 1, false, 1.);
                break;
            case 4:  // r2c of s_d_bar
                zr2c(c, c->zS, 1);
                axis(c, c->jS_y, 1, 1, -1);
                axis(c, c->jS_x, 1, 0, -1);
                break;
            case 5:  // r2c^T of the s cotangent, and c2r of the state's s
                axis(c, c->jQ_x, 2, 0, +1);
                axis(c, c->jQ_y, 2, 1, +1);
                zc2r(c, c->zQ, 1, false, 1.);
                zc2r(c, c->zQ + 1, 1);
                break;
            case 6:  // s_d only (the Poisson source of the state in Ys)
                axis(c, c->jA_x, 2, 0, +1, AX_XM);
                axis(c, c->jA_y, 3, 1, +1, AX_YI);
                zc2r(c, c->zA, 1, true);
                break;
        }
        CK(cudaGetLastError());
    }
    // inverse transforms of the (undealiased) state into R[20..23] for diagnostics
    static void inv_state(kf_ctx *c) {
        axis(c, c->jG_x, 4, 0, +1);
        axis(c, c->jG_y, 4, 1, +1);
        zc2r(c, c->zG, 2);
        CK(cudaGetLastError());
    }
};

template <typename T> struct Dispatch {
    static bool pick(kf_ctx *c) {
        switch (c->n) {
#define KF_CASE(NN)                                    \
    case NN:                                           \
        Impl<T, NN>::set_attrs();                      \
        c->rhs_fn = c->stretched ? &Impl<T, NN>::rhs_stretched : &Impl<T, NN>::rhs; \
        c->r2c_fn = &Impl<T, NN>::r2c;                 \
        c->c2r_fn = &Impl<T, NN>::c2r;                 \
        c->inv_state_fn = &Impl<T, NN>::inv_state;     \
        c->adj_fn = &Impl<T, NN>::adj_pass;            \
        return true;
            KF_CASE(16)
            KF_CASE(32)
            KF_CASE(64)
            KF_CASE(96)
            KF_CASE(128)
            KF_CASE(256)
#undef KF_CASE
            default:
                return false;
        }
    }
};

// radix stages and threads per line of the two transform plans of length n
template <int NN> void plan_info_n(int rad[2][4], int thr[2]) {
    for (int i = 0; i < 4; ++i) {
        rad[0][i] = PlanV<NN, 0>::radix[i];
        rad[1][i] = PlanV<NN, 1>::radix[i];
    }
    thr[0] = PlanV<NN, 0>::P;
    thr[1] = PlanV<NN, 1>::P;
}
void plan_info(int n, int rad[2][4], int thr[2]) {
    switch (n) {
        case 16: plan_info_n<16>(rad, thr); break;
        case 32: plan_info_n<32>(rad, thr); break;
        case 64: plan_info_n<64>(rad, thr); break;
        case 96: plan_info_n<96>(rad, thr); break;
        case 128: plan_info_n<128>(rad, thr); break;
        case 256: plan_info_n<256>(rad, thr); break;
        default: break;
    }
}

std::vector<double> plan_tw(int n, int v) {
    switch (n) {
        case 16: return v ? plan_twiddles<16, 1>() : plan_twiddles<16, 0>();
        case 32: return v ? plan_twiddles<32, 1>() : plan_twiddles<32, 0>();
        case 64: return v ? plan_twiddles<64, 1>() : plan_twiddles<64, 0>();
        case 96: return v ? plan_twiddles<96, 1>() : plan_twiddles<96, 0>();
        case 128: return v ? plan_twiddles<128, 1>() : plan_twiddles<128, 0>();
        default: return v ? plan_twiddles<256, 1>() : plan_twiddles<256, 0>();
    }
}

// FP64 sums of the charge density e^s - e^phi + n_d and the kinetic energy
// density 0.5 e^s |M e_x + u'|^2 (block partials in slots 0 and 1).
template <typename T>
__global__ void __launch_bounds__(RBS) k_diag_sums(const T *__restrict__ s, const T *__restrict__ ux,
                                                   const T *__restrict__ uy, const T *__restrict__ uz,
                                                   const double *__restrict__ phi, const double *__restrict__ nd,
                                                   double M, long N, double *__restrict__ partial,
                                                   const double *__restrict__ vol, int n) {
    __shared__ double sh[2 * RBS];
    double ch = 0., kin = 0.;
    for (long i = (long)blockIdx.x * RBS + threadIdx.x; i < N; i += (long)gridDim.x * RBS) {
        // cell volume / h^3: 1, or dS(x) dS(y) dS(z) on stretched axes
        double w = 1.;
        if (vol) w = vol[i / ((long)n * n)] * vol[(i / n) % n] * vol[i % n];
        const double n_i = exp((double)s[i]);
        ch += w * (n_i - exp(phi[i]) + nd[i]);
        const double vx = M + (double)ux[i], vy = (double)uy[i], vz = (double)uz[i];
        kin += w * (0.5 * n_i * (vx * vx + vy * vy + vz * vz));
    }
    sh[threadIdx.x] = kin;
    sh[RBS + threadIdx.x] = ch;
    __syncthreads();
    for (int w = RBS / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            sh[threadIdx.x] += sh[threadIdx.x + w];
            sh[RBS + threadIdx.x] += sh[RBS + threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        partial[(long)blockIdx.x * KF_RED + 0] = sh[0];
        partial[(long)blockIdx.x * KF_RED + 1] = sh[RBS];
    }
}

__global__ void k_diag_final(const double *__restrict__ partial, int nb, double *__restrict__ out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double a = 0., b = 0.;
        for (int i = 0; i < nb; ++i) {
            a += partial[(long)i * KF_RED + 0];
            b += partial[(long)i * KF_RED + 1];
        }
        out[0] = a;
        out[1] = b;
    }
}

void build_tables(kf_ctx *c) {
    const int n = c->n, nzc = c->nzc;
    const double L = c->cfg.L;
    std::vector<double> kv(n), q2(n);
    const double kmax = k_val_at(n / 2, n, L);
    const double kzq = k_val_at(nzc / 2, n, L);  // operations.hpp:25 quirk: field_imag::Nz = n/2+1
    for (int i = 0; i < n; ++i) {
        kv[i] = k_val_at(i, n, L);
        q2[i] = pow(kv[i] / kmax, 2.);
    }
    // the tables depend on |kx|, |ky| and are the same with the two exchanged (the
    // sums' first two terms): formed for n/2 >= i >= j, copied elsewhere
    std::vector<double> SV(c->Nc), PF(c->Nc);
    auto at = [&](int i, int j) { return (size_t)nzc * ((size_t)j + (size_t)i * n); };
    for (int i = 0; i <= n / 2; ++i)
        for (int j = 0; j <= i; ++j)
            for (int k = 0; k < nzc; ++k) {
                const size_t ijk = at(i, j) + k;
                const double kx = kv[i], ky = kv[j], kz = kv[k];
                // rhs_standard.cpp:64-71 (field_SV), optional cut at sv_cut
                const double knorm = sqrt(pow(kx / kmax, 2.) + pow(ky / kmax, 2.) + pow(kz / kmax, 2.));
                const double filter = 1. - exp(-8. * pow(sqrt(knorm), 8.));
                double svv = c->cfg.sv_eps * filter;
                if (c->cfg.sv_cut > 0. && !(knorm > c->cfg.sv_cut)) svv = 0.;
                SV[ijk] = svv;
                // operations.hpp:35-40 with the filter of rhs_standard.cpp:220
                const double kq = sqrt(pow(kx / kmax, 2.) + pow(ky / kmax, 2.) + pow(kz / kzq, 2.));
                PF[ijk] = exp(-2000. * pow(kq, 15.));
            }
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j) {
            const int a = std::min(i, n - i), b = std::min(j, n - j);
            const size_t src = at(std::max(a, b), std::min(a, b)), dst = at(i, j);
            if (src == dst) continue;
            std::copy_n(&SV[src], nzc, &SV[dst]);
            std::copy_n(&PF[src], nzc, &PF[dst]);
        }
    c->q2 = dalloc<double>(c, sizeof(double) * n);
    CK(cudaMemcpy(c->q2, q2.data(), sizeof(double) * n, cudaMemcpyHostToDevice));
    auto cols = [&](const std::vector<int> &pb, kf_ctx::Cols &o) {
        const int tc = c->fp32 ? Tile<float>::TC : Tile<double>::TC;
        const TruncTab t = trunc_table(pb, n, tc);
        o.nkz = t.nkz;
        o.nt = (int)t.tl.size();
        o.mp = std::min((t.nkz + tc - 1) / tc * tc, nzc);
        for (int b : pb) o.cols += b >= 0 ? n : 0;
        if (!o.nkz) return;
        o.jb = dalloc<int>(c, sizeof(int) * t.jb.size());
        o.tl = dalloc<int>(c, sizeof(int) * t.tl.size());
        CK(cudaMemcpy(o.jb, t.jb.data(), sizeof(int) * t.jb.size(), cudaMemcpyHostToDevice));
        CK(cudaMemcpy(o.tl, t.tl.data(), sizeof(int) * t.tl.size(), cudaMemcpyHostToDevice));
    };
    {
        const std::vector<int> pb = dealias_bounds(q2, n, dealias_threshold());
        c->pb = dalloc<int>(c, sizeof(int) * pb.size());
        CK(cudaMemcpy(c->pb, pb.data(), sizeof(int) * pb.size(), cudaMemcpyHostToDevice));
        cols(pb, c->tr);
        for (int b : pb)
            if (b >= 0) c->tr_ball += 2 * b + 1;
        // PF falls with every |k_d|, so a column's largest value is that of row 0
        std::vector<int> pf((size_t)n * nzc);
        for (size_t e = 0; e < pf.size(); ++e)
            pf[e] = (c->fp32 ? (float)PF[e] != 0.f : PF[e] != 0.) ? 0 : -1;
        cols(pf, c->pf);
    }
    if (c->fp32) {
        std::vector<float> kvf(n), SVf(c->Nc), PFf(c->Nc);
        for (int i = 0; i < n; ++i) kvf[i] = (float)kv[i];
        for (long i = 0; i < c->Nc; ++i) { SVf[i] = (float)SV[i]; PFf[i] = (float)PF[i]; }
        c->kv = dalloc<void>(c, 4 * n);
        c->SV = dalloc<void>(c, 4 * c->Nc);
        c->PF = dalloc<void>(c, 4 * c->Nc);
        CK(cudaMemcpy(c->kv, kvf.data(), 4 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(c->SV, SVf.data(), 4 * c->Nc, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(c->PF, PFf.data(), 4 * c->Nc, cudaMemcpyHostToDevice));
    } else {
        c->kv = dalloc<void>(c, 8 * n);
        c->SV = dalloc<void>(c, 8 * c->Nc);
        c->PF = dalloc<void>(c, 8 * c->Nc);
        CK(cudaMemcpy(c->kv, kv.data(), 8 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(c->SV, SV.data(), 8 * c->Nc, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(c->PF, PF.data(), 8 * c->Nc, cudaMemcpyHostToDevice));
    }
    for (int v = 0; v < 2; ++v) {
        const std::vector<double> w = plan_tw(n, v);
        c->tw[v] = dalloc<void>(c, c->es * w.size());
        if (c->fp32) {
            const std::vector<float> wf(w.begin(), w.end());
            CK(cudaMemcpy(c->tw[v], wf.data(), 4 * w.size(), cudaMemcpyHostToDevice));
        } else {
            CK(cudaMemcpy(c->tw[v], w.data(), 8 * w.size(), cudaMemcpyHostToDevice));
        }
    }
    if (c->stretched) {
        const std::vector<double> met = metric_table(n, L, c->cfg.stretch_m, dealias_threshold());
        std::vector<double> vol(n);
        for (int i = 0; i < n; ++i) vol[i] = dS_at(i, n, L, c->cfg.stretch_m);
        c->met = dalloc<void>(c, c->es * n);
        c->vol = dalloc<double>(c, 8 * n);
        if (c->fp32) {
            std::vector<float> mf(met.begin(), met.end());
            CK(cudaMemcpy(c->met, mf.data(), 4 * n, cudaMemcpyHostToDevice));
        } else {
            CK(cudaMemcpy(c->met, met.data(), 8 * n, cudaMemcpyHostToDevice));
        }
        CK(cudaMemcpy(c->vol, vol.data(), 8 * n, cudaMemcpyHostToDevice));
    }
}

void cc_setup(kf_ctx *c);


void build_levels(kf_ctx *c) {
    const kf_config &cf = c->cfg;
    int nl = 1;
    if (cf.poisson_mode == KF_PS_FAS) nl = cf.mg_levels > 1 ? cf.mg_levels : 1;
    if (cf.poisson_mode == KF_PS_CASCADIC) nl = 4;
    for (int l = 1; l < nl; ++l)
        if ((c->n >> l) < 2 || ((c->n >> (l - 1)) % 2))
            throw KfError{KF_ERR_ARG, "too many multigrid levels for this grid"};
    // a red-black order needs even grids: with an odd level the half sweeps read
    // and write past the level's end
    if (cf.poisson_mode == KF_PS_FAS && (c->n >> (nl - 1)) % 2)
        throw KfError{KF_ERR_ARG, "an FAS level with an odd number of points per axis; fewer levels needed"};
    if (cf.poisson_mode == KF_PS_CASCADIC && c->n % 8) throw KfError{KF_ERR_ARG, "cascadic plan needs n % 8 == 0"};
    if (cf.poisson_mode == KF_PS_FAS && ((long)(c->n >> (nl - 1)) * (c->n >> (nl - 1)) * (c->n >> (nl - 1)) > 8192))
        throw KfError{KF_ERR_ARG, "coarsest FAS level above 8192 points (shared-memory solve); add levels"};
    CK(cudaFuncSetAttribute(k_coarse_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    march_attrs();
    c->march_maps = encode_tiled() != nullptr;  // before the levels: L.t depends on it
    c->lv.resize(nl);
    for (int l = 0; l < nl; ++l) {
        LevelBuf &L = c->lv[l];
        const int n = c->n >> l;
        L.n = n;
        const double Lb = cf.L;
        std::vector<double> H(n + 1), dd(n), dp(n), dm(n), ip(n), im(n), rp(n), rm(n), gam(n, 0.);
        const double sm = cf.stretch_m;
        for (int i = 0; i < n + 1; ++i) H[i] = val_at(i, n, Lb, sm) - val_at(i - 1, n, Lb, sm);  // H_create (:112-126)
        for (int i = 0; i < n; ++i) {
            dd[i] = 2. / (H[i + 1] * H[i]);
            dp[i] = H[i + 1] * (H[i + 1] + H[i]);
            dm[i] = H[i] * (H[i + 1] + H[i]);
            ip[i] = 2. / dp[i];
            im[i] = 2. / dm[i];
            rp[i] = div_reciprocal(dp[i]);
            rm[i] = div_reciprocal(dm[i]);
        }
        for (int m = 1; m < n; m += 2) {  // OP_hto2h gamma on this (fine) axis
            const double x1 = val_at(m - 1, n, Lb, sm), x2 = val_at(m + 1, n, Lb, sm), x = val_at(m, n, Lb, sm);
            gam[m] = (x - x1) / (x2 - x1);
        }
        L.dd = dalloc<double>(c, 8 * n);
        L.dp = dalloc<double>(c, 8 * n);
        L.dm = dalloc<double>(c, 8 * n);
        L.gam = dalloc<double>(c, 8 * n);
        L.ip = dalloc<double>(c, 8 * n);
        L.im = dalloc<double>(c, 8 * n);
        L.rp = dalloc<double>(c, 8 * n);
        L.rm = dalloc<double>(c, 8 * n);
        CK(cudaMemcpy(L.rp, rp.data(), 8 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(L.rm, rm.data(), 8 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(L.ip, ip.data(), 8 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(L.im, im.data(), 8 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(L.dd, dd.data(), 8 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(L.dp, dp.data(), 8 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(L.dm, dm.data(), 8 * n, cudaMemcpyHostToDevice));
        CK(cudaMemcpy(L.gam, gam.data(), 8 * n, cudaMemcpyHostToDevice));
        L.tab = std::make_shared<AxTab>();  // n <= KF_TAB_N for every grid size
        for (int m = 0; m < n; ++m) {
            L.tab->dd[m] = dd[m];
            L.tab->ip[m] = ip[m];
            L.tab->im[m] = im[m];
        }
        const size_t bytes = sizeof(double) * (size_t)n * n * n;
        L.r = dalloc<double>(c, bytes);
        if (cf.poisson_mode == KF_PS_FAS && march_level(L) && c->march_maps) {
            L.t = dalloc<double>(c, bytes);
            CUtensorMap probe;  // the encoder must accept this level's row copies
            if (!row_map(&probe, L.t, n)) L.t = nullptr;
        }
        if (l == 0) {
            L.phi = c->phi;
            L.rho = c->rho;
        } else {
            L.phi = dalloc<double>(c, bytes);
            L.rho = dalloc<double>(c, bytes);
            L.phi0 = dalloc<double>(c, bytes);
        }
        // above the sizes that the cluster takes, where bandwidth counts
        L.sp = cf.poisson_mode == KF_PS_FAS && nl > 1 && l + 1 < nl && n > CC_MAX_N && n % 16 == 0;
        if (L.sp) {
            std::vector<double> t(3 * n);
            for (int k = 0; k < n; ++k) {
                const int e = (k & 1) * (n / 2) + k / 2;
                t[e] = dd[k];
                t[n + e] = ip[k];
                t[2 * n + e] = im[k];
            }
            L.ddk = dalloc<double>(c, 8 * t.size());
            L.ipk = L.ddk + n;
            L.imk = L.ipk + n;
            CK(cudaMemcpy(L.ddk, t.data(), 8 * t.size(), cudaMemcpyHostToDevice));
            if (l == 0) {
                c->phi_cs = dalloc<double>(c, bytes);
                c->rho_cs = dalloc<double>(c, bytes);
                CK(cudaMemset(c->rho_cs, 0, bytes));  // kf_autotune reads it, with or without a solve before
            }
            L.ph = l == 0 ? c->phi_cs : L.phi;
            L.rh = l == 0 ? c->rho_cs : L.rho;
        }
    }
    for (const void *k : {(const void *)k_cc<false>, (const void *)k_cc<true>}) {
        CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CC_SMEM_MAX));
        CK(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    }
    cc_setup(c);
}

// The coarse levels that k_cc takes: from the first level below the finest with
// n <= 32 down, in a cluster of as many CTAs as divide the coarsest n (one plane
// of it each at 16^3: the chain of sweeps there is what the size serves), as long
// as the levels fit the kernel and the device can hold such a cluster; -1 with
// the switch off.  (From 64^3 down a cluster's 16 SMs would be slower than the
// whole chip with its launches.)
void cc_setup(kf_ctx *c) {
    c->cc_level = -1;
    const int nl = (int)c->lv.size();
    if (!c->coarse_block || c->cfg.poisson_mode != KF_PS_FAS || nl < 2) return;
    int lb = 1;
    while (lb < nl - 1 && (c->lv[lb].n > CC_MAX_N || nl - lb > CC_LEVELS)) ++lb;
    if (c->lv[lb].n > CC_MAX_N) return;
    ClusterCycle C{};
    C.nl = nl - lb;
    for (int m = 0; m < C.nl; ++m) {
        const LevelBuf &L = c->lv[lb + m];
        C.n[m] = L.n;
        C.dd[m] = L.dd;
        C.ip[m] = L.ip;
        C.im[m] = L.im;
        C.gam[m] = L.gam;
    }
    const int nc = c->lv[nl - 1].n;
    for (int cl = std::min(nc, CC_MAX_CTAS); cl >= 1; --cl) {
        const size_t sm = cc_smem(C, cl, true);
        if (nc % cl || sm > (size_t)CC_SMEM_MAX) continue;
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3(cl);
        lc.blockDim = dim3(CC_THREADS);
        lc.dynamicSmemBytes = sm;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = cl;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        lc.attrs = &at;
        lc.numAttrs = 1;
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, k_cc<true>, &lc) != cudaSuccess) {
            cudaGetLastError();
            fit = 0;
        }
        if (fit < 1) continue;
        c->ccyc = C;
        c->cc_ctas = cl;
        c->cc_level = lb;
        return;
    }
}

void build_jobs(kf_ctx *c) {
    std::vector<AxisJob> J;
    std::vector<ZJob> Z;
    auto aj = [&](const void *in, void *out, int mul) { J.push_back(AxisJob{in, out, mul, 0}); };
    auto zj = [&](const void *ia, int ma, const void *ib, int mb, void *oa, void *ob) {
        Z.push_back(ZJob{ia, ib, oa, ob, ma, mb});
    };
    void **CX = c->CX, **CY = c->CY, **R = c->R;
    // A
    c->jA_x = (int)J.size();
    aj(c->Ys[3], CX[0], MUL_P);
    aj(c->Ys[3], CX[1], MUL_P_IK);
    c->jA_y = (int)J.size();
    aj(CX[0], CY[0], MUL_NONE);
    aj(CX[0], CY[1], MUL_IK);
    aj(CX[1], CY[2], MUL_NONE);
    c->zA = (int)Z.size();
    zj(CY[0], MUL_NONE, nullptr, 0, R[0], nullptr);
    // B
    c->jB_y = (int)J.size();  // CX[8], CY[12]: not written by round D's u', s part
    aj(CX[8], CY[12], MUL_NONE);
    c->jB_x = (int)J.size();
    aj(CY[12], c->phihat, MUL_NONE);
    // D
    c->jD_x = (int)J.size();
    for (int q = 0; q < 3; ++q) {
        aj(c->Ys[q], CX[2 + 2 * q], MUL_P);
        aj(c->Ys[q], CX[3 + 2 * q], MUL_P_IK);
    }
    for (int q = 0; q < 4; ++q) aj(c->LIN[q], CX[8 + q], MUL_NONE);
    c->jD_y = (int)J.size();
    for (int q = 0; q < 3; ++q) {
        aj(CX[2 + 2 * q], CY[3 + 3 * q], MUL_NONE);
        aj(CX[2 + 2 * q], CY[4 + 3 * q], MUL_IK);
        aj(CX[3 + 2 * q], CY[5 + 3 * q], MUL_NONE);
    }
    for (int q = 0; q < 4; ++q) aj(CX[8 + q], CY[12 + q], MUL_NONE);
    c->zD = (int)Z.size();
    for (int q = 0; q < 3; ++q) {
        zj(CY[3 + 3 * q], MUL_NONE, CY[3 + 3 * q], MUL_IK, R[1 + q], R[4 + 3 * q + 2]);  // U_c, d_z U_c
        zj(CY[4 + 3 * q], MUL_NONE, CY[5 + 3 * q], MUL_NONE, R[4 + 3 * q + 1], R[4 + 3 * q + 0]);  // d_y, d_x
    }
    zj(CY[1], MUL_NONE, CY[2], MUL_NONE, R[14], R[13]);  // d_y s, d_x s
    zj(CY[0], MUL_IK, nullptr, 0, R[15], nullptr);       // d_z s
    zj(CY[12], MUL_NONE, CY[13], MUL_NONE, R[16], R[17]);
    zj(CY[14], MUL_NONE, CY[15], MUL_NONE, R[18], R[19]);
    // F
    c->zF = (int)Z.size();
    zj(R[20], 0, R[21], 0, CX[0], CX[1]);
    zj(R[22], 0, R[23], 0, CX[2], CX[3]);
    c->jF_y = (int)J.size();
    for (int q = 0; q < 4; ++q) aj(CX[q], CY[q], MUL_NONE);
    // standalone transforms: r2c R[0] -> CX[0] ; c2r CX[0] -> R[0]
    c->zT = (int)Z.size();
    zj(R[0], 0, nullptr, 0, CX[1], nullptr);
    zj(CY[0], MUL_NONE, nullptr, 0, R[0], nullptr);
    c->jTf_y = (int)J.size();
    aj(CX[1], CY[1], MUL_NONE);
    c->jTf_x = (int)J.size();
    aj(CY[1], CX[0], MUL_NONE);
    c->jT_x = (int)J.size();
    aj(CX[0], CX[1], MUL_NONE);
    c->jT_y = (int)J.size();
    aj(CX[1], CY[0], MUL_NONE);
    // diagnostics: c2r of the state (Y) -> R[20..23]
    c->jG_x = (int)J.size();
    for (int q = 0; q < 4; ++q) aj(c->Y[q], CX[q], MUL_NONE);
    c->jG_y = (int)J.size();
    for (int q = 0; q < 4; ++q) aj(CX[q], CY[q], MUL_NONE);
    c->zG = (int)Z.size();
    zj(CY[0], MUL_NONE, CY[1], MUL_NONE, R[20], R[21]);
    zj(CY[2], MUL_NONE, CY[3], MUL_NONE, R[22], R[23]);
    if (c->stretched) {
        void **SX = c->SX;
        // D': raw derivatives c2r(P i k_d F) of u'_c (R[4+3c+d], with U_c in
        // R[1+c]), of s (R[13+d]; its x and y passes are round A's) and of F1
        // (in CX[10]; R[16+d])
        c->jS_Dx = (int)J.size();
        for (int q = 0; q < 3; ++q) {
            aj(c->Ys[q], CX[2 + 2 * q], MUL_P);
            aj(c->Ys[q], CX[3 + 2 * q], MUL_P_IK);
        }
        aj(CX[10], CX[8], MUL_P);
        aj(CX[10], CX[9], MUL_P_IK);
        c->jS_Dy = (int)J.size();
        for (int q = 0; q < 3; ++q) {
            aj(CX[2 + 2 * q], CY[3 + 3 * q], MUL_NONE);
            aj(CX[2 + 2 * q], CY[4 + 3 * q], MUL_IK);
            aj(CX[3 + 2 * q], CY[5 + 3 * q], MUL_NONE);
        }
        aj(CX[8], CY[12], MUL_NONE);
        aj(CX[8], CY[13], MUL_IK);
        aj(CX[9], CY[14], MUL_NONE);
        c->zS_D = (int)Z.size();
        for (int q = 0; q < 3; ++q) {
            zj(CY[3 + 3 * q], MUL_NONE, CY[3 + 3 * q], MUL_IK, R[1 + q], R[4 + 3 * q + 2]);
            zj(CY[4 + 3 * q], MUL_NONE, CY[5 + 3 * q], MUL_NONE, R[4 + 3 * q + 1], R[4 + 3 * q + 0]);
        }
        zj(CY[1], MUL_NONE, CY[2], MUL_NONE, R[14], R[13]);
        zj(CY[0], MUL_IK, nullptr, 0, R[15], nullptr);
        zj(CY[14], MUL_NONE, CY[13], MUL_NONE, R[16], R[17]);
        zj(CY[12], MUL_IK, nullptr, 0, R[18], nullptr);
        // G': the 12 scaled derivatives R[4..15], filtered (k_x_filter between the y passes)
        c->zS_F = (int)Z.size();
        for (int j = 0; j < 12; j += 2) zj(R[4 + j], 0, R[5 + j], 0, CY[j], CY[j + 1]);
        c->jS_Fy = (int)J.size();
        for (int j = 0; j < 12; ++j) aj(CY[j], SX[j], MUL_NONE);
        c->jS_Gx = (int)J.size();
        for (int j = 0; j < 12; ++j) aj(SX[j], CY[j], MUL_NONE);
        c->jS_Gy = (int)J.size();
        for (int j = 0; j < 12; ++j) aj(CY[j], SX[j], MUL_NONE);
        c->zS_G = (int)Z.size();
        for (int j = 0; j < 12; j += 2) zj(SX[j], MUL_NONE, SX[j + 1], MUL_NONE, R[4 + j], R[5 + j]);
    }
    c->hj = J;
    c->hz = Z;
    c->dj = dalloc<AxisJob>(c, sizeof(AxisJob) * J.size());
    c->dz = dalloc<ZJob>(c, sizeof(ZJob) * Z.size());
    CK(cudaMemcpy(c->dj, J.data(), sizeof(AxisJob) * J.size(), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(c->dz, Z.data(), sizeof(ZJob) * Z.size(), cudaMemcpyHostToDevice));
}

void create(kf_ctx *c) {
    const kf_config &cf = c->cfg;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) throw KfError{KF_ERR_NO_DEVICE, "no CUDA device"};
    int dev = 0;
    CK(cudaGetDevice(&dev));
    cudaDeviceProp prop;
    CK(cudaGetDeviceProperties(&prop, dev));
    if (prop.major != 10) throw KfError{KF_ERR_NO_DEVICE, "this library targets sm_100a (B200)"};
    if (cf.precision != KF_FP64 && cf.precision != KF_FP32_BULK) throw KfError{KF_ERR_ARG, "precision"};
    if (cf.pen_eta > 0.) throw KfError{KF_ERR_ARG, "penalization damping must be <= 0 (effect_penalization.cpp:7-12)"};
    if (!(cf.L > 0.) || !(cf.theta != 0.)) throw KfError{KF_ERR_ARG, "L > 0 and theta != 0 required"};
    if (!(cf.stretch_m >= 0.) || !(2. * acos(-1.) * cf.stretch_m < cf.L))
        throw KfError{KF_ERR_ARG, "stretch_m must satisfy 0 <= 2 pi m < L (a monotone axis_CoSiSt map)"};
    if (!(cf.mg_omega >= 0.) || !(cf.mg_omega < 2.))
        throw KfError{KF_ERR_ARG, "mg_omega must lie in [0, 2) (0: the plain Newton step)"};
    c->stretched = cf.stretch_m != 0.;
    c->fp32 = cf.precision == KF_FP32_BULK;
    c->es = c->fp32 ? 4 : 8;
    c->cs = 2 * c->es;
    c->n = cf.n;
    c->nzc = cf.n / 2 + 1;
    c->N = (long)cf.n * cf.n * cf.n;
    c->Nc = (long)cf.n * cf.n * c->nzc;
    bool ok = c->fp32 ? Dispatch<float>::pick(c) : Dispatch<double>::pick(c);
    if (!ok) throw KfError{KF_ERR_ARG, "grid size must be one of 16, 32, 64, 96, 128, 256"};
    CK(cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking));
    c->own_stream = true;
    CK(cudaStreamCreateWithFlags(&c->st_body, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&c->st_side, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&c->ev_fork, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&c->ev_join, cudaEventDisableTiming));
    const size_t cb = c->cs * c->Nc, rb = c->es * c->N;
    for (int q = 0; q < 4; ++q) {
        c->Y[q] = dalloc<void>(c, cb);
        c->Ys[q] = dalloc<void>(c, cb);
        c->ACC[q] = dalloc<void>(c, cb);
        c->K[q] = dalloc<void>(c, cb);
        c->LIN[q] = dalloc<void>(c, cb);
    }
    for (int i = 0; i < 12; ++i) c->CX[i] = dalloc<void>(c, cb);
    for (int i = 0; i < 16; ++i) c->CY[i] = dalloc<void>(c, cb);
    for (int i = 0; i < 24; ++i) c->R[i] = dalloc<void>(c, rb);
    if (c->stretched)
        for (int i = 0; i < 12; ++i) c->SX[i] = dalloc<void>(c, cb);
    c->phihat = dalloc<void>(c, cb);
    c->phi = dalloc<double>(c, 8 * c->N);
    c->rho = dalloc<double>(c, 8 * c->N);
    c->nd = dalloc<double>(c, 8 * c->N);
    c->H = dalloc<void>(c, rb);
    c->stage64 = dalloc<double>(c, (size_t)16 * (c->Nc > c->N ? c->Nc : c->N));
    CK(cudaMemset(c->phi, 0, 8 * c->N));
    CK(cudaMemset(c->rho, 0, 8 * c->N));
    CK(cudaMemset(c->nd, 0, 8 * c->N));
    CK(cudaMemset(c->H, 0, rb));
    for (int q = 0; q < 4; ++q) {
        CK(cudaMemset(c->Y[q], 0, cb));
        CK(cudaMemset(c->Ys[q], 0, cb));
        CK(cudaMemset(c->K[q], 0, cb));  // k_xfwd_stage writes only what the 2/3 rule keeps
    }
    c->npartial = 1184;
    c->partial = dalloc<double>(c, sizeof(double) * KF_RED * c->npartial);
    c->red = dalloc<double>(c, sizeof(double) * 8);
    c->d_sweeps = dalloc<int>(c, sizeof(int) * 4);
    c->d_box = dalloc<int>(c, sizeof(int) * 4);
    CK(cudaMemset(c->d_box, 0xff, sizeof(int) * 4));  // max i = -1: no row
    c->d_err = dalloc<int>(c, sizeof(int));
    CK(cudaMemset(c->d_err, 0, sizeof(int)));
    CK(cudaMallocHost(&c->h_err, sizeof(int)));
    c->d_max = dalloc<unsigned long long>(c, 64 * sizeof(unsigned long long));
    CK(cudaMallocHost(&c->h_max, 64 * sizeof(unsigned long long)));
    if (cf.phi_extrap) c->phi_a = dalloc<double>(c, 8 * c->N);
    CK(cudaMallocHost(&c->h_red, sizeof(double) * 8));
    c->d_js = dalloc<JacState>(c, 2 * sizeof(JacState));
    for (auto &q : c->jc_part) {
        q = dalloc<JcStat>(c, 592 * sizeof(JcStat));
        CK(cudaMemset(q, 0, 592 * sizeof(JcStat)));
    }
    CK(cudaMallocHost(&c->h_js, sizeof(JacState)));
    CK(cudaMallocHost(&c->h_pois, sizeof(DevPois)));
    c->dtime = dalloc<DevTime>(c, sizeof(DevTime));
    c->dpois = dalloc<DevPois>(c, sizeof(DevPois));
    CK(cudaMemset(c->dtime, 0, sizeof(DevTime)));
    CK(cudaMemset(c->dpois, 0, sizeof(DevPois)));
    build_tables(c);
    build_levels(c);
    build_jobs(c);
    CK(cudaDeviceSynchronize());
}

// The caller's host arrays to and from the device, on c->st
void put_host(kf_ctx *c, void *dst, const void *src, size_t bytes) { CK(c->pipe.copy(dst, src, bytes, true, c->st)); }
void get_host(kf_ctx *c, void *dst, const void *src, size_t bytes) { CK(c->pipe.copy(dst, src, bytes, false, c->st)); }

// H2D of a host FP64 array of `count` doubles into a bulk-precision device array
void put_bulk(kf_ctx *c, void *dst, const double *src, long count) {
    if (!c->fp32) {
        put_host(c, dst, src, 8 * count);
    } else {
        put_host(c, c->stage64, src, 8 * count);
        Launch L_(c, KC_MISC, 12. * count);
        k_from_f64<float><<<nblk(count, 256), 256, 0, c->st>>>((float *)dst, c->stage64, count);
    }
}

void get_bulk(kf_ctx *c, double *dst, const void *src, long count) {
    if (!c->fp32) {
        get_host(c, dst, src, 8 * count);
    } else {
        {
            Launch L_(c, KC_MISC, 12. * count);
            k_to_f64<float><<<nblk(count, 256), 256, 0, c->st>>>(c->stage64, (const float *)src, count);
        }
        get_host(c, dst, c->stage64, 8 * count);
    }
}

void copy_state(kf_ctx *c, void *const *dst, void *const *src) {
    for (int q = 0; q < 4; ++q)
        CK(cudaMemcpyAsync(dst[q], src[q], c->cs * c->Nc, cudaMemcpyDeviceToDevice, c->st));
}

// One stage: the right-hand side of Ys and the stage's combination, in the
// right-hand side's last kernel.
void rk_stage(kf_ctx *c, double cdt, int mode) {
    c->rk_mode = mode;
    c->rk_c = cdt;
    try {
        c->rhs_fn(c);
    } catch (...) {
        c->rk_mode = 3;
        throw;
    }
    c->rk_mode = 3;
}

// One RK4 step (RKO4.cpp:105-238) on Y (== Ys on entry).  Optional hooks of
// the adjoint: X (16 buffers) receives the four stage inputs, PH (4) the four
// stage potentials; with PHin the stage potentials are taken from there and
// no Poisson problem is solved.
void rk4_step(kf_ctx *c, double dt, void *const *X, double *const *PH, double *const *PHin) {
    const double t0 = c->t;
    const double ts[4] = {t0, t0 + 0.5 * dt, t0 + 0.5 * dt, t0 + 1.0 * dt};
    const double cdt[4] = {0.5 * dt, 0.5 * dt, 1.0 * dt, dt / 6.};
    const int mode[4] = {0, 1, 1, 2};
    static const char *const kStage[4] = {"kf RK4 stage 1", "kf RK4 stage 2", "kf RK4 stage 3", "kf RK4 stage 4"};
    for (int i = 0; i < 4; ++i) {
        NvtxRange nv(kStage[i]);
        c->t_stage = ts[i];
        c->stage_idx = i;
        if (X) copy_state(c, X + 4 * i, c->Ys);
        if (PHin) {
            CK(cudaMemcpyAsync(c->phi, PHin[i], 8 * c->N, cudaMemcpyDeviceToDevice, c->st));
            c->phi_given = true;
        }
        rk_stage(c, cdt[i], mode[i]);
        c->phi_given = false;
        if (PH) CK(cudaMemcpyAsync(PH[i], c->phi, 8 * c->N, cudaMemcpyDeviceToDevice, c->st));
    }
    c->t = t0 + dt;
}

// Whether kf_rk4_steps replays a captured step graph: FAS or no Poisson solve (the
// Jacobi and cascadic solves, graphs of their own, are launched from the host).
bool graph_path(kf_ctx *c) {
    const kf_config &cf = c->cfg;
    if (host_driven(c)) return false;
    const bool pois = (cf.terms & T_POISSON) && (cf.terms & T_E_INT);
    return !pois || cf.poisson_mode == KF_PS_FAS;
}

// Capture one RK4 step (the sequence of rk4_step) with device-side stage
// times, warm starts and convergence loops; with wait_u, stage 1 waits for
// ev_u after its Poisson solve.
void capture_step(kf_ctx *c, double dt, bool wait_u, cudaGraphExec_t *out);

void build_step_graph(kf_ctx *c, double dt, bool with_wait = false) {
    if (c->step_graph && c->step_dt != dt) {
        cudaGraphExecDestroy(c->step_graph);
        c->step_graph = nullptr;
        if (c->step_graph_wait) cudaGraphExecDestroy(c->step_graph_wait);
        c->step_graph_wait = nullptr;
    }
    if (!c->step_graph) capture_step(c, dt, false, &c->step_graph);
    if (with_wait && !c->step_graph_wait) capture_step(c, dt, true, &c->step_graph_wait);
    c->step_dt = dt;
}

void capture_step(kf_ctx *c, double dt, bool wait_u, cudaGraphExec_t *out) {
    const double xs[4] = {0., 0.5 * dt, 0.5 * dt, 1.0 * dt};
    const double cdt[4] = {0.5 * dt, 0.5 * dt, 1.0 * dt, dt / 6.};
    const int mode[4] = {0, 1, 1, 2};
    const kf_config &cf = c->cfg;
    const bool pois = (cf.terms & T_POISSON) && (cf.terms & T_E_INT);
    const long long l0 = c->launches;
    c->cycle_kernels = 0;
    c->capturing = true;
    c->capture_wait_u = wait_u;
    CK(cudaStreamBeginCapture(c->st, cudaStreamCaptureModeThreadLocal));
    try {
        for (int i = 0; i < 4; ++i) {
            if (!(pois && cf.phi_extrap)) {  // else with the solve's history (k_hist_post)
                Launch L_(c, KC_MISC, 0.);
                k_time<<<1, 32, 0, c->st>>>(c->dtime, xs[i], 0);
            }
            c->stage_idx = i;
            c->stage_x = xs[i];
            rk_stage(c, cdt[i], mode[i]);
        }
        {
            Launch L_(c, KC_MISC, 0.);
            k_time<<<1, 32, 0, c->st>>>(c->dtime, dt, 1);
        }
    } catch (...) {
        cudaGraph_t g = nullptr;
        cudaStreamEndCapture(c->st, &g);
        if (g) cudaGraphDestroy(g);
        c->capturing = false;
        c->capture_wait_u = false;
        c->launches = l0;
        throw;
    }
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(c->st, &g);
    c->capturing = false;
    c->capture_wait_u = false;
    CK(e);
    e = cudaGraphInstantiate(out, g, 0);
    cudaGraphDestroy(g);
    CK(e);
    c->step_kernels = c->launches - l0 - (pois ? 4 * c->cycle_kernels : 0);
    c->launches = l0;
}

// nsteps replays of the step graph; the host's time and warm-start record is
// handed to the device before and read back after, with the solve statistics.
void graph_begin(kf_ctx *c, double dt) {
    build_step_graph(c, dt);
    DevTime ht{c->t, c->t_stage, c->tau_a, c->tau_b, c->nhist, 0, 0, 0};
    CK(cudaMemcpyAsync(c->dtime, &ht, sizeof(DevTime), cudaMemcpyHostToDevice, c->st));
}

void graph_step(kf_ctx *c) {
    NvtxRange nv("kf RK4 step (captured graph)");
    CK(cudaGraphLaunch(c->step_graph, c->st));
    c->launches += c->step_kernels;
}

void graph_end(kf_ctx *c) {
    DevTime ht;
    DevPois hp;
    CK(cudaMemcpyAsync(&ht, c->dtime, sizeof(DevTime), cudaMemcpyDeviceToHost, c->st));
    CK(cudaMemcpyAsync(&hp, c->dpois, sizeof(DevPois), cudaMemcpyDeviceToHost, c->st));
    kerr_fetch(c);
    CK(cudaStreamSynchronize(c->st));
    kerr_check(c);
    c->t = ht.t;
    c->t_stage = ht.t_stage;
    c->tau_a = ht.tau_a;
    c->tau_b = ht.tau_b;
    c->nhist = ht.nhist;
    const DevPois &o = c->hpois;
    c->launches += (hp.total_cycles - o.total_cycles) * c->cycle_kernels;
    c->diag.solves += hp.solves - o.solves;
    c->diag.total_iterations += hp.total_cycles - o.total_cycles;
    if (hp.solves != o.solves) {
        c->diag.last_iterations = hp.last_cycles;
        c->diag.last_residual = hp.last_residual;
    }
    c->diag.not_converged += hp.not_converged - o.not_converged;
    for (int s = 0; s < 4; ++s) c->diag.stage_cycles[s] += hp.stage_cycles[s] - o.stage_cycles[s];
    const bool nan = hp.nans != o.nans, nc = hp.not_converged != o.not_converged;
    c->hpois = hp;
    if (nan) throw KfError{KF_ERR_NAN, "NaN in the multigrid solve"};
    if (nc) throw KfError{KF_ERR_NOT_CONVERGED, "Poisson solve did not reach its tolerance"};
}

void rk4_steps_graph(kf_ctx *c, int nsteps, double dt) {
    graph_begin(c, dt);
    for (int s = 0; s < nsteps; ++s) graph_step(c);
    graph_end(c);
}

// interface_ode_solver::solve with the state in host arrays, in place: the
// upload of s goes first on the compute stream; u' is uploaded on a copy
// stream while stage 1's Poisson solve runs (the captured step of the first
// step waits for it just before it needs u'); the result is copied back.  That
// order hides the upload for page-locked arrays; a pageable u' holds the host until
// it is staged, before the step is launched.
void step_host(kf_ctx *c, int nsteps, double dt, double *const *host) {
    if (!c->st_copy) {
        CK(cudaStreamCreateWithFlags(&c->st_copy, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&c->ev_u, cudaEventDisableTiming));
        if (c->fp32) c->stage64b = dalloc<double>(c, 16 * (size_t)c->Nc);
    }
    build_step_graph(c, dt, true);
    put_bulk(c, c->Y[3], host[3], 2 * c->Nc);
    CK(cudaMemcpyAsync(c->Ys[3], c->Y[3], c->cs * c->Nc, cudaMemcpyDeviceToDevice, c->st));
    for (int q = 0; q < 3; ++q) {
        if (!c->fp32) {
            CK(cudaMemcpyAsync(c->Y[q], host[q], 16 * c->Nc, cudaMemcpyHostToDevice, c->st_copy));
        } else {
            CK(cudaMemcpyAsync(c->stage64b, host[q], 16 * c->Nc, cudaMemcpyHostToDevice, c->st_copy));
            const long M = 2 * c->Nc;
            Launch L_(c, KC_MISC, 12. * M);
            k_from_f64<float><<<nblk(M, 256), 256, 0, c->st_copy>>>((float *)c->Y[q], c->stage64b, M);
        }
        CK(cudaMemcpyAsync(c->Ys[q], c->Y[q], c->cs * c->Nc, cudaMemcpyDeviceToDevice, c->st_copy));
    }
    CK(cudaEventRecord(c->ev_u, c->st_copy));
    c->nhist = 0;  // as kf_set_state
    DevTime ht{c->t, c->t_stage, c->tau_a, c->tau_b, c->nhist, 0, 0, 0};
    CK(cudaMemcpyAsync(c->dtime, &ht, sizeof(DevTime), cudaMemcpyHostToDevice, c->st));
    CK(cudaGraphLaunch(c->step_graph_wait, c->st));
    c->launches += c->step_kernels;
    for (int s = 1; s < nsteps; ++s) graph_step(c);
    graph_end(c);
    for (int q = 0; q < 4; ++q) get_bulk(c, host[q], c->Y[q], 2 * c->Nc);
    CK(cudaStreamSynchronize(c->st));
}

template <typename F> int guarded(kf_ctx *c, F f) {
    if (!c) return KF_ERR_ARG;
    try {
        f();
        return KF_OK;
    } catch (const KfError &e) {
        c->err = e.msg;
        return e.code;
    } catch (const std::exception &e) {
        c->err = e.what();
        return KF_ERR_ARG;
    }
}

}  // namespace

#include "kf_adjoint_host.cuh"
#include "kf_driver.cuh"

namespace {

// Captured graphs hold the kernel variants they were captured with; dropped
// when the variants change and rebuilt by their next use.
void drop_graphs(kf_ctx *c) {
    CK(cudaStreamSynchronize(c->st));
    if (c->step_graph) cudaGraphExecDestroy(c->step_graph);
    c->step_graph = nullptr;
    if (c->step_graph_wait) cudaGraphExecDestroy(c->step_graph_wait);
    c->step_graph_wait = nullptr;
    if (c->vgraph) cudaGraphExecDestroy(c->vgraph);
    c->vgraph = nullptr;
    if (c->solve_graph) cudaGraphExecDestroy(c->solve_graph);
    c->solve_graph = nullptr;
    if (c->adj && c->adj->graph) {
        cudaGraphExecDestroy(c->adj->graph);
        c->adj->graph = nullptr;
    }
}

// The mask's window of rows (RowBox), with its size for the profile's bytes
void mask_box(kf_ctx *c) {
    const int n = c->n;
    int b[4] = {n, -1, n, -1};
    CK(cudaMemcpyAsync(c->d_box, b, sizeof(b), cudaMemcpyHostToDevice, c->st));
    {
        Launch L_(c, KC_MISC, (double)c->N * c->es);
        const dim3 g(1, (n + 7) / 8, n);
        if (c->fp32)
            k_mask_box<float><<<g, mg_block(), 0, c->st>>>((const float *)c->H, n, c->d_box);
        else
            k_mask_box<double><<<g, mg_block(), 0, c->st>>>((const double *)c->H, n, c->d_box);
    }
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(b, c->d_box, sizeof(b), cudaMemcpyDeviceToHost, c->st));
    CK(cudaStreamSynchronize(c->st));
    c->bx_i = b[1] >= 0 ? b[1] - b[0] + 1 : 0;
    c->bx_j = b[1] >= 0 ? b[3] - b[2] + 1 : 0;
}

// milliseconds per call of f: two untimed calls, then reps calls between
// CUDA events on the context's stream
template <typename F> double time_candidate(kf_ctx *c, int reps, F f) {
    cudaEvent_t a = nullptr, b = nullptr;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    float ms = 0.f;
    cudaError_t e = cudaSuccess;
    try {
        f();
        f();
        CK(cudaEventRecord(a, c->st));
        for (int r = 0; r < reps; ++r) f();
        CK(cudaEventRecord(b, c->st));
        CK(cudaEventSynchronize(b));
        e = cudaEventElapsedTime(&ms, a, b);
    } catch (...) {
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        throw;
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    CK(e);
    return (double)ms / reps;
}

void autotune(kf_ctx *c, int reps, kf_tune_out *o) {
    if (c->capturing) throw KfError{KF_ERR_ARG, "kf_autotune during a capture"};
    kf_tune_out r{};
    plan_info(c->n, r.fft_radices, r.fft_threads);
    // transform plans: the right-hand side with the potential held writes
    // only scratch arrays and K (the stage derivative, consumed within a step)
    const bool pg = c->phi_given;
    const int si = c->stage_idx, fv = c->fftv, by = c->rbgs_by;
    c->phi_given = true;
    c->stage_idx = 0;
    try {
        for (int v = 0; v < 2; ++v) {
            c->fftv = v;
            copy_state(c, c->Ys, c->Y);
            r.fft_ms[v] = time_candidate(c, reps, [&] { c->rhs_fn(c); });
        }
    } catch (...) {
        c->phi_given = pg;
        c->stage_idx = si;
        c->fftv = fv;
        throw;
    }
    c->phi_given = pg;
    c->stage_idx = si;
    r.fft_plan = r.fft_ms[1] < r.fft_ms[0] ? 1 : 0;
    // smoother shapes: sweeps of a copy of the finest-level potential
    // (rows 0: the streaming k_rbgs_march where the level allows it)
    const int rows[4] = {4, 8, 16, 0};
    r.rbgs_rows = by;
    if (c->rho && !c->lv.empty()) {
        LevelBuf &L0 = c->lv[0];
        double *tmp = nullptr;
        CK(cudaMalloc(&tmp, 8 * (size_t)c->N));
        try {
            // the last solve's source in both orders (a captured solve leaves it in
            // split order only, one with the streaming smoother in natural order)
            if (split_on(c, 0))
                unsplit_field(c, c->rho_cs, c->rho);
            else if (c->rho_cs)
                split_field(c, c->rho, c->rho_cs);
            int best = -1;
            for (int k = 0; k < 4; ++k) {
                c->rbgs_by = rows[k];
                if (rows[k] == 0 && !march_ok(c, L0)) {
                    r.rbgs_ms[k] = -1.;
                    continue;
                }
                const bool sp = split_on(c, 0);
                if (sp)
                    split_field(c, c->phi, tmp);
                else
                    CK(cudaMemcpyAsync(tmp, c->phi, 8 * (size_t)c->N, cudaMemcpyDeviceToDevice, c->st));
                r.rbgs_ms[k] = 0.5 * time_candidate(c, reps, [&] {
                                   if (sp)
                                       smooth_split(c, L0, tmp, c->rho_cs, 2, KC_RBGS);
                                   else
                                       smooth(c, L0, tmp, c->rho, nullptr, 2, KC_RBGS);
                               });
                if (best < 0 || r.rbgs_ms[k] < r.rbgs_ms[best]) best = k;
            }
            r.rbgs_rows = rows[best];
        } catch (...) {
            c->rbgs_by = by;
            c->fftv = fv;
            cudaStreamSynchronize(c->st);
            cudaFree(tmp);
            throw;
        }
        CK(cudaStreamSynchronize(c->st));
        CK(cudaFree(tmp));
    }
    c->fftv = r.fft_plan;
    c->rbgs_by = r.rbgs_rows;
    drop_graphs(c);
    if (o) *o = r;
}

}  // namespace

// Message of the last failure that has no context (kf_ctx_create and the
// context-free entry points); kf_last_error(NULL) returns it.
std::string &kf_global_error() {
    static thread_local std::string s;
    return s;
}

extern "C" {

int kf_ctx_create(const kf_config *cfg, kf_ctx **out) {
    if (!cfg || !out) return KF_ERR_ARG;
    kf_ctx *c = new kf_ctx;
    c->cfg = *cfg;
    int rc = guarded(c, [&] { create(c); });
    if (rc) {
        kf_global_error() = c->err;
        kf_ctx_destroy(c);
        *out = nullptr;
        return rc;
    }
    *out = c;
    return KF_OK;
}

int kf_ctx_destroy(kf_ctx *c) {
    if (!c) return KF_ERR_ARG;
    if (c->st) cudaStreamSynchronize(c->st);
    for (auto &r : c->recs) {
        cudaEventDestroy(r.a);
        cudaEventDestroy(r.b);
    }
    for (auto e : c->evfree) cudaEventDestroy(e);
    if (c->vgraph) cudaGraphExecDestroy(c->vgraph);
    if (c->solve_graph) cudaGraphExecDestroy(c->solve_graph);
    if (c->step_graph) cudaGraphExecDestroy(c->step_graph);
    if (c->step_graph_wait) cudaGraphExecDestroy(c->step_graph_wait);
    if (c->ev_u) cudaEventDestroy(c->ev_u);
    if (c->st_copy) cudaStreamDestroy(c->st_copy);
    if (c->st_body) cudaStreamDestroy(c->st_body);
    if (c->st_side) cudaStreamDestroy(c->st_side);
    if (c->ev_fork) cudaEventDestroy(c->ev_fork);
    if (c->ev_join) cudaEventDestroy(c->ev_join);
    adj_release(c);
    out_release(c);
    for (void *p : c->allocs) cudaFree(p);
    for (auto &g : c->jac) cudaGraphExecDestroy(g.exec);
    if (c->h_js) cudaFreeHost(c->h_js);
    if (c->h_pois) cudaFreeHost(c->h_pois);
    if (c->h_red) cudaFreeHost(c->h_red);
    if (c->h_max) cudaFreeHost(c->h_max);
    if (c->h_err) cudaFreeHost(c->h_err);
    if (c->st && c->own_stream) cudaStreamDestroy(c->st);
    delete c;
    return KF_OK;
}

const char *kf_last_error(const kf_ctx *c) { return c ? c->err.c_str() : kf_global_error().c_str(); }

int kf_set_stream(kf_ctx *c, void *stream) {
    return guarded(c, [&] {
        CK(cudaStreamSynchronize(c->st));
        if (c->own_stream) CK(cudaStreamDestroy(c->st));
        if (stream) {
            c->st = (cudaStream_t)stream;
            c->own_stream = false;
        } else {
            CK(cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking));
            c->own_stream = true;
        }
    });
}

int kf_synchronize(kf_ctx *c) {
    return guarded(c, [&] { CK(cudaStreamSynchronize(c->st)); CK(cudaGetLastError()); });
}

int kf_set_state(kf_ctx *c, const double *ux, const double *uy, const double *uz, const double *s) {
    return guarded(c, [&] {
        if (!ux || !uy || !uz || !s) throw KfError{KF_ERR_ARG, "null state array"};
        const double *src[4] = {ux, uy, uz, s};
        for (int q = 0; q < 4; ++q) put_bulk(c, c->Y[q], src[q], 2 * c->Nc);
        copy_state(c, c->Ys, c->Y);
        c->nhist = 0;
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_get_state(kf_ctx *c, double *ux, double *uy, double *uz, double *s) {
    return guarded(c, [&] {
        double *dst[4] = {ux, uy, uz, s};
        for (int q = 0; q < 4; ++q)
            if (dst[q]) get_bulk(c, dst[q], c->Y[q], 2 * c->Nc);
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_set_sources(kf_ctx *c, const double *nd, const double *mask) {
    return guarded(c, [&] {
        if (nd) put_host(c, c->nd, nd, 8 * c->N);
        if (mask) {
            put_bulk(c, c->H, mask, c->N);
            mask_box(c);
        }
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_set_phi(kf_ctx *c, const double *phi) {
    return guarded(c, [&] {
        put_host(c, c->phi, phi, 8 * c->N);
        c->nhist = 0;
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_get_phi(kf_ctx *c, double *phi) {
    return guarded(c, [&] {
        get_host(c, phi, c->phi, 8 * c->N);
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_rhs_eval(kf_ctx *c, double t) {
    return guarded(c, [&] {
        c->t_stage = t;  // selects the start of the Poisson solve only
        c->stage_idx = 0;
        copy_state(c, c->Ys, c->Y);
        c->rhs_fn(c);
        copy_state(c, c->Y, c->K);
        copy_state(c, c->Ys, c->K);
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_step_host(kf_ctx *c, int nsteps, double dt, double *ux, double *uy, double *uz, double *s) {
    return guarded(c, [&] {
        if (!ux || !uy || !uz || !s) throw KfError{KF_ERR_ARG, "null state array"};
        if (nsteps < 0) throw KfError{KF_ERR_ARG, "nsteps < 0"};
        double *host[4] = {ux, uy, uz, s};
        if (nsteps > 0 && graph_path(c)) {
            step_host(c, nsteps, dt, host);
            return;
        }
        for (int q = 0; q < 4; ++q) put_bulk(c, c->Y[q], host[q], 2 * c->Nc);
        copy_state(c, c->Ys, c->Y);
        c->nhist = 0;
        for (int k = 0; k < nsteps; ++k) rk4_step(c, dt, nullptr, nullptr, nullptr);
        for (int q = 0; q < 4; ++q) get_bulk(c, host[q], c->Y[q], 2 * c->Nc);
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_rk4_steps(kf_ctx *c, int nsteps, double dt) {
    return guarded(c, [&] {
        if (nsteps < 0) throw KfError{KF_ERR_ARG, "nsteps < 0"};
        // Ys == Y on entry; stage times t, t + dt/2, t + dt/2, t + dt (RKO4.cpp:105-212)
        if (nsteps > 0 && graph_path(c)) {
            rk4_steps_graph(c, nsteps, dt);
            return;
        }
        for (int s = 0; s < nsteps; ++s) rk4_step(c, dt, nullptr, nullptr, nullptr);
        CK(cudaGetLastError());
    });
}

int kf_autotune(kf_ctx *c, int reps, kf_tune_out *out) {
    return guarded(c, [&] { autotune(c, reps > 0 ? reps : 5, out); });
}

int kf_set_tuning(kf_ctx *c, int fft_plan, int rbgs_rows) {
    return guarded(c, [&] {
        if ((fft_plan != 0 && fft_plan != 1) ||
            (rbgs_rows != 0 && rbgs_rows != 4 && rbgs_rows != 8 && rbgs_rows != 16))
            throw KfError{KF_ERR_ARG, "kf_set_tuning: fft_plan 0 or 1, rbgs_rows 0, 4, 8 or 16"};
        if (c->capturing) throw KfError{KF_ERR_ARG, "kf_set_tuning during a capture"};
        const bool changed = fft_plan != c->fftv || rbgs_rows != c->rbgs_by;
        c->fftv = fft_plan;
        c->rbgs_by = rbgs_rows;
        if (changed) drop_graphs(c);
    });
}

int kf_set_coarse_block(kf_ctx *c, int on) {
    return guarded(c, [&] {
        if (on != 0 && on != 1) throw KfError{KF_ERR_ARG, "kf_set_coarse_block: on is 0 or 1"};
        if (c->capturing) throw KfError{KF_ERR_ARG, "kf_set_coarse_block during a capture"};
        if (c->coarse_block == (on == 1)) return;
        c->coarse_block = on == 1;
        cc_setup(c);
        drop_graphs(c);
    });
}

int kf_set_overlap(kf_ctx *c, int on) {
    return guarded(c, [&] {
        if (on != 0 && on != 1) throw KfError{KF_ERR_ARG, "kf_set_overlap: on is 0 or 1"};
        if (c->capturing) throw KfError{KF_ERR_ARG, "kf_set_overlap during a capture"};
        if (c->overlap_d == (on == 1)) return;
        c->overlap_d = on == 1;
        drop_graphs(c);
    });
}

int kf_batch_rk4_steps(kf_ctx *const *ctxs, int nctx, int nsteps, const double *dts) {
    if (!ctxs || !dts || nctx < 0 || nsteps < 0) {
        kf_global_error() = "kf_batch_rk4_steps: invalid argument";
        return KF_ERR_ARG;
    }
    for (int i = 0; i < nctx; ++i) {
        if (!ctxs[i]) {
            kf_global_error() = "kf_batch_rk4_steps: null context";
            return KF_ERR_ARG;
        }
        if (!graph_path(ctxs[i])) {
            ctxs[i]->err = "kf_batch_rk4_steps needs a context whose step can be captured "
                           "(KF_PS_FAS or no Poisson solve, profile off)";
            kf_global_error() = ctxs[i]->err;
            return KF_ERR_ARG;
        }
    }
    int rc = KF_OK;
    std::vector<char> begun(nctx, 0);
    for (int i = 0; i < nctx && rc == KF_OK; ++i) {
        rc = guarded(ctxs[i], [&] { graph_begin(ctxs[i], dts[i]); });
        begun[i] = rc == KF_OK;
        if (rc != KF_OK) kf_global_error() = ctxs[i]->err;
    }
    // step-major: every instance's step s is queued before any step s + 1
    for (int s = 0; s < nsteps && rc == KF_OK; ++s)
        for (int i = 0; i < nctx && rc == KF_OK; ++i) {
            rc = guarded(ctxs[i], [&] { graph_step(ctxs[i]); });
            if (rc != KF_OK) kf_global_error() = ctxs[i]->err;
        }
    for (int i = 0; i < nctx; ++i) {
        if (!begun[i]) continue;
        const int r = guarded(ctxs[i], [&] { graph_end(ctxs[i]); });
        if (r != KF_OK && rc == KF_OK) {
            rc = r;
            kf_global_error() = ctxs[i]->err;
        }
    }
    return rc;
}

int kf_poisson_solve_to(kf_ctx *c, const double *phi0, const double *rho, double *phi) {
    return guarded(c, [&] {
        if (!phi0 || !rho || !phi) throw KfError{KF_ERR_ARG, "null array"};
        put_host(c, c->phi, phi0, 8 * c->N);
        put_host(c, c->rho, rho, 8 * c->N);
        int r = poisson(c);
        get_host(c, phi, c->phi, 8 * c->N);
        CK(cudaStreamSynchronize(c->st));
        if (r) throw KfError{KF_ERR_NOT_CONVERGED, "Poisson solve did not reach its tolerance"};
    });
}

int kf_poisson_solve(kf_ctx *c, double *phi_io, const double *rho) { return kf_poisson_solve_to(c, phi_io, rho, phi_io); }

int kf_diag(kf_ctx *c, kf_diag_out *out) {
    return guarded(c, [&] {
        if (!out) throw KfError{KF_ERR_ARG, "null output"};
        c->inv_state_fn(c);
        const int nb = red_blocks(c->N);
        Launch L_(c, KC_MISC, (double)c->N * (4 * c->es + 16));
        if (c->fp32)
            k_diag_sums<float><<<nb, RBS, 0, c->st>>>((const float *)c->R[23], (const float *)c->R[20],
                                                     (const float *)c->R[21], (const float *)c->R[22], c->phi, c->nd,
                                                     c->cfg.M, c->N, c->partial, c->vol, c->n);
        else
            k_diag_sums<double><<<nb, RBS, 0, c->st>>>((const double *)c->R[23], (const double *)c->R[20],
                                                      (const double *)c->R[21], (const double *)c->R[22], c->phi,
                                                      c->nd, c->cfg.M, c->N, c->partial, c->vol, c->n);
        k_diag_final<<<1, 32, 0, c->st>>>(c->partial, nb, c->red);
        c->launches++;
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(c->h_red, c->red, sizeof(double) * 2, cudaMemcpyDeviceToHost, c->st));
        CK(cudaStreamSynchronize(c->st));
        const double h = c->cfg.L / c->n, h3 = h * h * h;
        *out = c->diag;
        out->kinetic = c->h_red[0] * h3;
        out->charge = c->h_red[1] * h3;
    });
}

int kf_fft_r2c(kf_ctx *c, const double *in, double *out) {
    return guarded(c, [&] {
        put_bulk(c, c->R[0], in, c->N);
        c->r2c_fn(c);
        get_bulk(c, out, c->CX[0], 2 * c->Nc);
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_fft_c2r(kf_ctx *c, const double *in, double *out) {
    return guarded(c, [&] {
        put_bulk(c, c->CX[0], in, 2 * c->Nc);
        c->c2r_fn(c);
        get_bulk(c, out, c->R[0], c->N);
        CK(cudaStreamSynchronize(c->st));
    });
}

int kf_state_device_ptrs(kf_ctx *c, void **ux, void **uy, void **uz, void **s) {
    return guarded(c, [&] {
        void **o[4] = {ux, uy, uz, s};
        for (int q = 0; q < 4; ++q)
            if (o[q]) *o[q] = c->Y[q];
    });
}

long long kf_launch_count(const kf_ctx *c) { return c ? c->launches : -1; }

int kf_profile_enable(kf_ctx *c, int on) {
    return guarded(c, [&] {
        prof_flush(c);
        for (int k = 0; k < KC_N; ++k) {
            c->prof_ms[k] = 0.;
            c->prof_bytes[k] = 0.;
            c->prof_n[k] = 0;
        }
        c->prof = on != 0;
    });
}

int kf_profile_read(kf_ctx *c, int cls, double *ms, long long *launches, double *bytes) {
    return guarded(c, [&] {
        if (cls < 0 || cls >= KC_N) throw KfError{KF_ERR_ARG, "kernel class out of range"};
        prof_flush(c);
        if (ms) *ms = c->prof_ms[cls];
        if (launches) *launches = c->prof_n[cls];
        if (bytes) *bytes = c->prof_bytes[cls];
    });
}

const char *kf_profile_class_name(int cls) { return (cls >= 0 && cls < KC_N) ? kKClsName[cls] : ""; }

}  // extern "C"
