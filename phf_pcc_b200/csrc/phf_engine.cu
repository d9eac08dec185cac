// Plan, grid-point pipeline and C ABI of the projected-HF grid kernel.
//
// The reference (PHF_fort/PHFTools.f90:84-170) loops over grid points w = (il, iy, ipg) and,
// per point, forms R = Ref^H R1 R2 Rpg Ref (five M^3 products), the M x M transition density
// rho_w, the dense O(M^4) MakeGamma, and M^3 gradient products.  This engine instead runs
// chunks of b grid points through a fixed sequence of batched kernels, keeping every
// per-point quantity in the rank-N form (M x N, never M x M except where the dense
// two-electron operator needs vec(rho)):
//
//   Y_w  = R_w ket                          R applied to the N occupied columns only
//   S_w  = bra^H Y_w ; S_w^-1, det, logdet  FP64 Gauss-Jordan, one CTA per point
//   X_w  = Y_w S_w^-1                       rho_w = X_w bra^H
//   HX_w = H1 X_w ; e1_w = tr(bra^H HX_w)   one-electron energy tr(H1 rho)
//   GX_w = Gamma(rho_w) X_w                 dense: Gamma = H2r vec(rho); Cholesky: T = V^H X,
//                                           T' = tr(T) 1 - T, Q = X T', GX = sum_L B_L Q_L
//   e2_w = 1/2 tr(Gamma rho)                dense: tr(bra^H GX)/2; Cholesky: sum_L (d^2 - tr T^2)/2
//   W_w  = bra^H (HX_w + GX_w)
//   Yg_w = N_w [(HX + GX - X W) + h_w X],   Yr_w = N_w X_w,   h_w = e1 + e2   (Gradient :291-308)
//   acc_a += sum_w Wt[a, w] (N h, N, Yg, Yr)   Wigner x character x spin weights (:120-166)
//
// and at the end Gradmat_a = Yg_a bra^H, Rdmmat_a = Yr_a bra^H (Ref-MO basis).
// In the Cholesky form the spin-orbital index runs in the interleaved order r' = 2p + sigma
// so that B_L (x) I_2 acts on plain row-major blocks.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <limits>
#include <memory>
#include <string>
#include <vector>

#include <cublas_v2.h>

#include "phf_common.cuh"
#include <mutex>

#include "phf_internal.h"

namespace phf {

unsigned long long g_launches = 0;
int g_narrow_mma = 0;
int g_fx_i8 = 1;

// Whether a tensor-core plan forms its densities (and F X) by int8 slice products: n > 64 with up to seven slices, but
// in the residue form from n > 128 only.  Up to there the FP64 products are the faster ones, without slicing passes
// over X, the densities and Gamma: an evaluation at n = 72 (112 points) takes 0.62 against 0.68 ms, n = 101 (156
// points) 1.53 against 1.61, n = 128 (800 points) 11.8 against 12.2; n = 150 (156 points) 11.46 against 11.34.
static bool density_i8(const PlanImpl &p) {
    return !oz_rho_slice_ok(p.n) && p.slices <= 7 && !(p.rz && p.n <= 128);
}

// ---------------------------------------------------------------- per-class event timing
namespace {
struct ProfState {
    bool on = false;
    std::vector<cudaEvent_t> ev;       // pairs (start, end)
    std::vector<int> cls;              // class of each recorded pair
    size_t used = 0;
};
ProfState g_prof;
thread_local int t_prof_class = PROF_GEMM;
}  // namespace

void prof_set_class(int c) { t_prof_class = c; }
int prof_class() { return t_prof_class; }

ProfScope::ProfScope(cudaStream_t s, int c) : st(s), slot(-1) {
    if (!g_prof.on) return;
    if (g_prof.used * 2 + 2 > g_prof.ev.size()) {
        for (int i = 0; i < 512; ++i) {
            cudaEvent_t e;
            if (cudaEventCreate(&e) != cudaSuccess) return;
            g_prof.ev.push_back(e);
        }
    }
    slot = (int)g_prof.used++;
    if ((int)g_prof.cls.size() <= slot) g_prof.cls.resize(slot + 1);
    g_prof.cls[slot] = (c < 0) ? t_prof_class : c;
    cudaEventRecord(g_prof.ev[2 * slot], st);
}

ProfScope::~ProfScope() {
    if (slot >= 0) cudaEventRecord(g_prof.ev[2 * slot + 1], st);
}

int profile_enable(int on) {
    g_prof.on = on != 0;
    g_prof.used = 0;
    return PHF_OK;
}

int profile_read(int c, double *ms, unsigned long long *count) {
    double tot = 0.0;
    unsigned long long n = 0;
    for (size_t i = 0; i < g_prof.used; ++i) {
        if (g_prof.cls[i] != c) continue;
        float t = 0.f;
        cudaEventSynchronize(g_prof.ev[2 * i + 1]);
        if (cudaEventElapsedTime(&t, g_prof.ev[2 * i], g_prof.ev[2 * i + 1]) == cudaSuccess) tot += t;
        ++n;
    }
    if (ms) *ms = tot;
    if (count) *count = n;
    return PHF_OK;
}

// ---------------------------------------------------------------- memory of one-shot calls
namespace {
constexpr size_t kPoolKeep = (size_t)16 << 30;
constexpr int kPoolDevices = 64;
std::mutex g_pool_mu;
cudaMemPool_t g_pools[kPoolDevices] = {};  // one per device, created at first use, kept until exit

cudaMemPool_t current_pool(bool create) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kPoolDevices) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (!g_pools[dev] && create) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        unsigned long long keep = kPoolKeep;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        g_pools[dev] = pool;
    }
    return g_pools[dev];
}
}  // namespace

cudaError_t pool_alloc(void **p, size_t bytes) {
    cudaMemPool_t pool = current_pool(true);
    if (!pool) return cudaErrorMemoryAllocation;
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, 0);
    if (e == cudaErrorMemoryAllocation) {  // give back what is kept and try once more
        cudaGetLastError();
        pool_release();
        e = cudaMallocFromPoolAsync(p, bytes, pool, 0);
    }
    return e;
}

void pool_free(void *p) { cudaFreeAsync(p, 0); }

namespace {
// bytes held by the pool and in use of it (no pool: zero)
void pool_bytes(cudaMemPool_t pool, size_t &held, size_t &used) {
    unsigned long long h = 0, u = 0;
    if (pool) {
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &h);
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &u);
    }
    held = (size_t)h;
    used = (size_t)std::min(u, h);
}
}  // namespace

size_t pool_kept_bytes() {
    size_t held, used;
    pool_bytes(current_pool(false), held, used);
    return held - used;
}

void pool_release() {
    cudaMemPool_t pool = current_pool(false);
    if (!pool) return;
    cudaStreamSynchronize(0);  // frees that are queued there
    cudaMemPoolTrimTo(pool, 0);
}

void pool_trim() {
    cudaMemPool_t pool = current_pool(false);
    size_t fr = 0, tot = 0, held, used;
    if (!pool || cudaMemGetInfo(&fr, &tot) != cudaSuccess) return;
    pool_bytes(pool, held, used);
    // keep at most half of what would be free without the kept part
    const size_t keep = std::min(kPoolKeep, (fr + (held - used)) / 2);
    if (held - used > keep) {
        cudaStreamSynchronize(0);
        cudaMemPoolTrimTo(pool, used + keep);
    }
}

static thread_local std::string t_last_error;
static thread_local int t_last_status = PHF_OK;

void set_error(int status, const std::string &msg) {
    t_last_status = status;
    t_last_error = msg;
}
int last_status() { return t_last_status; }
std::string &last_error_string() { return t_last_error; }

namespace {



inline View vz(const void *p, long long rs, long long cs, long long bs0 = 0, long long bs1 = 0, int conj = 0) {
    View v;
    v.p = p;
    v.rs = rs;
    v.cs = cs;
    v.bs0 = bs0;
    v.bs1 = bs1;
    v.conj = conj;
    v.real = 0;
    return v;
}
inline View vd(const void *p, long long rs, long long cs, long long bs0 = 0, long long bs1 = 0) {
    View v = vz(p, rs, cs, bs0, bs1, 0);
    v.real = 1;
    return v;
}
inline OutView vo(zc *p, long long rs, long long cs, long long bs0 = 0, long long bs1 = 0) {
    OutView o;
    o.p = p;
    o.rs = rs;
    o.cs = cs;
    o.bs0 = bs0;
    o.bs1 = bs1;
    return o;
}

const zc Z1{1.0, 0.0}, Z0{0.0, 0.0}, ZM1{-1.0, 0.0};

double wigner_small_d(int j, int n, int m, double beta) {
    auto fact = [](int k) {
        double r = 1.0;
        for (int i = 2; i <= k; ++i) r *= i;
        return r;
    };
    double pre = std::sqrt(fact(j + n) * fact(j - n) * fact(j + m) * fact(j - m));
    int smax = std::min(j + m, j - n), smin = std::max(0, m - n);
    double acc = 0.0;
    for (int s = smin; s <= smax; ++s) {
        int p1 = n - m + s, p2 = 2 * j + m - n - 2 * s, p3 = n - m + 2 * s;
        double num = ((p1 & 1) ? -1.0 : 1.0) * std::pow(std::cos(beta / 2), p2) * std::pow(std::sin(beta / 2), p3);
        acc += num / (fact(j + m - s) * fact(s) * fact(n - m + s) * fact(j - n - s));
    }
    return pre * acc;
}

// Wignerfac (PHF_fort/PHFTools.f90:350-376)
cd wignerfac(int j, int n, int m, double a, double b, double g) {
    return std::exp(cd(0.0, -n * a)) * wigner_small_d(j, n, m, b) * std::exp(cd(0.0, -m * g));
}

}  // namespace

namespace {

int check_device(int *dev) {
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0) {
        cudaGetLastError();
        set_error(PHF_ERR_NO_DEVICE, "no CUDA device available");
        return PHF_ERR_NO_DEVICE;
    }
    PHF_CUDA(cudaGetDevice(dev));
    return PHF_OK;
}

// complex128 Fortran array element
inline cd fz(const phf_complex *a, size_t idx) { return cd(a[idx].re, a[idx].im); }

int upload(zc *dst, const std::vector<cd> &src) {
    PHF_CUDA(cudaMemcpy(dst, src.data(), src.size() * sizeof(zc), cudaMemcpyHostToDevice));
    return PHF_OK;
}

int validate(const phf_plan_desc *d) {
    if (!d || d->nso <= 0 || d->nocc <= 0 || d->nocc > d->nso || !d->ngrid || d->ngrid[0] <= 0 || d->ngrid[1] <= 0 ||
        d->npg <= 0 || d->ncisp <= 0 || d->ncipg <= 0 || d->qj < 0 || !d->ref || !d->r1 || !d->r2 || !d->rpg ||
        !d->weightsp || !d->weightpg || !d->roota || !d->rootb || !d->rooty) {
        set_error(PHF_ERR_ARG, "missing or non-positive plan argument");
        return PHF_ERR_ARG;
    }
    const int ncik = d->cmplxconj == 2 ? 2 : 1;
    if (d->cmplxconj < 0 || d->cmplxconj > 2) {
        set_error(PHF_ERR_ARG, "cmplxconj must be 0, 1 or 2");
        return PHF_ERR_ARG;
    }
    if (d->nci != d->ncisp * d->ncipg * ncik) {
        set_error(PHF_ERR_ARG, "nci != ncisp * ncipg * ncik");
        return PHF_ERR_ARG;
    }
    if (d->ncisp != 2 * d->qj + 1) {
        set_error(PHF_ERR_ARG, "ncisp must equal 2*qj + 1 (Wigner slots ni, nj = -qj..qj)");
        return PHF_ERR_ARG;
    }
    if (d->nchol > 0) {
        if (!d->h || !d->bvec || (d->nso & 1)) {
            set_error(PHF_ERR_ARG, "Cholesky form needs h, bvec and an even nso");
            return PHF_ERR_ARG;
        }
    } else if (!d->hone || !d->htwo) {
        set_error(PHF_ERR_ARG, "dense form needs hone and htwo");
        return PHF_ERR_ARG;
    }
    if (d->nocc > kMaxOverlapN) {
        set_error(PHF_ERR_UNSUPPORTED, "nocc > " + std::to_string(kMaxOverlapN) +
                                           " (the overlap inverse keeps the N x N matrix in shared memory)");
        return PHF_ERR_UNSUPPORTED;
    }
    if (d->precision < PHF_PREC_FP64 || d->precision > PHF_PREC_TF32) {
        set_error(PHF_ERR_ARG, "unknown precision");
        return PHF_ERR_ARG;
    }
    if (d->precision != PHF_PREC_FP64 && d->nchol <= 0) {
        set_error(PHF_ERR_UNSUPPORTED, "tensor-core precisions are implemented for the Cholesky form");
        return PHF_ERR_UNSUPPORTED;
    }
    if (d->gradient_mode < 0 || d->gradient_mode > 1) {
        set_error(PHF_ERR_ARG, "gradient_mode must be 0 or 1");
        return PHF_ERR_ARG;
    }
    if (d->gradient_mode == 1 && (d->nchol <= 0 || d->jk_form == 2 || d->nci != 1 || d->cmplxconj == 2)) {
        set_error(PHF_ERR_UNSUPPORTED,
                  "the exact gradient needs an exchange-matrix form (stored or streamed), nci == 1 and cmplxconj 0/1");
        return PHF_ERR_UNSUPPORTED;
    }
    if (d->jk_form < 0 || d->jk_form > 3) {
        set_error(PHF_ERR_ARG, "jk_form must be 0, 1, 2 or 3");
        return PHF_ERR_ARG;
    }
    if (d->exchange_panel < 0) {
        set_error(PHF_ERR_ARG, "exchange_panel must be >= 0");
        return PHF_ERR_ARG;
    }
    if (d->exchange_symmetry < 0 || d->exchange_symmetry > 2) {
        set_error(PHF_ERR_ARG, "exchange_symmetry must be 0, 1 or 2");
        return PHF_ERR_ARG;
    }
    return PHF_OK;
}

}  // namespace

namespace {
int build_exchange_matrix(PlanImpl &p);
constexpr int kDSplit = 4;  // split-k of the Coulomb GEMM d = B vec P (small output, k = n^2)

// Spatial indices i per exchange panel of the streamed form: panels of at most 8192 exchange rows
// (i, k), with the fewest padded rows over all panels (GEMM tiles are 128 rows), ties to the larger
// panel (fewer launches).  n = 200: 32 (6 panels of 6400 rows and one of 1600).
int choose_ipanel(int n) {
    int best = 1;
    long long best_rows = -1;
    for (int I = 1; I <= n && (long long)I * n <= std::max<long long>(8192, n); ++I) {
        const long long full = n / I, rest = n % I;
        const long long rows = full * oz_pad_rows((long long)I * n) + (rest ? oz_pad_rows(rest * n) : 0);
        if (best_rows < 0 || rows <= best_rows) {
            best_rows = rows;
            best = I;
        }
    }
    return best;
}
}  // namespace

namespace {
// Residues of the products of a chunk of b points: of one exchange product over `points` of them (all, or equal parts
// of at most 1 GiB, whole 256-row tiles) and of the larger of the Coulomb products.  Returned: a bound of the bytes that
// does not fall as b grows.
struct RzScratch {
    long long points;
    size_t c, cj;
};
size_t rz_scratch(const PlanImpl &p, long long b, RzScratch *out) {
    const size_t tile = rz_product_bytes(2 * kRzModuli, 1, p.rz_rows);
    const long long groups = (b + 31) / 32, cap = std::max<long long>(1, (long long)(((size_t)1 << 30) / tile));
    const auto coulomb = [&](long long points) {
        return std::max(rz_product_bytes(kRzModuli, 2 * points, p.rz_rows), rz_product_bytes(kRzModuli, 2 * b, p.L));
    };
    if (out) {
        const long long parts = (groups + cap - 1) / cap;
        out->points = std::min(b, 32 * ((groups + parts - 1) / parts));
        out->c = rz_product_bytes(2 * kRzModuli, 8 * out->points, p.rz_rows);
        out->cj = coulomb(out->points);
    }
    const long long most = std::min(groups, cap);
    return tile * (size_t)most + coulomb(32 * most);
}

// f(B[p][q], B[q][p]) over the pairs of one vector until it returns false (16 x 16 tiles, so that both sides stay in cache)
template <typename F>
bool over_pairs(const double *B, int n, F &&f) {
    const int T = 16;
    for (int q0 = 0; q0 < n; q0 += T)
        for (int p0 = 0; p0 <= q0; p0 += T)
            for (int q = q0; q < std::min(q0 + T, n); ++q)
                for (int p = p0; p < std::min(p0 + T, q); ++p)
                    if (!f(B[p + (size_t)n * q], B[q + (size_t)n * p])) return false;
    return true;
}

// How the Cholesky vectors compare with their transposes: 2 = every B_L is exactly symmetric, 1 = to rounding,
// 0 = neither (or not finite).  To rounding: no difference above 2 sqrt(n) units in the last place of the largest
// element of B_L.  Vectors brought to another basis, X^T B X, are sums of n products on either side and differ by
// 2 (n = 5), 6 (64), 8 (128) and 10 (200) such units; a difference of that size says nothing about the integrals,
// and the full rows of vectors that are not symmetric cost twice the exchange work.
int cholesky_symmetry(const phf_plan_desc *d) {
    const int n = d->nso / 2;
    int level = 2;
    for (int l = 0; l < d->nchol; ++l) {
        const double *B = d->bvec + (size_t)n * n * l;
        if (over_pairs(B, n, [](double a, double b) { return a == b; })) continue;
        double mx = 0.0;
        for (size_t e = 0; e < (size_t)n * n; ++e) mx = std::max(mx, std::fabs(B[e]));
        const double limit = 2.0 * std::sqrt((double)n) * std::numeric_limits<double>::epsilon() * mx;
        if (!std::isfinite(limit) || !over_pairs(B, n, [=](double a, double b) { return std::fabs(a - b) <= limit; }))
            return 0;
        level = 1;
    }
    return level;
}
}  // namespace

int plan_create(const phf_plan_desc *d, phf_plan **out, bool one_shot) {
    *out = nullptr;
    PHF_TRY(validate(d));
    auto P = std::make_unique<phf_plan>();
    PlanImpl &p = P->impl;
    p.arena.pooled = one_shot;
    p.graphs_ok = !one_shot;  // a graph captured for one evaluation costs more than its launches
    PHF_TRY(check_device(&p.device));
    p.chol = d->nchol > 0;
    p.M = d->nso;
    p.n = d->nso / 2;
    p.N = d->nocc;
    p.L = d->nchol;
    p.prec = d->precision;
    // operand format of the tensor-core GEMMs: int8 slice count, or a floating-point format code
    p.slices = p.prec == PHF_PREC_BF16X3 ? OZ_FMT_BF16X3
             : p.prec == PHF_PREC_TF32  ? OZ_FMT_TF32
                                        : (d->slices > 0 ? d->slices : 5);
    // automatic form: the stored spatial-ERI exchange matrix for n <= 128 (n^4 doubles: 2.1 GB at
    // n = 128); above, the streamed form, which regenerates the exchange rows panel by panel from the
    // Cholesky vectors instead of holding the n^4 matrix (the factorized form has ~3L/(4n) times the
    // flops of either and is chosen only explicitly)
    if (p.chol) {
        const int form = d->jk_form != 0 ? d->jk_form : (d->nso / 2 <= 128 ? 1 : 3);
        p.eri = (form == 1 || form == 3);
        p.streamed = (form == 3);
    }
    p.exact = d->gradient_mode == 1;
    p.autotune = d->autotune != 0;
    p.library_gemm = (d->fp64_library_gemm != 0) && p.eri && p.prec == PHF_PREC_FP64;
    if (p.library_gemm) {
        cublasHandle_t h = nullptr;
        if (cublasCreate(&h) != CUBLAS_STATUS_SUCCESS) {
            set_error(PHF_ERR_CUDA, "cublasCreate failed");
            return PHF_ERR_CUDA;
        }
        p.cublas = h;
    }
    if (p.exact && !p.eri) {
        set_error(PHF_ERR_UNSUPPORTED, "the exact gradient needs an exchange-matrix form (jk_form 0, 1 or 3)");
        return PHF_ERR_UNSUPPORTED;
    }
    if (p.prec != PHF_PREC_FP64 && !p.eri) {
        set_error(PHF_ERR_UNSUPPORTED, "the tensor-core precisions need an exchange-matrix form (jk_form 0, 1 or 3)");
        return PHF_ERR_UNSUPPORTED;
    }
    // the exchange symmetry (n >= 2): the streamed form in FP64, and in the tensor-core forms whose densities
    // are sliced apart from the density GEMM (n > 64); the stored form in FP64 and int8 (residues, and slices with
    // n > 64).  All but the streamed FP64 form need symmetric Cholesky vectors: K(rho^T) = K(rho)^T holds for any
    // real vectors, their Coulomb term over pairs l <= j only for symmetric ones (vectors symmetric to rounding are
    // replaced by (B + B^T) / 2).  The full rows do twice the
    // exchange work: an evaluation takes 9.5 ms with them and 5.7 ms without (FP64, n = 64, 800 points),
    // 25.0 and 16.1 ms (int8, n = 128, 800 points), 5.3 and 4.4 ms (int8, n = 101, 312 points)
    const int symmetry = p.chol ? cholesky_symmetry(d) : 0;
    const bool symmetric = symmetry > 0;
    const bool sym_slices = p.prec == PHF_PREC_FP64 || !oz_rho_slice_ok(d->nso / 2);
    if (p.streamed) {
        const int n = d->nso / 2;
        p.ek_ipanel = d->exchange_panel > 0 ? std::min(d->exchange_panel, n) : choose_ipanel(n);
        p.ek_npanel = (n + p.ek_ipanel - 1) / p.ek_ipanel;
        const bool sym_ok = n >= 2 && n <= 65535 && sym_slices;
        if (d->exchange_symmetry == 1 && !sym_ok) {
            set_error(PHF_ERR_UNSUPPORTED, "exchange_symmetry needs the FP64 form or n > 64 (tensor-core forms)");
            return PHF_ERR_UNSUPPORTED;
        }
        // (the tensor-core forms contract the Coulomb term over the pairs l <= j, the FP64 form over all (l, j))
        p.ek_sym = sym_ok && d->exchange_symmetry != 2 && (p.prec == PHF_PREC_FP64 || symmetric);
        if (p.ek_sym) {
            // panels of indices i with Gram blocks (i n + l) x ((k >= i0) n + j) of at most ek_ipanel n x n^2
            const long long budget = (long long)p.ek_ipanel * n;
            p.ek_i0.clear();
            for (int i0 = 0; i0 < n;) {
                p.ek_i0.push_back(i0);
                i0 += (int)std::max<long long>(1, std::min<long long>(n - i0, budget / (n - i0)));
            }
            p.ek_i0.push_back(n);
            p.ek_npanel = (int)p.ek_i0.size() - 1;
        }
    } else if (p.eri) {
        const int n = d->nso / 2;
        p.ek_sym = n >= 2 && n <= 65535 && (sym_slices || (d->slices == 0 && rz_ok(n, d->nchol))) &&
                   d->exchange_symmetry != 2 && (p.prec == PHF_PREC_FP64 || p.prec == PHF_PREC_OZAKI_I8) && symmetric;
        if (p.ek_sym) p.ek_i0 = {0, n};  // one panel: every row, formed once at plan creation
        p.ek_npanel = 1;
    }
    p.rz = p.ek_sym && p.prec == PHF_PREC_OZAKI_I8 && d->slices == 0 && symmetric &&
           rz_ok(d->nso / 2, d->nchol);
    p.nl = d->ngrid[0];
    p.ny = d->ngrid[1];
    p.npg = d->npg;
    p.nomega = p.nl * p.ny * p.npg;
    p.wbeg = 0;
    p.wend = p.nomega;
    if (d->point_begin != 0 || d->point_end != 0) {
        if (d->point_begin < 0 || d->point_end > p.nomega || d->point_begin >= d->point_end) {
            set_error(PHF_ERR_ARG, "point range outside [0, number of grid points)");
            return PHF_ERR_ARG;
        }
        p.wbeg = d->point_begin;
        p.wend = d->point_end;
    }
    p.nci = d->nci;
    p.ncisp = d->ncisp;
    p.ncipg = d->ncipg;
    p.cmplxconj = d->cmplxconj;
    p.qj = d->qj;
    p.sp = d->sp;
    p.nb = p.ncisp * p.ncipg;
    const int M = p.M, N = p.N, n = p.n;
    const size_t MM = (size_t)M * M;

    // working order
    p.perm.resize(M);
    for (int r = 0; r < M; ++r) p.perm[r] = p.chol ? ((r & 1) * n + (r >> 1)) : r;
    std::vector<int> inv(M);
    for (int r = 0; r < M; ++r) inv[p.perm[r]] = r;

    // rotation matrices in working order, row-major
    auto rot = [&](const phf_complex *src, int cnt, zc **dst) -> int {
        PHF_TRY(p.arena.alloc(dst, (size_t)cnt * MM));
        std::vector<cd> h((size_t)cnt * MM);
        for (int g = 0; g < cnt; ++g)
            for (int i = 0; i < M; ++i)
                for (int j = 0; j < M; ++j)
                    h[(size_t)g * MM + (size_t)i * M + j] =
                        fz(src, (size_t)g + (size_t)cnt * ((size_t)p.perm[i] + (size_t)M * p.perm[j]));
        return upload(*dst, h);
    };
    // dense form: R acts in the reference AO order (Y is mapped to MO afterwards with Ref^H)
    PHF_TRY(rot(d->r1, p.nl, &p.R1));
    PHF_TRY(rot(d->r2, p.ny, &p.R2));
    PHF_TRY(rot(d->rpg, p.npg, &p.Rpg));
    // Cholesky forms: a spin rotation R1 is block diagonal in the interleaved order (one 2 x 2 block
    // per spatial orbital); when every R1[il] is exactly that, Y = R1 T2 needs two terms per element
    // instead of an M x M product (the dropped terms are exact zeros)
    if (p.chol) {
        std::vector<cd> blocks((size_t)p.nl * p.n * 4);
        bool spin_blocks = true;
        for (int g = 0; g < p.nl && spin_blocks; ++g)
            for (int i = 0; i < M && spin_blocks; ++i)
                for (int j = 0; j < M; ++j) {
                    const cd v = fz(d->r1, (size_t)g + (size_t)p.nl * ((size_t)p.perm[i] + (size_t)M * p.perm[j]));
                    if ((i >> 1) == (j >> 1)) {
                        blocks[((size_t)g * p.n + (i >> 1)) * 4 + 2 * (i & 1) + (j & 1)] = v;
                    } else if (v != cd(0, 0)) {
                        spin_blocks = false;
                        break;
                    }
                }
        if (spin_blocks) {
            PHF_TRY(p.arena.alloc(&p.R1b, blocks.size()));
            PHF_TRY(upload(p.R1b, blocks));
        }
    }

    // Ref (row-major, reference order kept on the host; rows in working order on the device)
    p.ref_host.resize(MM);
    for (int i = 0; i < M; ++i)
        for (int j = 0; j < M; ++j) p.ref_host[(size_t)i * M + j] = fz(d->ref, (size_t)i + (size_t)M * j);
    {
        std::vector<cd> rw(MM);
        for (int r = 0; r < M; ++r)
            for (int j = 0; j < M; ++j) rw[(size_t)r * M + j] = p.ref_host[(size_t)p.perm[r] * M + j];
        PHF_TRY(p.arena.alloc(&p.Refw, MM));
        PHF_TRY(upload(p.Refw, rw));
        if (p.chol) {  // Ref must be unitary for the AO-basis formulation
            double dev = 0.0;
            for (int i = 0; i < M; ++i)
                for (int j = 0; j < M; ++j) {
                    cd s = 0;
                    for (int k = 0; k < M; ++k) s += std::conj(p.ref_host[(size_t)k * M + i]) * p.ref_host[(size_t)k * M + j];
                    dev = std::max(dev, std::abs(s - cd(i == j ? 1.0 : 0.0)));
                }
            if (dev > 1e-8) {
                set_error(PHF_ERR_ARG, "Cholesky form needs a unitary Ref (max |Ref^H Ref - I| = " + std::to_string(dev) + ")");
                return PHF_ERR_ARG;
            }
        }
    }
    {  // [0, M): working -> reference index; [M, 2M): reference -> working index
        std::vector<int> both(2 * (size_t)M);
        for (int r = 0; r < M; ++r) {
            both[r] = p.perm[r];
            both[M + r] = inv[r];
        }
        PHF_TRY(p.arena.alloc(&p.permdev, 2 * (size_t)M));
        PHF_CUDA(cudaMemcpy(p.permdev, both.data(), 2 * (size_t)M * sizeof(int), cudaMemcpyHostToDevice));
    }

    // weight table Wt[s, w], s = m + nb n over the base block, w = (il ny + iy) npg + ipg
    {
        const int nb = p.nb, nw = p.nomega;
        std::vector<cd> Wt((size_t)nb * nb * nw, cd(0, 0));
        const int qj = p.qj;
        for (int il = 0; il < p.nl; ++il)
            for (int iy = 0; iy < p.ny; ++iy)
                for (int ig = 0; ig < p.npg; ++ig) {
                    const int w = (il * p.ny + iy) * p.npg + ig;
                    const double wsp = d->weightsp[(size_t)il + (size_t)p.nl * iy];
                    for (int ni = -qj; ni <= qj; ++ni)
                        for (int nj = -qj; nj <= qj; ++nj) {
                            cd wig = (p.sp == 2) ? wignerfac(qj, ni, nj, d->roota[il], d->rootb[iy], d->rooty[il])
                                                 : wignerfac(qj, ni, nj, d->roota[il], d->rootb[il], d->rooty[iy]);
                            for (int pp = 0; pp < p.ncipg; ++pp)
                                for (int q = 0; q < p.ncipg; ++q) {
                                    double wpg = d->weightpg[(size_t)ig + (size_t)p.npg * ((size_t)pp + (size_t)p.ncipg * q)];
                                    int m = ni + qj + pp * p.ncisp, nn = nj + qj + q * p.ncisp;
                                    Wt[(size_t)(m + nb * nn) * nw + w] += wsp * wpg * wig;
                                }
                        }
                }
        PHF_TRY(p.arena.alloc(&p.Wt, Wt.size()));
        PHF_TRY(upload(p.Wt, Wt));
        // slot maps of the four (bra, ket) variants (PHFTools.f90:149-162)
        std::vector<int> sm(4 * (size_t)nb * nb);
        const int dm[4] = {0, 0, 1, 1}, dn[4] = {0, 1, 1, 0};
        for (int v = 0; v < 4; ++v)
            for (int m = 0; m < nb; ++m)
                for (int nn = 0; nn < nb; ++nn)
                    sm[(size_t)v * nb * nb + m + nb * nn] = (m + dm[v] * nb) + p.nci * (nn + dn[v] * nb);
        PHF_TRY(p.arena.alloc(&p.slotmap, sm.size()));
        PHF_CUDA(cudaMemcpy(p.slotmap, sm.data(), sm.size() * sizeof(int), cudaMemcpyHostToDevice));
        // GEMM offsets of Y_w = R1[il] T2[iy, ig]
        std::vector<long long> offs(3 * (size_t)nw);
        for (int w = 0; w < nw; ++w) {
            int il = w / (p.ny * p.npg), rem = w % (p.ny * p.npg);
            offs[3 * w] = (long long)il * MM;
            offs[3 * w + 1] = (long long)rem * N;  // column block of T2 (M x ny npg N)
            offs[3 * w + 2] = 0;
        }
        PHF_TRY(p.arena.alloc(&p.offs, offs.size()));
        PHF_CUDA(cudaMemcpy(p.offs, offs.data(), offs.size() * sizeof(long long), cudaMemcpyHostToDevice));
        if (d->gradient_mode == 1) {  // R1[il]^H, R2[iy]^H, Rpg[ig]^H per point
            std::vector<long long> ok(9 * (size_t)nw, 0);
            for (int w = 0; w < nw; ++w) {
                const int il = w / (p.ny * p.npg), iy = (w / p.npg) % p.ny, ig = w % p.npg;
                ok[3 * ((size_t)0 * nw + w)] = (long long)il * MM;
                ok[3 * ((size_t)1 * nw + w)] = (long long)iy * MM;
                ok[3 * ((size_t)2 * nw + w)] = (long long)ig * MM;
            }
            PHF_TRY(p.arena.alloc(&p.offs_k, ok.size()));
            PHF_CUDA(cudaMemcpy(p.offs_k, ok.data(), ok.size() * sizeof(long long), cudaMemcpyHostToDevice));
        }
    }

    // Hamiltonian
    if (p.chol) {
        const int L = p.L;
        // exactly symmetric vectors need no transposition
        const bool as_given = symmetry == 2, mean = symmetry == 1 && p.ek_sym && !(p.streamed && p.prec == PHF_PREC_FP64);
        std::vector<double> hh((size_t)n * n), Bst(as_given ? 0 : (size_t)L * n * n);
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < n; ++j) hh[(size_t)i * n + j] = d->h[(size_t)i + (size_t)n * j];
        for (int l = 0; l < L && !as_given; ++l) {
            const double *B = d->bvec + (size_t)n * n * l;
            for (int pp = 0; pp < n; ++pp)
                for (int q = 0; q < n; ++q) {
                    const double a = B[(size_t)pp + (size_t)n * q];
                    Bst[((size_t)l * n + pp) * n + q] = mean ? 0.5 * a + 0.5 * B[(size_t)q + (size_t)n * pp] : a;
                }
        }
        PHF_TRY(p.arena.alloc(&p.h, hh.size()));
        PHF_TRY(p.arena.alloc(&p.Bst, (size_t)L * n * n));
        PHF_CUDA(cudaMemcpy(p.h, hh.data(), hh.size() * sizeof(double), cudaMemcpyHostToDevice));
        PHF_CUDA(cudaMemcpy(p.Bst, as_given ? d->bvec : Bst.data(), (size_t)L * n * n * sizeof(double),
                            cudaMemcpyHostToDevice));
        if (p.eri) PHF_TRY(build_exchange_matrix(p));
        // exchange-matrix forms: with h exactly symmetric (H1 = H1^H), H1 is added to Gamma where J is,
        // so one product gives F X = (H1 + J - K) X and e1 = tr(bra^H H1 X) = sum conj(H1 bra) X
        p.fold_h = p.eri;
        for (int i = 0; i < n && p.fold_h; ++i)
            for (int j = 0; j < i; ++j)
                if (hh[(size_t)i * n + j] != hh[(size_t)j * n + i]) {
                    p.fold_h = false;
                    break;
                }
    } else {
        std::vector<cd> h1(MM);
        for (int i = 0; i < M; ++i)
            for (int j = 0; j < M; ++j) h1[(size_t)i * M + j] = fz(d->hone, (size_t)i + (size_t)M * j);
        PHF_TRY(p.arena.alloc(&p.H1, MM));
        PHF_TRY(upload(p.H1, h1));
        zc *h2 = nullptr;
        PHF_TRY(p.arena.alloc(&p.H2r, MM * MM));
        PHF_TRY(p.arena.alloc(&h2, MM * MM));
        cudaError_t e = cudaMemcpy(h2, d->htwo, MM * MM * sizeof(zc), cudaMemcpyHostToDevice);
        int st = (e == cudaSuccess) ? launch_permute_h2(M, h2, p.H2r, 0) : PHF_ERR_CUDA;
        if (e == cudaSuccess && st == PHF_OK) e = cudaStreamSynchronize(0);
        p.arena.free_one(h2);
        if (e != cudaSuccess) {
            set_error(PHF_ERR_CUDA, std::string("uploading HTwo: ") + cudaGetErrorString(e));
            return PHF_ERR_CUDA;
        }
        PHF_TRY(st);
    }

    // per-evaluation buffers
    const size_t MN = (size_t)M * N;
    PHF_TRY(p.arena.alloc(&p.bra, MN));
    PHF_TRY(p.arena.alloc(&p.ket, MN));
    PHF_TRY(p.arena.alloc(&p.kety, MN));
    PHF_TRY(p.arena.alloc(&p.newmo, MN));
    PHF_TRY(p.arena.alloc(&p.newmoc, MN));
    PHF_TRY(p.arena.alloc(&p.T1, (size_t)p.npg * MN));
    PHF_TRY(p.arena.alloc(&p.T2, (size_t)p.ny * p.npg * MN));
    if (p.chol) PHF_TRY(p.arena.alloc(&p.V, (size_t)p.L * MN));
    const size_t nslot = (size_t)p.nci * p.nci;
    // the accumulators in one buffer, cleared by one launch: the sums, their compensations, the status word
    p.acc_bytes = ((size_t)(p.exact ? 8 : 4) * nslot * MN + 4 * nslot) * sizeof(zc) + sizeof(int);
    unsigned char *acc = nullptr;
    PHF_TRY(p.arena.alloc(&acc, p.acc_bytes));
    p.accG = reinterpret_cast<zc *>(acc);
    p.compG = p.accG + nslot * MN;
    p.accR = p.compG + nslot * MN;
    p.compR = p.accR + nslot * MN;
    zc *next = p.compR + nslot * MN;
    if (p.exact) {
        p.accKG = next;
        p.compKG = p.accKG + nslot * MN;
        p.accKR = p.compKG + nslot * MN;
        p.compKR = p.accKR + nslot * MN;
        next = p.compKR + nslot * MN;
    }
    p.accHS = next;
    p.compHS = p.accHS + 2 * nslot;
    p.flag = reinterpret_cast<int *>(p.compHS + 2 * nslot);
    PHF_TRY(p.arena.alloc(&p.tmpG, MN));
    PHF_TRY(p.arena.alloc(&p.outMM, 2 * nslot * MM));  // every slot's Gradmat and Rdmmat block
    if (p.exact || p.fold_h) PHF_TRY(p.arena.alloc(&p.Hb, MN));

    // chunk size from the workspace budget.  The streamed form regenerates its exchange rows once
    // per chunk (2 n^4 L flops against 16 n^4 per point), so by default it takes up to 45 % of the
    // free device memory to keep the chunk (and the regeneration's share, L / (8 b)) large.
    {
        size_t budget = d->workspace_bytes ? d->workspace_bytes : ((size_t)6 << 30);
        if (!d->workspace_bytes && p.streamed) {
            size_t fr = 0, tot = 0;
            if (cudaMemGetInfo(&fr, &tot) == cudaSuccess)  // (what is kept for one-shot calls can be had, too)
                budget = std::max(budget, (size_t)(0.45 * (double)(fr + pool_kept_bytes())));
            cudaGetLastError();
        }
        size_t per = 5 * MN + 3 * (size_t)N * N + 8;
        const size_t n2 = (size_t)n * n;
        if (p.chol && p.eri) {
            per += MM;                                          // Rho and Gam
            if (!p.rz) per += 2 * n2 + p.L;                     // Pvec, Jvec, dvec
            if (p.prec == PHF_PREC_FP64) per += 8 * n2;         // Kin, Kvec
            else if (p.rz)  // the operands (their products are counted below)
                per += (rz_operand_bytes(2 * kRzModuli, 8, n * (n + 1) / 2) + rz_operand_bytes(kRzModuli, 2, n * (n + 1) / 2) +
                        rz_operand_bytes(kRzModuli, 2, p.L)) / sizeof(zc) + 2;
            else per += (8 * (n2 + 64) * oz_slots(p.slices)) / sizeof(zc) + 1  // exchange slices
                        + (2 * n2 + 2 * (size_t)p.L) * oz_slots(p.slices) / sizeof(zc) + 1    // Coulomb slices
                        + p.L + n2;                                                // d^T, J pairs
            // int8 density GEMM: the X rows' slices and exponents
            if (p.prec != PHF_PREC_FP64 && density_i8(p)) {
                per += ((size_t)M * oz_pad_k(2LL * N) * oz_slots(p.slices) + 4 * (size_t)M) / sizeof(zc) + 1;
                // F X on the int8 path: the slices and exponents of X's columns and F's rows
                if (g_fx_i8 && oz_fx_ok(M, p.slices))
                    per += ((size_t)(2 * M + N) * oz_pad_k(2LL * M) * oz_slots(p.slices) + 4 * (size_t)(2 * M + N)) /
                               sizeof(zc) + 1;
            }
        } else if (p.chol) {
            per += (size_t)p.L * N * N + (size_t)p.L * MN + p.L;
        } else {
            per += 2 * MM;
        }
        if (p.exact) per += 5 * MN;
        per *= sizeof(zc);
        long long bmax = (long long)(budget / std::max<size_t>(per, 1));
        bmax = std::max<long long>(1, std::min<long long>(bmax, 4096));
        if (p.rz) {  // the largest chunk whose residue products fit too
            long long lo = 1, hi = bmax;
            while (lo < hi) {
                const long long mid = (lo + hi + 1) / 2;
                if (per * (size_t)mid + rz_scratch(p, mid, nullptr) <= budget) lo = mid;
                else hi = mid - 1;
            }
            bmax = lo;
        }
        p.b = (int)std::min<long long>(bmax, p.wend - p.wbeg);
        // whole Lebedev-point blocks (ny npg points sharing R1[il]) per chunk when they fit
        const int blk = p.ny * p.npg;
        if (p.b >= blk) p.b = (p.b / blk) * blk;
    }
    const size_t bMN = (size_t)p.b * MN, bNN = (size_t)p.b * N * N;
    PHF_TRY(p.arena.alloc(&p.Ys, bMN));
    if (!p.chol) PHF_TRY(p.arena.alloc(&p.Ys2, bMN));
    PHF_TRY(p.arena.alloc(&p.S, bNN));
    PHF_TRY(p.arena.alloc(&p.Sinv, bNN));
    PHF_TRY(p.arena.alloc(&p.W, bNN));
    PHF_TRY(p.arena.alloc(&p.Xs, bMN));
    if (p.exact) {
        PHF_TRY(p.arena.alloc(&p.Vk, bMN));
        PHF_TRY(p.arena.alloc(&p.Pk, bMN));
        PHF_TRY(p.arena.alloc(&p.Pk2, bMN));
        PHF_TRY(p.arena.alloc(&p.Prk, bMN));
        PHF_TRY(p.arena.alloc(&p.Prk2, bMN));
    }
    if (!p.fold_h) PHF_TRY(p.arena.alloc(&p.HX, bMN));
    PHF_TRY(p.arena.alloc(&p.GX, bMN));
    {
        unsigned char *sc = nullptr;
        PHF_TRY(p.arena.alloc(&sc, accumulate_scratch_bytes(p.nb * p.nb, M, N, p.b)));
        p.acc_scratch = sc;
    }
    PHF_TRY(p.arena.alloc(&p.det, p.b));
    PHF_TRY(p.arena.alloc(&p.logdet, p.b));
    PHF_TRY(p.arena.alloc(&p.e1, p.b));
    PHF_TRY(p.arena.alloc(&p.e2, p.b));
    if (p.chol && p.eri) {
        const size_t n2 = (size_t)n * n, b = (size_t)p.b;
        PHF_TRY(p.arena.alloc(&p.Gam, b * MM));
        p.Rho = p.Gam;  // the densities are gathered into the operands before Gamma is written
        if (!p.rz) {
            PHF_TRY(p.arena.alloc(&p.Pvec, b * n2));
            PHF_TRY(p.arena.alloc(&p.Jvec, b * n2));
            PHF_TRY(p.arena.alloc(&p.dvec, b * p.L));
        }
        if (p.prec == PHF_PREC_FP64) {
            PHF_TRY(p.arena.alloc(&p.Kin, 4 * b * n2));
            PHF_TRY(p.arena.alloc(&p.Kvec, 4 * b * n2));
        } else {
            if (p.rz) {
                const long long kk = (long long)n * (n + 1) / 2;
                PHF_TRY(p.arena.alloc(&p.rzK, rz_operand_bytes(2 * kRzModuli, 8LL * b, kk)));
                PHF_TRY(p.arena.alloc(&p.rzKe, 16 * b));
                PHF_TRY(p.arena.alloc(&p.rzP, rz_operand_bytes(kRzModuli, 2LL * b, kk)));
                PHF_TRY(p.arena.alloc(&p.rzPe, 2 * b));
                PHF_TRY(p.arena.alloc(&p.rzD, rz_operand_bytes(kRzModuli, 2LL * b, p.L)));
                PHF_TRY(p.arena.alloc(&p.rzDe, 2 * b));
                RzScratch sz;
                rz_scratch(p, p.b, &sz);
                p.rz_sub = (int)sz.points;
                PHF_TRY(p.arena.alloc(&p.rzC, sz.c));
                PHF_TRY(p.arena.alloc(&p.rzCJ, sz.cj));
            } else {
                const long long npadK = oz_pad_cols(8 * (long long)b);
                size_t bsl = oz_slice_bytes(npadK, (long long)n2, p.slices);
                if (p.ek_sym) {  // symmetric-half columns (k = n(n+1)/2), then the antisymmetric halves
                    p.bsl_a_off = oz_slice_bytes(npadK, (long long)n * (n + 1) / 2, p.slices);
                    bsl = std::max(bsl, p.bsl_a_off + oz_slice_bytes(npadK, (long long)n * (n - 1) / 2, p.slices));
                    PHF_TRY(p.arena.alloc(&p.eb_a, (size_t)npadK));
                }
                PHF_TRY(p.arena.alloc(&p.Bsl, bsl));
                PHF_CUDA(cudaMemset(p.Bsl, 0, bsl));
                PHF_TRY(p.arena.alloc(&p.eb, (size_t)npadK));
                const long long c2 = oz_pad_cols(2 * (long long)b);
                const size_t psl = oz_slice_bytes(c2, (long long)n2, p.slices);
                const size_t dsl = oz_slice_bytes(c2, p.L, p.slices);
                PHF_TRY(p.arena.alloc(&p.Psl, psl));
                PHF_TRY(p.arena.alloc(&p.dsl, dsl));
                PHF_CUDA(cudaMemset(p.Psl, 0, psl));
                PHF_CUDA(cudaMemset(p.dsl, 0, dsl));
                PHF_TRY(p.arena.alloc(&p.ePc, (size_t)c2));
                PHF_TRY(p.arena.alloc(&p.edc, (size_t)c2));
                PHF_TRY(p.arena.alloc(&p.dT, 2 * b * (size_t)p.L));
                PHF_TRY(p.arena.alloc(&p.dpart, (size_t)kDSplit * 2 * b * (size_t)p.L));
                PHF_TRY(p.arena.alloc(&p.Jr, 2 * b * n2));
            }
            // rho_w = X_w bra^H for the whole chunk as one int8 GEMM
            p.rho_i8 = density_i8(p);
            if (p.rho_i8) {
                const long long xrows = oz_pad_rows((long long)M * p.b), brows = oz_pad_cols(2LL * M);
                PHF_TRY(p.arena.alloc(&p.Xsl, oz_slice_bytes(xrows, 2LL * N, p.slices)));
                PHF_TRY(p.arena.alloc(&p.eX, (size_t)xrows));
                PHF_TRY(p.arena.alloc(&p.BRop, (size_t)2 * M * 2 * N));
                PHF_TRY(p.arena.alloc(&p.BRsl, oz_slice_bytes(brows, 2LL * N, p.slices)));
                PHF_TRY(p.arena.alloc(&p.eBR, (size_t)brows));
                PHF_CUDA(cudaMemset(p.Xsl, 0, oz_slice_bytes(xrows, 2LL * N, p.slices)));
                PHF_CUDA(cudaMemset(p.BRsl, 0, oz_slice_bytes(brows, 2LL * N, p.slices)));
            }
            // F X = (H1 + J - K) X on the int8 path too: its slices are part of the per-point workspace, so
            // one sub-batch takes the whole chunk (unless a cap is set for tests)
            p.fx_i8 = p.rho_i8 && g_fx_i8 && oz_fx_ok(M, p.slices);
            if (p.fx_i8) {
                p.fx_b = std::min(p.b, 65535);
                if (g_fx_i8 > 1) p.fx_b = std::min(p.fx_b, g_fx_i8);
                p.fx_a_rows = oz_pad_rows((long long)p.fx_b * N);
                p.fx_b_rows = oz_pad_cols(2LL * M * p.fx_b);
                const size_t xb = oz_slice_bytes(p.fx_a_rows, 2LL * M, p.slices);
                const size_t fb = oz_slice_bytes(p.fx_b_rows, 2LL * M, p.slices);
                PHF_TRY(p.arena.alloc(&p.XTsl, xb));
                PHF_TRY(p.arena.alloc(&p.FXsl, fb));
                PHF_TRY(p.arena.alloc(&p.eXT, (size_t)p.fx_a_rows));
                PHF_TRY(p.arena.alloc(&p.eFX, (size_t)p.fx_b_rows));
                PHF_CUDA(cudaMemset(p.XTsl, 0, xb));
                PHF_CUDA(cudaMemset(p.FXsl, 0, fb));
                PHF_CUDA(cudaMemset(p.eXT, 0, (size_t)p.fx_a_rows * sizeof(int)));
                PHF_CUDA(cudaMemset(p.eFX, 0, (size_t)p.fx_b_rows * sizeof(int)));
            }
        }
    } else if (p.chol) {
        PHF_TRY(p.arena.alloc(&p.T, (size_t)p.L * bNN));
        PHF_TRY(p.arena.alloc(&p.Q, (size_t)p.L * bMN));
        PHF_TRY(p.arena.alloc(&p.e2part, (size_t)p.L * p.b));
    } else {
        PHF_TRY(p.arena.alloc(&p.Pv, (size_t)p.b * MM));
        PHF_TRY(p.arena.alloc(&p.Gv, (size_t)p.b * MM));
    }
    *out = P.release();
    return PHF_OK;
}

namespace {

// EK[(i n + k) n^2 + (l n + j)] = sum_L B_L[i][l] B_L[k][j] = (il|kj): the exchange operator
// K(rho)_ik = sum_{lj} (il|jk) rho_lj as an n^2 x n^2 matrix acting on vec(rho) (built as n^2
// batched n x n x L products); sliced (int8 digits, BF16 pairs or TF32) for the tensor-core back-end.
// Coulomb operands of the tensor-core path: B (L x n^2, rows of Bst) and B^T (n^2 x L, strided rows of
// Bst).  B^T's slices are also both operands of the streamed form's Gram blocks.
// With the exchange symmetry the Coulomb contraction d_L = sum_lj B_L[l][j] P[l][j] runs over the pairs
// l <= j (B_L symmetric): B's rows hold B_L[l][j] (2 - delta_lj) in pair order and the density operand
// the symmetric half of P.
int build_coulomb_slices(PlanImpl &p) {
    const int n = p.n, L = p.L;
    if (p.rz) {  // residues over the pairs: B_L (2 - delta) (rows L) and B_L[pair] (rows pair)
        const long long kk = (long long)n * (n + 1) / 2;
        PHF_TRY(p.arena.alloc(&p.rzB1, rz_operand_bytes(kRzModuli, L, kk)));
        PHF_TRY(p.arena.alloc(&p.rzB1e, (size_t)L));
        PHF_TRY(p.arena.alloc(&p.rzB2, rz_operand_bytes(kRzModuli, kk, L)));
        PHF_TRY(p.arena.alloc(&p.rzB2e, (size_t)kk));
        double *Bp = nullptr;
        PHF_TRY(p.arena.alloc(&Bp, (size_t)(L * kk)));
        PHF_TRY(oz_cholesky_pairs(n, L, p.Bst, p.pairs_le, Bp, 0, 2.0));
        PHF_TRY(rz_rows(L, (int)kk, Bp, kk, 1, p.rzB1, p.rzB1e, 0));
        PHF_TRY(oz_cholesky_pairs(n, L, p.Bst, p.pairs_le, Bp, 0, 1.0));
        PHF_TRY(rz_rows(kk, L, Bp, 1, kk, p.rzB2, p.rzB2e, 0));
        PHF_CUDA(cudaDeviceSynchronize());
        p.arena.free_one(Bp);
        if (!p.streamed) return PHF_OK;
    }
    const long long n2 = (long long)n * n, kc = p.ek_sym ? (long long)n * (n + 1) / 2 : n2;
    const size_t b1 = oz_slice_bytes(oz_pad_rows(L), kc, p.slices);
    const size_t b2 = oz_slice_bytes(oz_pad_rows(n2), L, p.slices);
    PHF_TRY(p.arena.alloc(&p.B2sl, b2));
    PHF_CUDA(cudaMemset(p.B2sl, 0, b2));
    PHF_TRY(p.arena.alloc(&p.eB2, (size_t)oz_pad_rows(n2)));
    if (!p.rz) {
        PHF_TRY(p.arena.alloc(&p.B1sl, b1));
        PHF_CUDA(cudaMemset(p.B1sl, 0, b1));
        PHF_TRY(p.arena.alloc(&p.eB1, (size_t)oz_pad_rows(L)));
    }
    if (p.ek_sym && !p.rz) {
        double *Bp = nullptr;
        PHF_TRY(p.arena.alloc(&Bp, (size_t)(L * kc)));
        PHF_TRY(oz_cholesky_pairs(n, L, p.Bst, p.pairs_le, Bp, 0));
        PHF_TRY(oz_slice_rows_strided(L, (int)kc, Bp, kc, 1, p.slices, oz_pad_rows(L), p.B1sl, p.eB1, 0));
        PHF_CUDA(cudaDeviceSynchronize());
        p.arena.free_one(Bp);
    } else if (!p.rz) {
        PHF_TRY(oz_slice_rows_strided(L, (int)n2, p.Bst, n2, 1, p.slices, oz_pad_rows(L), p.B1sl, p.eB1, 0));
    }
    PHF_TRY(oz_slice_rows_strided((int)n2, L, p.Bst, 1, n2, p.slices, oz_pad_rows(n2), p.B2sl, p.eB2, 0));
    return PHF_OK;
}

// Rows of panel [i0, i0 + ip) in the symmetric exchange form: pairs (i, k >= i) and (i, k > i).
inline long long sym_rows(int n, int i0, int ip) { return (long long)ip * (n - i0) - (long long)ip * (ip - 1) / 2; }
inline long long pair_index_le(long long n, long long l, long long j) { return l * n - l * (l - 1) / 2 + (j - l); }
inline long long pair_index_lt(long long n, long long l, long long j) {
    return l * (n - 1) - l * (l - 1) / 2 + (j - l - 1);
}

// The pair tables of the symmetric form (i << 16 | k in row order, i <= k and i < k), on the device.
int upload_pair_tables(PlanImpl &p) {
    const int n = p.n;
    std::vector<int> le, lt;
    le.reserve((size_t)n * (n + 1) / 2);
    lt.reserve((size_t)n * (n - 1) / 2);
    for (int i = 0; i < n; ++i)
        for (int k = i; k < n; ++k) {
            le.push_back(i << 16 | k);
            if (k > i) lt.push_back(i << 16 | k);
        }
    PHF_TRY(p.arena.alloc(&p.pairs_le, le.size()));
    PHF_TRY(p.arena.alloc(&p.pairs_lt, std::max<size_t>(lt.size(), 1)));
    PHF_CUDA(cudaMemcpy(p.pairs_le, le.data(), le.size() * sizeof(int), cudaMemcpyHostToDevice));
    if (!lt.empty()) PHF_CUDA(cudaMemcpy(p.pairs_lt, lt.data(), lt.size() * sizeof(int), cudaMemcpyHostToDevice));
    return PHF_OK;
}

int build_exchange_matrix(PlanImpl &p) {
    const int n = p.n, L = p.L;
    const long long n2 = (long long)n * n;
    if (p.prec != PHF_PREC_FP64) {
        PHF_TRY(p.arena.alloc(&p.ozerr, 1));
        PHF_CUDA(cudaMemset(p.ozerr, 0, sizeof(int)));
    }
    if (p.streamed) {  // buffers of one exchange panel; the rows themselves are formed per chunk
        // (symmetric form: a panel's Gram block, ip n x (n - i0) n, and its rows, rows_s x n(n+1)/2 plus
        // rows_a x n(n-1)/2 with rows_a < rows_s <= ip (n - i0), fit in the full form's ek_ipanel n x n^2)
        const long long rows = (long long)p.ek_ipanel * n;
        PHF_TRY(p.arena.alloc(&p.Gp, (size_t)(rows * n2)));
        if (p.ek_sym) PHF_TRY(upload_pair_tables(p));
        if (p.prec == PHF_PREC_FP64) {
            PHF_TRY(p.arena.alloc(&p.EKp, (size_t)(rows * n2)));
        } else {
            size_t bytes = oz_slice_bytes(oz_pad_rows(rows), n2, p.slices);
            long long erows = oz_pad_rows(rows);
            if (p.ek_sym) {
                const long long kks = (long long)n * (n + 1) / 2, kka = (long long)n * (n - 1) / 2;
                bytes = 0;
                erows = 0;
                for (int pi = 0; pi < p.ek_npanel; ++pi) {
                    const int i0 = p.ek_i0[pi], ip = p.ek_i0[pi + 1] - i0;
                    const long long rs = oz_pad_rows(sym_rows(n, i0, ip)),
                                    ra = oz_pad_rows(std::max<long long>(sym_rows(n, i0, ip) - ip, 1));
                    bytes = std::max(bytes, oz_slice_bytes(rs, kks, p.slices) + oz_slice_bytes(ra, kka, p.slices));
                    erows = std::max(erows, rs + ra);
                }
            }
            if (p.rz) {
                const long long kks = (long long)n * (n + 1) / 2;
                for (int pi = 0; pi < p.ek_npanel; ++pi)
                    p.rz_rows = std::max(p.rz_rows, sym_rows(n, p.ek_i0[pi], p.ek_i0[pi + 1] - p.ek_i0[pi]));
                PHF_TRY(p.arena.alloc(&p.rzE, rz_operand_bytes(2 * kRzModuli, p.rz_rows, kks)));
                PHF_TRY(p.arena.alloc(&p.rzEe, (size_t)(2 * p.rz_rows)));
            } else {
                PHF_TRY(p.arena.alloc(&p.EKpsl, bytes));
                PHF_CUDA(cudaMemset(p.EKpsl, 0, bytes));
                PHF_TRY(p.arena.alloc(&p.eEKp, (size_t)erows));
                PHF_CUDA(cudaMemset(p.eEKp, 0, (size_t)erows * sizeof(int)));
            }
            PHF_TRY(build_coulomb_slices(p));
        }
        PHF_CUDA(cudaDeviceSynchronize());
        return PHF_OK;
    }
    if (p.ek_sym) {
        // The symmetric and antisymmetric rows of all pairs from the Gram block, in panels of indices i of at most 1 GiB
        // of it: the whole block is twice the FP64 rows kept (n = 128: 2.1 GB beside 1.1), and made a plan that fits
        // run out of memory while it was formed.  (Slices take the whole block; it and they are less than the full
        // rows and theirs.)
        const long long kks = (long long)n * (n + 1) / 2, kka = (long long)n * (n - 1) / 2, nn = n;
        const bool slices = p.prec != PHF_PREC_FP64 && !p.rz;
        const int panel = slices ? n : (int)std::max<long long>(1, std::min(nn, (1LL << 27) / (nn * n2)));
        const long long rs = oz_pad_rows(kks), ra = oz_pad_rows(kka);
        size_t bs = 0;
        PHF_TRY(upload_pair_tables(p));
        if (p.prec == PHF_PREC_FP64) {
            PHF_TRY(p.arena.alloc(&p.EK, (size_t)(kks * kks + kka * kka)));
        } else if (p.rz) {
            p.rz_rows = kks;
            PHF_TRY(p.arena.alloc(&p.rzE, rz_operand_bytes(2 * kRzModuli, kks, kks)));
            PHF_TRY(p.arena.alloc(&p.rzEe, (size_t)(2 * kks)));
        } else {
            bs = oz_slice_bytes(rs, kks, p.slices);
            const size_t ba = oz_slice_bytes(ra, kka, p.slices);
            PHF_TRY(p.arena.alloc(&p.EKsl, bs + ba));
            PHF_CUDA(cudaMemset(p.EKsl, 0, bs + ba));
            PHF_TRY(p.arena.alloc(&p.ea, (size_t)(rs + ra)));
            PHF_CUDA(cudaMemset(p.ea, 0, (size_t)(rs + ra) * sizeof(int)));
        }
        double *G = nullptr;
        PHF_TRY(p.arena.alloc(&G, (size_t)(panel * nn * n2)));
        for (int i0 = 0; i0 < n; i0 += panel) {
            const int ip = std::min(panel, n - i0);
            const long long gcols = (nn - i0) * nn, ts0 = pair_index_le(nn, i0, i0),
                            ta0 = i0 + 1 < n ? pair_index_lt(nn, i0, i0 + 1) : kka;
            OutView go = vo(reinterpret_cast<zc *>(G), gcols, 1);
            go.real = 1;
            PHF_TRY(zgemm_strided(ip * n, (int)gcols, L, 1, 1, Z1, vd(p.Bst + (size_t)i0 * n, 1, n2),
                                  vd(p.Bst + (size_t)i0 * n, n2, 1), Z0, go, nullptr, 0));
            if (p.prec == PHF_PREC_FP64)
                PHF_TRY(launch_ek_sym_panel(n, i0, ip, i0, p.pairs_le, G, gcols, p.EK + ts0 * kks,
                                            p.EK + kks * kks + ta0 * kka, 0));
            else if (p.rz)
                PHF_TRY(rz_exchange_rows(n, i0, ip, i0, p.pairs_le, G, gcols, kks,
                                         p.rzE + (size_t)ts0 * rz_operand_bytes(1, 1, kks), p.rzEe + ts0, 0));
            else
                PHF_TRY(oz_slice_ek_sym_panel(n, 0, n, 0, p.pairs_le, G, n2, p.slices, rs, p.EKsl, p.ea, ra, p.EKsl + bs,
                                              p.ea + rs, 0));
        }
        PHF_CUDA(cudaDeviceSynchronize());
        p.arena.free_one(G);
        if (p.prec == PHF_PREC_FP64) {
            // the Coulomb term over pairs: B_L[l][j] (2 - delta_lj)
            PHF_TRY(p.arena.alloc(&p.Bpair, (size_t)(L * kks)));
            PHF_TRY(oz_cholesky_pairs(n, L, p.Bst, p.pairs_le, p.Bpair, 0));
        } else {
            PHF_TRY(build_coulomb_slices(p));
        }
        PHF_CUDA(cudaDeviceSynchronize());
        return PHF_OK;
    }
    double *EK = nullptr;
    PHF_TRY(p.arena.alloc(&EK, (size_t)(n2 * n2)));
    OutView o = vo(reinterpret_cast<zc *>(EK), n, 1, n2, n2 * n);
    o.real = 1;
    View Bv = vd(p.Bst, n2, 1, n, 0);
    PHF_TRY(zgemm_strided(n, n, L, n, n, Z1, vd(p.Bst, 1, n2, 0, n), Bv, Z0, o, nullptr, 0));
    if (p.prec != PHF_PREC_FP64) {
        const size_t bytes = oz_slice_bytes(oz_pad_rows(n2), n2, p.slices);
        PHF_TRY(p.arena.alloc(&p.EKsl, bytes));
        PHF_CUDA(cudaMemset(p.EKsl, 0, bytes));
        PHF_TRY(p.arena.alloc(&p.ea, (size_t)oz_pad_rows(n2)));
        PHF_TRY(oz_slice_rows((int)n2, (int)n2, EK, n2, p.slices, oz_pad_rows(n2), p.EKsl, p.ea, 0));
        PHF_TRY(build_coulomb_slices(p));
    }
    PHF_CUDA(cudaDeviceSynchronize());
    if (p.prec == PHF_PREC_FP64) {
        p.EK = EK;  // the FP64 back-end multiplies by it
    } else {
        p.arena.free_one(EK);  // the tensor-core back-end only needs its slices
        p.EK = nullptr;
    }
    return PHF_OK;
}

// Exchange term of the streamed form for one chunk.  For each panel of ek_ipanel spatial indices i:
// the Gram block G[(i, l)][(k, j)] = sum_L B_L[i][l] B_L[k][j] (rows (i, l) of B^T times B, k-dim L),
// its rows rearranged into the exchange rows EK[(i, k)][(l, j)] = (il|kj), and those rows times the
// chunk's density columns.  FP64 form: the panel's exchange rows times the gathered density blocks
// Kin into the matching rows of Kvec.  Tensor-core forms: the panel is sliced, and the product's
// epilogue writes -K of the panel's rows straight into Gamma.  The Gram block costs 2 n^2 ipanel L
// flops per panel (2 n^4 L per chunk against 16 n^4 per grid point).
// Symmetric form (p.ek_sym): panel p covers i in [ek_i0[p], ek_i0[p + 1]); its Gram block keeps only
// the columns (k >= i0, j), G[(i - i0) n + l][(k - i0) n + j] (row stride (n - i0) n), and yields the
// panel's symmetric rows (pairs i <= k) and antisymmetric rows (i < k), each multiplied by the matching
// half of the chunk's densities: half the exchange GEMM's and the Gram blocks' work of the full form.
int exchange_streamed_sym(PlanImpl &p, int bc, cudaStream_t st) {
    const int n = p.n, L = p.L, b = p.b;
    const long long nn = n, n2 = nn * nn, kks = nn * (nn + 1) / 2, kka = nn * (nn - 1) / 2;
    for (int pi = 0; pi < p.ek_npanel; ++pi) {
        const int i0 = p.ek_i0[pi], ip = p.ek_i0[pi + 1] - i0;
        const long long gcols = (nn - i0) * nn, rows_s = sym_rows(n, i0, ip), rows_a = rows_s - ip;
        const int grows = ip * n;
        const long long ts0 = pair_index_le(nn, i0, i0), ta0 = rows_a > 0 ? pair_index_lt(nn, i0, i0 + 1) : 0;
        if (p.prec == PHF_PREC_FP64) {
            double *EKs = p.streamed ? p.EKp : p.EK, *EKa = EKs + rows_s * kks;
            double *Kv = reinterpret_cast<double *>(p.Kvec);
            const double *Ki = reinterpret_cast<const double *>(p.Kin);
            if (p.library_gemm && cublasSetStream(reinterpret_cast<cublasHandle_t>(p.cublas), st) !=
                                      CUBLAS_STATUS_SUCCESS) {
                set_error(PHF_ERR_CUDA, "cublasSetStream failed");
                return PHF_ERR_CUDA;
            }
            if (!p.streamed) {
                // the stored rows
            } else if (p.library_gemm) {
                cublasHandle_t h = reinterpret_cast<cublasHandle_t>(p.cublas);
                const double one = 1.0, zero = 0.0;
                ProfScope prof(st, PROF_JK);
                // column-major: G^T (gcols x grows) = (columns k >= i0 of B^T) * (rows of B^T)^T
                if (cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, (int)gcols, grows, L, &one, p.Bst + (size_t)i0 * n,
                                (int)n2, p.Bst + (size_t)i0 * n, (int)n2, &zero, p.Gp, (int)gcols) !=
                        CUBLAS_STATUS_SUCCESS) {
                    set_error(PHF_ERR_CUDA, "cublasDgemm (exchange panel) failed");
                    return PHF_ERR_CUDA;
                }
            } else {
                OutView o = vo(reinterpret_cast<zc *>(p.Gp), gcols, 1);
                o.real = 1;
                PHF_TRY(zgemm_strided(grows, (int)gcols, L, 1, 1, Z1, vd(p.Bst + (size_t)i0 * n, 1, n2),
                                      vd(p.Bst + (size_t)i0 * n, n2, 1), Z0, o, nullptr, st));
            }
            if (p.streamed) PHF_TRY(launch_ek_sym_panel(n, i0, ip, i0, p.pairs_le, p.Gp, gcols, EKs, EKa, st));
            if (p.library_gemm) {
                cublasHandle_t h = reinterpret_cast<cublasHandle_t>(p.cublas);
                const double one = 1.0, zero = 0.0;
                ProfScope prof(st, PROF_JK);
                if (cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, 8 * bc, (int)rows_s, (int)kks, &one, Ki, 8 * b, EKs,
                                (int)kks, &zero, Kv + (size_t)ts0 * 8 * b, 8 * b) != CUBLAS_STATUS_SUCCESS ||
                    (rows_a > 0 &&
                     cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, 8 * bc, (int)rows_a, (int)kka, &one,
                                 Ki + (size_t)kks * 8 * b, 8 * b, EKa, (int)kka, &zero,
                                 Kv + (size_t)(kks + ta0) * 8 * b, 8 * b) != CUBLAS_STATUS_SUCCESS)) {
                    set_error(PHF_ERR_CUDA, "cublasDgemm (exchange rows) failed");
                    return PHF_ERR_CUDA;
                }
            } else {
                PHF_TRY(zgemm_strided((int)rows_s, 4 * bc, (int)kks, 1, 1, Z1, vd(EKs, kks, 1), vz(p.Kin, 4LL * b, 1),
                                      Z0, vo(p.Kvec + (size_t)ts0 * 4 * b, 4LL * b, 1), nullptr, st));
                if (rows_a > 0)
                    PHF_TRY(zgemm_strided((int)rows_a, 4 * bc, (int)kka, 1, 1, Z1, vd(EKa, kka, 1),
                                          vz(p.Kin + (size_t)kks * 4 * b, 4LL * b, 1), Z0,
                                          vo(p.Kvec + (size_t)(kks + ta0) * 4 * b, 4LL * b, 1), nullptr, st));
            }
        } else {
            const long long rps = oz_pad_rows(rows_s), rpa = oz_pad_rows(std::max<long long>(rows_a, 1));
            signed char *As = p.streamed ? p.EKpsl : p.EKsl, *Aa = As + oz_slice_bytes(rps, kks, p.slices);
            int *es = p.streamed ? p.eEKp : p.ea, *ea = es + rps;
            if (p.streamed) {
                OzEx gx;
                gx.b_rows_pad = oz_pad_rows(n2);
                gx.b_row0 = i0 * n;
                PHF_TRY(oz_gemm_ex(grows, (int)gcols, L, p.slices, p.B2sl, oz_pad_rows(n2), i0 * n, p.eB2, p.B2sl,
                                   p.eB2, p.Gp, gcols, 0, 0, p.ozerr, st, 0, 0, gx));
                if (p.rz)
                    PHF_TRY(rz_exchange_rows(n, i0, ip, i0, p.pairs_le, p.Gp, gcols, p.rz_rows, p.rzE, p.rzEe, st));
                else
                    PHF_TRY(oz_slice_ek_sym_panel(n, i0, ip, i0, p.pairs_le, p.Gp, gcols, p.slices, rps, As, es, rpa,
                                                  Aa, ea, st));
            }
            if (p.rz) {
                RzFock f;
                f.n = n;
                f.L = L;
                f.rows = (int)rows_s;
                f.pair0 = (int)ts0;
                f.pairs = p.pairs_le;
                f.K = p.rzK;
                f.ek = p.rzKe;
                f.k_rows = 8LL * b;
                f.E = p.rzE;
                f.ee = p.rzEe;
                f.e_rows = p.rz_rows;
                f.D = p.rzD;
                f.ed = p.rzDe;
                f.d_rows = 2LL * b;
                f.B2 = p.rzB2;
                f.e2 = p.rzB2e;
                f.C = p.rzC;
                f.CJ = p.rzCJ;
                f.h = p.fold_h ? p.h : nullptr;
                f.err = p.ozerr;
                for (int s0 = 0; s0 < bc; s0 += p.rz_sub) {
                    f.w0 = s0;
                    f.pts = std::min(p.rz_sub, bc - s0);
                    f.Gam = p.Gam + (size_t)s0 * p.M * p.M;
                    PHF_TRY(rz_fock(f, st));
                }
                continue;
            }
            OzEx sx;
            sx.gamma_mode = 1;
            sx.g_pairs = p.pairs_le;
            PHF_TRY(oz_gemm_ex((int)rows_s, 8 * bc, (int)kks, p.slices, As, rps, 0, es, p.Bsl, p.eb,
                               reinterpret_cast<double *>(p.Gam), 0, 0, 0, p.ozerr, st, n, (int)ts0, sx));
            if (rows_a > 0) {
                OzEx ax;
                ax.gamma_mode = 2;
                ax.g_pairs = p.pairs_lt;
                PHF_TRY(oz_gemm_ex((int)rows_a, 8 * bc, (int)kka, p.slices, Aa, rpa, 0, ea, p.Bsl + p.bsl_a_off,
                                   p.eb_a, reinterpret_cast<double *>(p.Gam), 0, 0, 0, p.ozerr, st, n, (int)ta0, ax));
            }
        }
    }
    return PHF_OK;
}

int exchange_streamed(PlanImpl &p, int bc, cudaStream_t st) {
    if (p.ek_sym) return exchange_streamed_sym(p, bc, st);
    const int n = p.n, L = p.L, b = p.b;
    const long long n2 = (long long)n * n, prow = (long long)p.ek_ipanel * n;
    for (int pi = 0; pi < p.ek_npanel; ++pi) {
        const int i0 = pi * p.ek_ipanel, ip = std::min(p.ek_ipanel, n - i0);
        const int rows = ip * n;
        if (p.prec == PHF_PREC_FP64) {
            if (p.library_gemm) {
                cublasHandle_t h = reinterpret_cast<cublasHandle_t>(p.cublas);
                const double one = 1.0, zero = 0.0;
                ProfScope prof(st, PROF_JK);
                // column-major: G^T (n^2 x rows) = (B^T) (n^2 x L) * (rows of B^T)^T
                if (cublasSetStream(h, st) != CUBLAS_STATUS_SUCCESS ||
                    cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_T, (int)n2, rows, L, &one, p.Bst, (int)n2,
                                p.Bst + (size_t)i0 * n, (int)n2, &zero, p.Gp, (int)n2) != CUBLAS_STATUS_SUCCESS) {
                    set_error(PHF_ERR_CUDA, "cublasDgemm (exchange panel) failed");
                    return PHF_ERR_CUDA;
                }
            } else {
                OutView o = vo(reinterpret_cast<zc *>(p.Gp), n2, 1);
                o.real = 1;
                PHF_TRY(zgemm_strided(rows, (int)n2, L, 1, 1, Z1, vd(p.Bst + (size_t)i0 * n, 1, n2), vd(p.Bst, n2, 1),
                                      Z0, o, nullptr, st));
            }
            PHF_TRY(launch_ek_panel(n, ip, p.Gp, n2, p.EKp, n2, st));
            if (p.library_gemm) {
                cublasHandle_t h = reinterpret_cast<cublasHandle_t>(p.cublas);
                const double one = 1.0, zero = 0.0;
                ProfScope prof(st, PROF_JK);
                if (cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, 8 * bc, rows, (int)n2, &one,
                                reinterpret_cast<const double *>(p.Kin), 8 * b, p.EKp, (int)n2, &zero,
                                reinterpret_cast<double *>(p.Kvec) + (size_t)i0 * n * 8 * b, 8 * b) !=
                    CUBLAS_STATUS_SUCCESS) {
                    set_error(PHF_ERR_CUDA, "cublasDgemm (exchange rows) failed");
                    return PHF_ERR_CUDA;
                }
            } else {
                PHF_TRY(zgemm_strided(rows, 4 * bc, (int)n2, 1, 1, Z1, vd(p.EKp, n2, 1), vz(p.Kin, 4LL * b, 1), Z0,
                                      vo(p.Kvec + (size_t)i0 * n * 4 * b, 4LL * b, 1), nullptr, st));
            }
        } else {
            PHF_TRY(oz_gemm_ex(rows, (int)n2, L, p.slices, p.B2sl, oz_pad_rows(n2), i0 * n, p.eB2, p.B2sl, p.eB2, p.Gp,
                               n2, 0, 0, p.ozerr, st, 0, 0));
            PHF_TRY(oz_slice_ek_panel(n, ip, p.Gp, n2, p.slices, oz_pad_rows(prow), p.EKpsl, p.eEKp, st));
            PHF_TRY(oz_gemm_ex(rows, 8 * bc, (int)n2, p.slices, p.EKpsl, oz_pad_rows(prow), 0, p.eEKp, p.Bsl, p.eb,
                               reinterpret_cast<double *>(p.Gam), 0, 0, 0, p.ozerr, st, n, i0 * n));
        }
    }
    return PHF_OK;
}

// Gamma(rho_w) X_w through the spatial ERI matrix:
//   rho_w = X_w bra^H;  J = B^T (B vec P), P = rho_aa + rho_bb;  K_st = EK vec(rho_st);
//   Gamma_w = I (x) J - K;  GX_w = Gamma_w X_w;  e2_w = tr(bra^H GX_w) / 2
// FP64 form: J and K in FP64 GEMMs, Gamma assembled from both.  Tensor-core forms: the exchange
// GEMM's epilogue writes -K into Gamma and J is then added to the diagonal spin blocks.
int gamma_x_eri(PlanImpl &p, int bc, cudaStream_t st) {
    const int M = p.M, N = p.N, n = p.n, L = p.L, b = p.b;
    const long long ld = (long long)b * N, MM = (long long)M * M, n2 = (long long)n * n;
    // tensor-core path with n <= 64: the operand columns are formed and sliced in one kernel, no density in HBM
    const bool fused = p.prec != PHF_PREC_FP64 && oz_rho_slice_ok(n) && !p.rz;
    // rho_i8: the densities of the whole chunk as ONE int8 GEMM.  Row (w, i) of X,
    // X_w[i][:] at Xs + (i b + w) N, is a row of 2N reals (re, im interleaved), and rho_w[i][j] =
    // sum_k X_w[i][k] conj(bra[j][k]) is its product with rows 2j (real part) and 2j + 1 (imaginary
    // part) of the bra's 2M x 2N operand: the (M bc) x 2M reals are the points' densities one after
    // another (rows (i, w) put a point's rows 15 MB apart at n = 200, and the operand kernels, which read
    // them along both indices, slowed down: 2.0 against 1.7 ms for 608 points)
    const long long rrs = M, rws = MM;
    if (p.rho_i8) {
        const long long xrows = oz_pad_rows((long long)M * b);
        PHF_TRY(oz_slice_point_rows(M, b, bc, 2 * N, reinterpret_cast<const double *>(p.Xs), 2LL * N, p.slices, xrows,
                                    p.Xsl, p.eX, st));
        PHF_TRY(launch_bra_rho_operand(M, N, p.bra, p.BRop, st));
        PHF_TRY(oz_slice_rows(2 * M, 2 * N, p.BRop, 2LL * N, p.slices, oz_pad_cols(2LL * M), p.BRsl, p.eBR, st));
        PHF_TRY(oz_gemm_ex((int)((long long)M * bc), 2 * M, 2 * N, p.slices, p.Xsl, xrows, 0, p.eX, p.BRsl, p.eBR,
                           reinterpret_cast<double *>(p.Rho), 2LL * M, 0, 0, p.ozerr, st, 0, 0));
    } else if (!fused) {
        PHF_TRY(zgemm_strided(M, M, N, bc, 1, Z1, vz(p.Xs, ld, 1, N), vz(p.bra, 1, N, 0, 0, 1), Z0,
                              vo(p.Rho, M, 1, MM), nullptr, st));
    }
    if (p.prec == PHF_PREC_FP64 && p.Bpair) {
        // over the pairs l <= j: P's symmetric half is the sum of Kin's aa and bb columns; J at pair rows
        const int kp = n * (n + 1) / 2;
        PHF_TRY(launch_gather_kin_sym(n, bc, p.pairs_le, p.Rho, p.Kin, 4LL * b, st, p.Pvec, b));
        PHF_TRY(zgemm_strided(L, bc, kp, 1, 1, Z1, vd(p.Bpair, kp, 1), vz(p.Pvec, b, 1), Z0, vo(p.dvec, b, 1), nullptr,
                              st));
        PHF_TRY(zgemm_strided(kp, bc, L, 1, 1, Z1, vd(p.Bpair, 1, kp), vz(p.dvec, b, 1), Z0, vo(p.Jvec, b, 1), nullptr,
                              st));
    } else if (p.prec == PHF_PREC_FP64) {
        PHF_TRY(launch_gather_p(n, bc, p.Rho, p.Pvec, b, st));
        PHF_TRY(zgemm_strided(L, bc, (int)n2, 1, 1, Z1, vd(p.Bst, n2, 1), vz(p.Pvec, b, 1), Z0, vo(p.dvec, b, 1),
                              nullptr, st));
        PHF_TRY(zgemm_strided((int)n2, bc, L, 1, 1, Z1, vd(p.Bst, 1, n2), vz(p.dvec, b, 1), Z0, vo(p.Jvec, b, 1),
                              nullptr, st));
    } else {
        if (fused)
            PHF_TRY(oz_rho_slice(n, N, bc, p.Xs, ld, p.bra, p.slices, p.Bsl, p.eb, p.Psl, p.ePc, st));
        else if (p.rz) {
            PHF_TRY(rz_density(n, bc, p.pairs_le, p.Rho, rrs, rws, 8LL * b, p.rzK, p.rzKe, 2LL * b, p.rzP, p.rzPe, st));
            PHF_TRY(rz_coulomb_d(n, L, bc, p.rzP, 2LL * b, p.rzPe, p.rzB1, p.rzB1e, p.rzCJ, p.rzD, p.rzDe, p.ozerr, st));
        } else if (p.ek_sym)
            PHF_TRY(oz_slice_density_sym(n, bc, p.pairs_le, p.Rho, rrs, rws, p.slices, p.Bsl, p.eb,
                                         p.Bsl + p.bsl_a_off, p.eb_a, oz_pad_cols(8LL * bc), p.Psl, p.ePc,
                                         oz_pad_cols(2LL * bc), st));
        else
            PHF_TRY(oz_slice_density(n, bc, p.Rho, rrs, rws, p.slices, p.Bsl, p.eb, oz_pad_cols(8LL * bc), p.Psl,
                                     p.ePc, oz_pad_cols(2LL * bc), st));
    }
    // tensor-core path: the Coulomb chain runs on a second stream beside the exchange GEMM (independent
    // operands and outputs; its small, latency-bound launches fill the SMs the exchange GEMM's last
    // wave leaves idle).  Joined before J is added to Gamma.  Not while per-launch profiling is on:
    // event times of overlapping kernels would count the shared time twice.
    cudaStream_t js = st;
    const bool fork = p.prec != PHF_PREC_FP64 && !p.rz && !g_prof.on;
    const int kcoul = p.ek_sym ? n * (n + 1) / 2 : (int)n2;  // Coulomb contraction over pairs l <= j, or all (l, j)
    if (p.prec != PHF_PREC_FP64 && !p.rz && !fork) {
        PHF_TRY(oz_gemm_splitk(L, 2 * bc, kcoul, p.slices, p.B1sl, p.eB1, p.Psl, p.ePc, p.dT, L, 1, kDSplit, p.dpart,
                               p.ozerr, st));
        PHF_TRY(oz_slice_rows_strided(2 * bc, L, p.dT, L, 1, p.slices, oz_pad_cols(2LL * bc), p.dsl, p.edc, st));
        PHF_TRY(oz_gemm_t((int)n2, 2 * bc, L, p.slices, p.B2sl, p.eB2, p.dsl, p.edc, p.Jr, n2, 0, 1, p.ozerr, st));
    }
    if (fork) {
        if (!p.side) {
            // highest priority: its few small launches get SMs as the exchange GEMM's CTAs retire
            int lo = 0, hi = 0;
            PHF_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
            PHF_CUDA(cudaStreamCreateWithPriority(&p.side, cudaStreamNonBlocking, hi));
            PHF_CUDA(cudaEventCreateWithFlags(&p.ev_fork, cudaEventDisableTiming));
            PHF_CUDA(cudaEventCreateWithFlags(&p.ev_join, cudaEventDisableTiming));
        }
        PHF_CUDA(cudaEventRecord(p.ev_fork, st));
        PHF_CUDA(cudaStreamWaitEvent(p.side, p.ev_fork, 0));
        js = p.side;
        // d^T (2 bc x L) = (B vec P)^T, then J (n^2 x 2 bc, real/imag pairs) = B^T d
        PHF_TRY(oz_gemm_splitk(L, 2 * bc, kcoul, p.slices, p.B1sl, p.eB1, p.Psl, p.ePc, p.dT, L, 1, kDSplit, p.dpart,
                               p.ozerr, js));
        PHF_TRY(oz_slice_rows_strided(2 * bc, L, p.dT, L, 1, p.slices, oz_pad_cols(2LL * bc), p.dsl, p.edc, js));
        // J^T (2 bc x n^2): transposed output keeps the epilogue's FP64 stores coalesced
        PHF_TRY(oz_gemm_t((int)n2, 2 * bc, L, p.slices, p.B2sl, p.eB2, p.dsl, p.edc, p.Jr, n2, 0, 1, p.ozerr, js));
        PHF_CUDA(cudaEventRecord(p.ev_join, js));
    }
    prof_set_class(PROF_JK);
    if (p.prec == PHF_PREC_FP64) {
        if (p.ek_sym) {
            if (!p.Bpair) PHF_TRY(launch_gather_kin_sym(n, bc, p.pairs_le, p.Rho, p.Kin, 4LL * b, st));
        } else

            PHF_TRY(launch_gather_kin(n, bc, p.Rho, p.Kin, 4LL * b, st));
        if (p.streamed || p.ek_sym) {
            PHF_TRY(exchange_streamed(p, bc, st));
        } else if (p.library_gemm) {
            // row-major Kvec (n^2 x 8bc reals) = EK (n^2 x n^2) Kin (n^2 x 8bc reals), i.e. column-major
            // Kvec^T = Kin^T EK^T
            cublasHandle_t h = reinterpret_cast<cublasHandle_t>(p.cublas);
            const double one = 1.0, zero = 0.0;
            ProfScope prof(st, PROF_JK);
            if (cublasSetStream(h, st) != CUBLAS_STATUS_SUCCESS ||
                cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, 8 * bc, (int)n2, (int)n2, &one,
                            reinterpret_cast<const double *>(p.Kin), 8 * b, p.EK, (int)n2, &zero,
                            reinterpret_cast<double *>(p.Kvec), 8 * b) != CUBLAS_STATUS_SUCCESS) {
                set_error(PHF_ERR_CUDA, "cublasDgemm failed");
                return PHF_ERR_CUDA;
            }
        } else {
            PHF_TRY(zgemm_strided((int)n2, 4 * bc, (int)n2, 1, 1, Z1, vd(p.EK, n2, 1), vz(p.Kin, 4LL * b, 1), Z0,
                                  vo(p.Kvec, 4LL * b, 1), nullptr, st));
        }
        prof_set_class(PROF_GEMM);
        PHF_TRY(launch_assemble_gamma(n, bc, p.Jvec, b, nullptr, 0, 0, p.Kvec, 4LL * b, nullptr, 0, 0, p.Gam, st,
                                      p.ek_sym ? (p.Bpair ? 2 : 1) : 0, p.fold_h ? p.h : nullptr));
    } else {
        // K (as K^T, 8 bc x n^2) written by the GEMM epilogue as -K into Gamma's complex M x M blocks
        if (p.streamed || p.ek_sym)
            PHF_TRY(exchange_streamed(p, bc, st));
        else
            PHF_TRY(oz_gemm_t((int)n2, 8 * bc, (int)n2, p.slices, p.EKsl, p.ea, p.Bsl, p.eb,
                              reinterpret_cast<double *>(p.Gam), 0, 0, 0, p.ozerr, st, n));
        if (fork) PHF_CUDA(cudaStreamWaitEvent(st, p.ev_join, 0));  // the Coulomb chain is done
        prof_set_class(PROF_GEMM);
        // (the residue form's J is in Gamma already)
        if (!p.rz) PHF_TRY(launch_add_coulomb_diag(n, bc, p.Jr, 1, n2, p.Gam, st, p.fold_h ? p.h : nullptr));
    }
    if (p.fx_i8) {
        // F_w X_w for the chunk's points on the int8 path, sub-batch by sub-batch
        for (int s0 = 0; s0 < bc; s0 += p.fx_b) {
            const int sb = std::min(p.fx_b, bc - s0);
            PHF_TRY(oz_slice_fock_rows(M, sb, p.Gam + (size_t)s0 * MM, MM, p.slices, p.fx_b_rows, p.FXsl, p.eFX, st));
            PHF_TRY(oz_slice_xcols(M, N, sb, p.Xs + (size_t)s0 * N, ld, p.slices, p.fx_a_rows, p.XTsl, p.eXT, st));
            PHF_TRY(oz_gemm_fx(M, N, sb, p.slices, p.XTsl, p.fx_a_rows, p.eXT, p.FXsl, p.fx_b_rows, p.eFX,
                               p.GX + (size_t)s0 * N, ld, p.ozerr, st));
        }
    } else {
        PHF_TRY(zgemm_strided(M, N, M, bc, 1, Z1, vz(p.Gam, M, 1, MM), vz(p.Xs, ld, 1, N), Z0, vo(p.GX, ld, 1, N),
                              nullptr, st));
    }
    if (p.fold_h)  // GX = F X: e2 = tr(bra^H F X) / 2 - e1 / 2
        PHF_TRY(launch_trace_conj(M, N, bc, p.bra, p.GX, ld, p.e2, 0.5, st, nullptr, p.e1, 0.5));
    else
        PHF_TRY(launch_trace_conj(M, N, bc, p.bra, p.GX, ld, p.e2, 0.5, st, p.HX));  // then GX <- HX + Gamma X
    return PHF_OK;
}

// Ket-side gradient of the chunk (exact mode): with V_w = (H1 + Gamma_w^H) C - C W_w^H + conj(h_w) C,
//   accKG += sum_w conj(Wt N_w) R_w^H V_w S_w^-H,   accKR += sum_w conj(Wt N_w) R_w^H C S_w^-H
// where R_w^H = Rpg[ig]^H R2[iy]^H R1[il]^H is applied factor by factor.
int ket_side(PlanImpl &p, int v, int bc, int w0, cudaStream_t st) {
    const int M = p.M, N = p.N, b = p.b;
    const long long ld = (long long)b * N, MM = (long long)M * M;
    PHF_TRY(zgemm_strided(M, N, M, bc, 1, Z1, vz(p.Gam, 1, M, MM, 0, 1), vz(p.bra, N, 1), Z0, vo(p.Vk, ld, 1, N),
                          nullptr, st));
    PHF_TRY(zgemm_strided(M, N, N, bc, 1, ZM1, vz(p.bra, N, 1), vz(p.W, 1, ld, N, 0, 1), Z1, vo(p.Vk, ld, 1, N),
                          nullptr, st));
    PHF_TRY(launch_ket_prep(M, N, bc, p.fold_h ? nullptr : p.Hb, p.bra, p.e1, p.e2, p.Vk, ld, st));
    PHF_TRY(zgemm_strided(M, N, N, bc, 1, Z1, vz(p.Vk, ld, 1, N), vz(p.Sinv, 1, ld, N, 0, 1), Z0, vo(p.Pk, ld, 1, N),
                          nullptr, st));
    PHF_TRY(zgemm_strided(M, N, N, bc, 1, Z1, vz(p.bra, N, 1), vz(p.Sinv, 1, ld, N, 0, 1), Z0, vo(p.Prk, ld, 1, N),
                          nullptr, st));
    const zc *Rs[3] = {p.R1, p.R2, p.Rpg};
    zc *src = p.Pk, *dst = p.Pk2, *srcr = p.Prk, *dstr = p.Prk2;
    for (int f = 0; f < 3; ++f) {
        const long long *offs = p.offs_k + 3LL * ((long long)f * p.nomega + w0);
        PHF_TRY(zgemm_strided(M, N, M, bc, 1, Z1, vz(Rs[f], 1, M, 0, 0, 1), vz(src, ld, 1, N), Z0, vo(dst, ld, 1, N),
                              offs, st));
        PHF_TRY(zgemm_strided(M, N, M, bc, 1, Z1, vz(Rs[f], 1, M, 0, 0, 1), vz(srcr, ld, 1, N), Z0, vo(dstr, ld, 1, N),
                              offs, st));
        std::swap(src, dst);
        std::swap(srcr, dstr);
    }
    const int nb2 = p.nb * p.nb;
    PHF_TRY(launch_accumulate(nb2, M, N, bc, p.Wt, p.nomega, w0, p.slotmap + (size_t)v * nb2, src, srcr, ld, p.det,
                              nullptr, nullptr, p.accKG, p.compKG, p.accKR, p.compKR, nullptr, nullptr, p.acc_scratch, st, 1));
    return PHF_OK;
}

// One (bra, ket) variant over all grid points, accumulated into slot map `v`.
// bra, ket: M x N row-major in the working basis; kety: the vector R_w multiplies
// (dense form: Ref ket in AO order; Cholesky form: ket itself).
int run_variant(PlanImpl &p, int v, cudaStream_t st) {
    const int M = p.M, N = p.N, n = p.n, L = p.L, b = p.b;
    const long long MN = (long long)M * N, ld = (long long)b * N, MM = (long long)M * M;
    // T1[g] = Rpg[g] kety ; T2[y, g] = R2[y] T1[g]
    PHF_TRY(zgemm_strided(M, N, M, p.npg, 1, Z1, vz(p.Rpg, M, 1, MM), vz(p.kety, N, 1, 0), Z0, vo(p.T1, N, 1, MN),
                          nullptr, st));
    const long long ld2 = (long long)p.ny * p.npg * N;  // T2 column-blocked: T2[r][(iy npg + ig) N + j]
    PHF_TRY(zgemm_strided(M, N, M, p.npg, p.ny, Z1, vz(p.R2, M, 1, 0, MM), vz(p.T1, N, 1, MN, 0), Z0,
                          vo(p.T2, ld2, 1, N, (long long)p.npg * N), nullptr, st));
    if (p.exact || p.fold_h)  // H1 bra (Cholesky forms: h applied to both spin rows of the interleaved order)
        PHF_TRY(zgemm_strided(n, 2 * N, n, 1, 1, Z1, vd(p.h, n, 1), vz(p.bra, 2 * N, 1), Z0, vo(p.Hb, 2 * N, 1), nullptr,
                              st));
    if (p.chol && !p.eri) {
        // V_L = (B_L (x) I_2) bra: (L n x n) x (n x 2N), rows (L, p), columns (sigma, j)
        PHF_TRY(zgemm_strided(L * n, 2 * N, n, 1, 1, Z1, vd(p.Bst, n, 1), vz(p.bra, 2 * N, 1), Z0, vo(p.V, 2 * N, 1),
                              nullptr, st));
    }
    for (int w0 = p.wbeg; w0 < p.wend; w0 += b) {
        const int bc = std::min(b, p.wend - w0);
        // Y_w = R1[il] T2[iy, ig]: one (M x M) x (M x ny npg N) product per Lebedev point when the
        // chunk holds whole blocks of ny npg points, else per point
        const int blk = p.ny * p.npg;
        if (p.R1b)
            PHF_TRY(launch_spin_block_y(n, N, bc, w0, blk, p.R1b, p.T2, ld2, p.Ys, ld, st));
        else if (w0 % blk == 0 && bc % blk == 0)
            PHF_TRY(zgemm_strided(M, (int)ld2, M, bc / blk, 1, Z1, vz(p.R1 + (size_t)(w0 / blk) * MM, M, 1, MM),
                                  vz(p.T2, ld2, 1), Z0, vo(p.Ys, ld, 1, ld2), nullptr, st));
        else
            PHF_TRY(zgemm_strided(M, N, M, bc, 1, Z1, vz(p.R1, M, 1), vz(p.T2, ld2, 1), Z0, vo(p.Ys, ld, 1, N),
                                  p.offs + 3LL * w0, st));
        zc *Y = p.Ys;
        if (!p.chol) {  // Ref-MO basis: Y <- Ref^H Y
            PHF_TRY(zgemm_strided(M, bc * N, M, 1, 1, Z1, vz(p.Refw, 1, M, 0, 0, 1), vz(p.Ys, ld, 1), Z0, vo(p.Ys2, ld, 1),
                                  nullptr, st));
            Y = p.Ys2;
        }
        // S_w = bra^H Y_w, formed as its transpose Y^T conj(bra) (bc N rows, N columns: for N <= 112 one
        // column tile of the FP64 GEMM instead of N rows padded to the row tile)
        PHF_TRY(zgemm_strided(bc * N, N, M, 1, 1, Z1, vz(Y, 1, ld), vz(p.bra, N, 1, 0, 0, 1), Z0, vo(p.S, 1, ld), nullptr,
                              st));
        PHF_TRY(overlap_inverse(N, bc, p.S, ld, N, p.Sinv, ld, N, p.det, p.logdet, p.flag, st));
        // X_w = Y_w S_w^-1
        PHF_TRY(zgemm_strided(M, N, N, bc, 1, Z1, vz(Y, ld, 1, N), vz(p.Sinv, ld, 1, N), Z0, vo(p.Xs, ld, 1, N), nullptr,
                              st));
        // HX and e1 = tr(bra^H H1 X)
        // (Cholesky form: X viewed as n x (2 ld) with spin sigma at column offset sigma*ld, batched over sigma)
        if (p.fold_h)  // H1 is part of Gamma: no HX; e1 = sum conj(H1 bra) X (H1 symmetric)
            PHF_TRY(launch_trace_conj(M, N, bc, p.Hb, p.Xs, ld, p.e1, 1.0, st));
        else if (p.chol)
            PHF_TRY(zgemm_strided(n, bc * N, n, 2, 1, Z1, vd(p.h, n, 1), vz(p.Xs, 2 * ld, 1, ld), Z0,
                                  vo(p.HX, 2 * ld, 1, ld), nullptr, st));
        else
            PHF_TRY(zgemm_strided(M, bc * N, M, 1, 1, Z1, vz(p.H1, M, 1), vz(p.Xs, ld, 1), Z0, vo(p.HX, ld, 1), nullptr, st));
        if (!p.fold_h) PHF_TRY(launch_trace_conj(M, N, bc, p.bra, p.HX, ld, p.e1, 1.0, st));
        // Gamma(rho_w) X_w and e2
        if (p.chol && p.eri) {
            PHF_TRY(gamma_x_eri(p, bc, st));
        } else if (p.chol) {  // factorized form (FP64 only: plan_create rejects the others)
            {
                prof_set_class(PROF_JK);
                // T_Lw = V_L^H X_w : batched over L, (N x M) x (M x bN)
                PHF_TRY(zgemm_strided(N, bc * N, M, L, 1, Z1, vz(p.V, 1, N, MN, 0, 1), vz(p.Xs, ld, 1), Z0,
                                      vo(p.T, ld, 1, (long long)N * ld), nullptr, st));
                PHF_TRY(launch_tprime(L, N, bc, p.T, ld, p.e2part, st));
                // Q_Lw = X_w T'_Lw : batched over (w, L)
                PHF_TRY(zgemm_strided(M, N, N, bc, L, Z1, vz(p.Xs, ld, 1, N, 0), vz(p.T, ld, 1, N, (long long)N * ld), Z0,
                                      vo(p.Q, ld, 1, N, (long long)M * ld), nullptr, st));
                // GX = [B_1 .. B_L] Q : (n x L n) x (L n x b N) for each spin sigma (column offset sigma*ld)
                PHF_TRY(zgemm_strided(n, bc * N, L * n, 2, 1, Z1, vd(p.Bst, 1, n), vz(p.Q, 2 * ld, 1, ld), Z0,
                                      vo(p.GX, 2 * ld, 1, ld), nullptr, st));
                prof_set_class(PROF_GEMM);
            }
            PHF_TRY(launch_rowsum(bc, L, p.e2part, p.e2, 0.5, st));
            PHF_TRY(launch_add_inplace(M, N, bc, p.HX, p.GX, ld, st));  // GX <- HX + Gamma X
        } else {
            prof_set_class(PROF_JK);
            // rho_w = X_w bra^H stored as vec: Pv[(l M + j) b + w]
            PHF_TRY(zgemm_strided(M, M, N, bc, 1, Z1, vz(p.Xs, ld, 1, N), vz(p.bra, 1, N, 0, 0, 1), Z0,
                                  vo(p.Pv, (long long)M * bc, bc, 1), nullptr, st));
            PHF_TRY(zgemm_strided((int)MM, bc, (int)MM, 1, 1, Z1, vz(p.H2r, MM, 1), vz(p.Pv, bc, 1), Z0, vo(p.Gv, bc, 1),
                                  nullptr, st));
            PHF_TRY(zgemm_strided(M, N, M, bc, 1, Z1, vz(p.Gv, (long long)M * bc, bc, 1), vz(p.Xs, ld, 1, N), Z0,
                                  vo(p.GX, ld, 1, N), nullptr, st));
            prof_set_class(PROF_GEMM);
            PHF_TRY(launch_trace_conj(M, N, bc, p.bra, p.GX, ld, p.e2, 0.5, st, p.HX));  // then GX <- HX + Gamma X
        }
        // GX now holds F X = HX + Gamma X:  W = bra^H F X (as its transpose, like S);  GX <- F X - X W
        PHF_TRY(zgemm_strided(bc * N, N, M, 1, 1, Z1, vz(p.GX, 1, ld), vz(p.bra, N, 1, 0, 0, 1), Z0, vo(p.W, 1, ld),
                              nullptr, st));
        PHF_TRY(zgemm_strided(M, N, N, bc, 1, ZM1, vz(p.Xs, ld, 1, N), vz(p.W, ld, 1, N), Z1, vo(p.GX, ld, 1, N), nullptr,
                              st));
        const int nb2 = p.nb * p.nb;
        PHF_TRY(launch_accumulate(nb2, M, N, bc, p.Wt, p.nomega, w0, p.slotmap + (size_t)v * nb2, p.GX, p.Xs, ld, p.det,
                                  p.e1, p.e2, p.accG, p.compG, p.accR, p.compR, p.accHS, p.compHS, p.acc_scratch, st));
        if (p.exact) PHF_TRY(ket_side(p, v, bc, w0, st));
    }
    return PHF_OK;
}

int zero_acc(PlanImpl &p, cudaStream_t st) {
    PHF_CUDA(cudaMemsetAsync(p.accG, 0, p.acc_bytes, st));
    return PHF_OK;
}

// The folded sums into outG, outR, outHS (rows mapped by `rowmap`; averaged with the ket side's sums when `ket`).
int fold_acc(PlanImpl &p, const int *rowmap, bool ket, zc *outG, zc *outR, zc *outHS, cudaStream_t st) {
    FoldSums S{p.accG, p.compG, p.accR, p.compR, nullptr, nullptr, nullptr, nullptr, p.accHS, p.compHS};
    if (ket) S.KG = p.accKG, S.cKG = p.compKG, S.KR = p.accKR, S.cKR = p.compKR;
    return launch_fold_out(p.nci * p.nci, p.M, p.N, rowmap, S, outG, outR, outHS, st);
}

// Status of an evaluation from its flag word and the tensor-core GEMM error word (host copies).
int flag_status(int flag, int oz) {
    if (oz) {
        set_error(PHF_ERR_CUDA, "tensor-core GEMM pipeline wait timed out (code " + std::to_string(oz) + ")");
        return PHF_ERR_CUDA;
    }
    if (flag & 1) {
        set_error(PHF_ERR_SINGULAR, "a rotated overlap bra^H R ket is exactly singular");
        return PHF_ERR_SINGULAR;
    }
    if (flag & 2) {
        set_error(PHF_ERR_NONFINITE, "non-finite rotated overlap");
        return PHF_ERR_NONFINITE;
    }
    return PHF_OK;
}

// Queues the device-to-host copies of the two status words on st (read after a synchronisation).
int enqueue_flags(PlanImpl &p, int *flag, int *oz, cudaStream_t st) {
    *flag = 0;
    *oz = 0;
    PHF_CUDA(cudaMemcpyAsync(flag, p.flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    if (p.ozerr) PHF_CUDA(cudaMemcpyAsync(oz, p.ozerr, sizeof(int), cudaMemcpyDeviceToHost, st));
    return PHF_OK;
}

int read_flag(PlanImpl &p, cudaStream_t st) {
    int flag = 0, oz = 0;
    PHF_TRY(enqueue_flags(p, &flag, &oz, st));
    PHF_CUDA(cudaStreamSynchronize(st));
    return flag_status(flag, oz);
}

// Hermiticity check of PHFTools.f90:195-200 on host copies
bool hermitian_ok(const std::vector<cd> &H, const std::vector<cd> &S, int nci) {
    double w1 = 0, w2 = 0, mh = 0, ms = 0;
    for (int i = 0; i < nci; ++i)
        for (int j = 0; j < nci; ++j) {
            cd a = H[i + (size_t)nci * j], at = H[j + (size_t)nci * i];
            cd s = S[i + (size_t)nci * j], stt = S[j + (size_t)nci * i];
            w1 = std::max(w1, std::abs((std::conj(at) - a).imag()));
            w2 = std::max(w2, std::abs((std::conj(stt) - s).imag()));
            mh = std::max(mh, std::abs(a));
            ms = std::max(ms, std::abs(s));
        }
    return !(w1 > mh * 1e-5 || w2 > ms * 1e-5);
}

}  // namespace

// Plans created with autotune: before the first capture, run `body` once directly while the GEMM
// launchers record their launches, then let the launch tuner time the candidates of every shape not
// yet tuned.  This evaluation's outputs are overwritten by the evaluation that follows.
template <typename F>
int maybe_tune(PlanImpl &p, cudaStream_t st, F &&body) {
    if (!p.autotune || p.tuned || g_prof.on) return PHF_OK;
    std::vector<TuneCall> calls;
    t_tune_record = &calls;
    const int rc = body(st);
    t_tune_record = nullptr;
    PHF_TRY(rc);
    PHF_CUDA(cudaStreamSynchronize(st));
    if (p.side) PHF_CUDA(cudaStreamSynchronize(p.side));
    PHF_TRY(tune_recorded(calls, st));
    p.tuned = true;
    return PHF_OK;
}

// buildhsg semantics: newMO = [I; Z] (MO basis), outputs in Fortran layout on the host.
// Run `body` (a fixed launch sequence of this plan) as a CUDA graph replayed on `st`: captured once
// on a private stream at first use, so per call the host submits one graph instead of ~100
// launches.  Falls back to direct launches while per-launch profiling is on, for the cuBLAS
// comparison form, or if capture is not possible.
template <typename F>
int launch_captured(PlanImpl &p, int key, cudaStream_t st, F &&body) {
    if (!p.graphs_ok || g_prof.on || p.library_gemm) return body(st);
    if (!p.gexec[key]) {
        if (!p.cap_stream && cudaStreamCreateWithFlags(&p.cap_stream, cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            p.graphs_ok = false;
            return body(st);
        }
        const unsigned long long l0 = g_launches;
        if (cudaStreamBeginCapture(p.cap_stream, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
            cudaGetLastError();
            p.graphs_ok = false;
            return body(st);
        }
        const int rc = body(p.cap_stream);
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(p.cap_stream, &g);
        const unsigned long long nl = g_launches - l0;
        g_launches = l0;
        cudaGraphExec_t ex = nullptr;
        if (rc == PHF_OK && e == cudaSuccess && g &&
            cudaGraphInstantiate(&ex, g, cudaGraphInstantiateFlagUseNodePriority) == cudaSuccess) {
            p.gexec[key] = ex;
            p.glaunch[key] = nl;
        } else {
            cudaGetLastError();
            p.graphs_ok = false;
        }
        if (g) cudaGraphDestroy(g);
        if (!p.gexec[key]) return rc != PHF_OK ? rc : body(st);
    }
    PHF_CUDA(cudaGraphLaunch(p.gexec[key], st));
    g_launches += p.glaunch[key];
    return PHF_OK;
}

int plan_buildhsg(PlanImpl &p, const phf_complex *z, phf_complex *hmat, phf_complex *smat, phf_complex *gradmat,
                  phf_complex *rdmmat) {
    const int M = p.M, N = p.N;
    const size_t MN = (size_t)M * N;
    cudaStream_t st = 0;
    PHF_CUDA(cudaSetDevice(p.device));
    // newMO and its conjugate in the MO basis
    std::vector<cd> mo(MN, cd(0, 0));
    for (int i = 0; i < N; ++i) mo[(size_t)i * N + i] = 1.0;
    for (int a = 0; a < M - N; ++a)
        for (int i = 0; i < N; ++i) {
            cd v = fz(z, (size_t)a + (size_t)(M - N) * i);
            if (p.cmplxconj == 0) v = cd(v.real(), 0.0);
            mo[(size_t)(N + a) * N + i] = v;
        }
    std::vector<cd> moc(MN);
    for (size_t i = 0; i < MN; ++i) moc[i] = std::conj(mo[i]);
    PHF_TRY(upload(p.newmo, mo));
    PHF_TRY(upload(p.newmoc, moc));

    PHF_TRY(zero_acc(p, st));
    const int nvar = p.cmplxconj == 2 ? 4 : 1;
    // variants (bra, ket): 0 (C, C), 1 (C, C*), 2 (C*, C*), 3 (C*, C)   -- RDM / RDMConj calls of :91-107.
    // The AO vectors Ref m are formed on the device (Refw holds Ref's rows in working order): in the
    // Cholesky form bra and ket are both Ref m in working order; in the dense form the bra stays in
    // the MO basis and the ket is Ref m in the reference order.
    for (int v = 0; v < nvar; ++v) {
        const bool cb = (v >= 2), ck = (v == 1 || v == 2);
        const zc *mb = cb ? p.newmoc : p.newmo, *mk = ck ? p.newmoc : p.newmo;
        if (p.chol)
            PHF_TRY(zgemm_strided(M, N, M, 1, 1, Z1, vz(p.Refw, M, 1), vz(mb, N, 1), Z0, vo(p.bra, N, 1), nullptr, st));
        else
            PHF_CUDA(cudaMemcpyAsync(p.bra, mb, MN * sizeof(zc), cudaMemcpyDeviceToDevice, st));
        PHF_TRY(zgemm_strided(M, N, M, 1, 1, Z1, vz(p.Refw, M, 1), vz(mk, N, 1), Z0, vo(p.kety, N, 1), nullptr, st));
        if (v == 0 && p.autotune && !p.tuned) {
            PHF_TRY(maybe_tune(p, st, [&](cudaStream_t s) -> int { return run_variant(p, 0, s); }));
            PHF_TRY(zero_acc(p, st));
        }
        PHF_TRY(launch_captured(p, v, st, [&](cudaStream_t s) -> int { return run_variant(p, v, s); }));
    }
    PHF_TRY(fold_acc(p, nullptr, false, p.accG, p.accR, p.accHS, st));

    // Gradmat_a = T Yg_a bra_a^H, Rdmmat likewise (T = Ref^H in the Cholesky form); every block is
    // formed on the device first, then all blocks and H, S come back in one synchronisation
    const int nci = p.nci, nb = p.nb;
    const long long ns = (long long)nci * nci;
    const size_t MMs = (size_t)M * M;
    for (int a = 0; a < nci * nci; ++a) {
        const int m = a % nci;
        const bool conj_bra = (p.cmplxconj == 2) && (m >= nb);
        const zc *nmo = conj_bra ? p.newmoc : p.newmo;
        for (int which = 0; which < 2; ++which) {
            zc *acc = (which == 0 ? p.accG : p.accR) + (size_t)a * MN;
            const zc *src = acc;
            if (p.chol) {
                PHF_TRY(zgemm_strided(M, N, M, 1, 1, Z1, vz(p.Refw, 1, M, 0, 0, 1), vz(acc, N, 1), Z0, vo(p.tmpG, N, 1),
                                      nullptr, st));
                src = p.tmpG;
            }
            // the M x M block in column-major order
            zc *outp = p.outMM + (2 * (size_t)a + which) * MMs;
            PHF_TRY(zgemm_strided(M, M, N, 1, 1, Z1, vz(src, N, 1), vz(nmo, 1, N, 0, 0, 1), Z0, vo(outp, 1, M),
                                  nullptr, st));
        }
    }
    std::vector<cd> blocks(2 * (size_t)ns * MMs), hs(2 * (size_t)ns);
    PHF_CUDA(cudaMemcpyAsync(blocks.data(), p.outMM, blocks.size() * sizeof(zc), cudaMemcpyDeviceToHost, st));
    PHF_CUDA(cudaMemcpyAsync(hs.data(), p.accHS, hs.size() * sizeof(zc), cudaMemcpyDeviceToHost, st));
    int flag = 0, oz = 0;
    PHF_TRY(enqueue_flags(p, &flag, &oz, st));
    PHF_CUDA(cudaStreamSynchronize(st));
    PHF_TRY(flag_status(flag, oz));  // on failure the host outputs are left untouched
    // scatter into the (nci, nci, M, M) Fortran-ordered arrays
    for (long long a = 0; a < ns; ++a)
        for (int which = 0; which < 2; ++which) {
            const cd *blk = blocks.data() + (2 * (size_t)a + which) * MMs;
            phf_complex *dst = which == 0 ? gradmat : rdmmat;
            for (size_t ij = 0; ij < MMs; ++ij) {
                dst[(size_t)a + (size_t)ns * ij].re = blk[ij].real();
                dst[(size_t)a + (size_t)ns * ij].im = blk[ij].imag();
            }
        }
    std::vector<cd> H(ns), S(ns);
    for (int a = 0; a < ns; ++a) {
        H[a] = hs[2 * a];
        S[a] = hs[2 * a + 1];
    }
    if (p.cmplxconj == 2) {  // PHFTools.f90:174-179
        const int d = nb;
        for (int i = 0; i < d; ++i)
            for (int j = 0; j < d; ++j) {
                H[(d + i) + (size_t)nci * j] = std::conj(H[j + (size_t)nci * (d + i)]);
                S[(d + i) + (size_t)nci * j] = std::conj(S[j + (size_t)nci * (d + i)]);
                H[(d + i) + (size_t)nci * (d + j)] = H[i + (size_t)nci * j];
                S[(d + i) + (size_t)nci * (d + j)] = S[i + (size_t)nci * j];
            }
    }
    bool finite = true;
    for (int a = 0; a < ns; ++a) {
        hmat[a].re = H[a].real();
        hmat[a].im = H[a].imag();
        smat[a].re = S[a].real();
        smat[a].im = S[a].imag();
        finite = finite && std::isfinite(H[a].real()) && std::isfinite(H[a].imag()) && std::isfinite(S[a].real()) &&
                 std::isfinite(S[a].imag());
    }
    if (!finite) {
        set_error(PHF_ERR_NONFINITE, "non-finite Hmat/Smat");
        return PHF_ERR_NONFINITE;
    }
    if (!hermitian_ok(H, S, nci)) {
        set_error(PHF_ERR_NOT_HERMITIAN, "Hmat/Smat are not Hermitian to 1e-5 (reference: STOP \"Not Hermitian\")");
        return PHF_ERR_NOT_HERMITIAN;
    }
    return PHF_OK;
}

void plan_release(PlanImpl &p) {
    if (p.cublas) {
        cublasDestroy(reinterpret_cast<cublasHandle_t>(p.cublas));
        p.cublas = nullptr;
    }
    for (auto &g : p.gexec)
        if (g) {
            cudaGraphExecDestroy(g);
            g = nullptr;
        }
    if (p.ev_fork) cudaEventDestroy(p.ev_fork);
    if (p.ev_join) cudaEventDestroy(p.ev_join);
    if (p.side) {
        // an evaluation that failed between the fork and the join leaves work here, and pooled memory (one-shot
        // calls) is reused in the order of the legacy default stream, which does not wait for this stream
        cudaStreamSynchronize(p.side);
        cudaStreamDestroy(p.side);
    }
    p.ev_fork = p.ev_join = nullptr;
    p.side = nullptr;
    if (p.cap_stream) {
        cudaStreamDestroy(p.cap_stream);
        p.cap_stream = nullptr;
    }
}

PlanImpl::~PlanImpl() { plan_release(*this); }

// Everything of one eval_device call enqueued on st, without the status check.  in_graph: the
// caller is capturing a batch graph, so the plan's own graph is not used.
int eval_enqueue(PlanImpl &p, const zc *d_c, zc *d_hs, zc *d_yg, zc *d_yr, cudaStream_t st, bool in_graph) {
    const int M = p.M, N = p.N;
    const long long MN = (long long)M * N;
    if (p.chol) {
        // rows of C from [alpha; beta] order to the working order: bra[r'] = C[perm[r']]
        PHF_TRY(launch_permute_rows(M, N, p.permdev, d_c, p.bra, p.kety, st));
    } else {
        PHF_CUDA(cudaMemcpyAsync(p.bra, d_c, MN * sizeof(zc), cudaMemcpyDeviceToDevice, st));
    }
    if (!p.chol) {
        // kety = Ref C (reference AO order)
        PHF_TRY(zgemm_strided(M, N, M, 1, 1, Z1, vz(p.Refw, M, 1), vz(p.bra, N, 1), Z0, vo(p.kety, N, 1), nullptr, st));
    }
    auto body = [&](cudaStream_t s) -> int {
        PHF_TRY(zero_acc(p, s));
        PHF_TRY(run_variant(p, 0, s));
        return PHF_OK;
    };
    if (in_graph) {
        PHF_TRY(body(st));
    } else {
        PHF_TRY(maybe_tune(p, st, body));
        PHF_TRY(launch_captured(p, 4, st, body));
    }
    // rows back to [alpha; beta] order where they were permuted; symmetrised bra + ket derivative in exact mode
    return fold_acc(p, p.chol ? p.permdev + M : nullptr, p.exact, d_yg, d_yr, d_hs, st);
}

int plan_eval_device(PlanImpl &p, const zc *d_c, zc *d_hs, zc *d_yg, zc *d_yr, cudaStream_t st) {
    if (p.cmplxconj == 2) {
        set_error(PHF_ERR_UNSUPPORTED, "phf_plan_eval_device: cmplxconj == 2 needs phf_plan_buildhsg");
        return PHF_ERR_UNSUPPORTED;
    }
    PHF_CUDA(cudaSetDevice(p.device));
    PHF_TRY(eval_enqueue(p, d_c, d_hs, d_yg, d_yr, st, false));
    return read_flag(p, st);
}

// phf_plan_eval_device without the host synchronisation: the status words are copied to device
// memory on the same stream for the caller to read together with its own results.
int plan_eval_device_async(PlanImpl &p, const zc *d_c, zc *d_hs, zc *d_yg, zc *d_yr, int *d_status, cudaStream_t st) {
    if (p.cmplxconj == 2) {
        set_error(PHF_ERR_UNSUPPORTED, "phf_plan_eval_device_async: cmplxconj == 2 needs phf_plan_buildhsg");
        return PHF_ERR_UNSUPPORTED;
    }
    PHF_CUDA(cudaSetDevice(p.device));
    PHF_TRY(eval_enqueue(p, d_c, d_hs, d_yg, d_yr, st, false));
    PHF_CUDA(cudaMemcpyAsync(d_status, p.flag, sizeof(int), cudaMemcpyDeviceToDevice, st));
    if (p.ozerr)
        PHF_CUDA(cudaMemcpyAsync(d_status + 1, p.ozerr, sizeof(int), cudaMemcpyDeviceToDevice, st));
    else
        PHF_CUDA(cudaMemsetAsync(d_status + 1, 0, sizeof(int), st));
    return PHF_OK;
}

// ------------------------------------------------------------------ batched evaluation
namespace {

__global__ void gather_flags_kernel(int *const *ptrs, int n, int *out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = ptrs[i] ? *ptrs[i] : 0;
}

constexpr int kMaxBranches = 16;

// The set of plans and buffers of the last batch, its graph if it was captured, and the status words' buffers (kept
// for later sets that fit).
struct BatchGraph {
    std::vector<const void *> key;  // plans and buffers
    unsigned long long epoch = 0;
    int device = -1, branches = 0, cap = 0;
    cudaGraphExec_t exec = nullptr;
    unsigned long long launches = 0;
    int *d_flags = nullptr;   // 2 per plan: overlap status, tensor-core pipeline status
    int **d_ptrs = nullptr;   // where those live
    std::vector<int *> h_ptrs;
    std::vector<int> h_flags;
    void drop() {
        if (exec) cudaGraphExecDestroy(exec);
        exec = nullptr;
        key.clear();
    }
    int reserve(int count, int dev) {
        if (cap >= count && device == dev) return PHF_OK;
        if (d_flags) cudaFree(d_flags);
        if (d_ptrs) cudaFree(d_ptrs);
        d_flags = nullptr;
        d_ptrs = nullptr;
        cap = 0;
        PHF_CUDA(cudaMalloc(&d_flags, 2 * (size_t)count * sizeof(int)));
        PHF_CUDA(cudaMalloc(&d_ptrs, 2 * (size_t)count * sizeof(int *)));
        cap = count;
        device = dev;
        return PHF_OK;
    }
};

std::mutex g_batch_mu;
BatchGraph g_batch;
unsigned long long g_plan_epoch = 0;  // advanced whenever a plan is destroyed

struct BatchStreams {
    int device = -1;
    cudaStream_t cap = nullptr, br[kMaxBranches] = {};
    cudaEvent_t fork = nullptr, join[kMaxBranches] = {};
} g_bs;

int batch_streams(int device) {
    if (g_bs.device == device && g_bs.cap) return PHF_OK;
    PHF_CUDA(cudaStreamCreateWithFlags(&g_bs.cap, cudaStreamNonBlocking));
    PHF_CUDA(cudaEventCreateWithFlags(&g_bs.fork, cudaEventDisableTiming));
    for (int i = 0; i < kMaxBranches; ++i) {
        PHF_CUDA(cudaStreamCreateWithFlags(&g_bs.br[i], cudaStreamNonBlocking));
        PHF_CUDA(cudaEventCreateWithFlags(&g_bs.join[i], cudaEventDisableTiming));
    }
    g_bs.device = device;
    return PHF_OK;
}

// The batch's launches over `nb` branches forked from and joined to `root`, then the status words of every plan.
int enqueue_batch(PlanImpl *const *plans, int count, const zc *const *d_c, zc *const *d_hs, zc *const *d_yg,
                  zc *const *d_yr, int nb, int **d_ptrs, int *d_flags,
                  cudaStream_t root) {
    int rc = PHF_OK;
    cudaError_t e = cudaEventRecord(g_bs.fork, root);
    for (int b = 0; b < nb && e == cudaSuccess; ++b) e = cudaStreamWaitEvent(g_bs.br[b], g_bs.fork, 0);
    for (int i = 0; i < count && rc == PHF_OK && e == cudaSuccess; ++i)
        rc = eval_enqueue(*plans[i], d_c[i], d_hs[i], d_yg[i], d_yr[i], g_bs.br[i % nb], true);
    for (int b = 0; b < nb && e == cudaSuccess; ++b) {
        e = cudaEventRecord(g_bs.join[b], g_bs.br[b]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(root, g_bs.join[b], 0);
    }
    if (rc == PHF_OK && e == cudaSuccess) {
        gather_flags_kernel<<<(2 * count + 255) / 256, 256, 0, root>>>(d_ptrs, 2 * count, d_flags);
        ++g_launches;
        e = cudaGetLastError();
    }
    if (rc == PHF_OK && e != cudaSuccess) {
        cudaGetLastError();
        set_error(PHF_ERR_CUDA, std::string("phf_eval_batch: ") + cudaGetErrorString(e));
        rc = PHF_ERR_CUDA;
    }
    return rc;
}

// Capture the batch into *exec (and its kernel count into *nl).
int capture_batch(PlanImpl *const *plans, int count, const zc *const *d_c, zc *const *d_hs, zc *const *d_yg,
                  zc *const *d_yr, int nb, int **d_ptrs, int *d_flags,
                  cudaGraphExec_t *exec, unsigned long long *nl) {
    const unsigned long long l0 = g_launches;
    PHF_CUDA(cudaStreamBeginCapture(g_bs.cap, cudaStreamCaptureModeRelaxed));
    const int rc = enqueue_batch(plans, count, d_c, d_hs, d_yg, d_yr, nb, d_ptrs, d_flags, g_bs.cap);
    cudaGraph_t g = nullptr;
    const cudaError_t e2 = cudaStreamEndCapture(g_bs.cap, &g);
    *nl = g_launches - l0;
    g_launches = l0;
    if (rc != PHF_OK || e2 != cudaSuccess || !g) {
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        if (rc != PHF_OK) return rc;
        set_error(PHF_ERR_CUDA, "phf_eval_batch: graph capture failed");
        return PHF_ERR_CUDA;
    }
    const cudaError_t e3 = cudaGraphInstantiate(exec, g, cudaGraphInstantiateFlagUseNodePriority);
    cudaGraphDestroy(g);
    if (e3 != cudaSuccess) {
        cudaGetLastError();
        set_error(PHF_ERR_CUDA, std::string("phf_eval_batch: graph instantiation failed: ") + cudaGetErrorString(e3));
        return PHF_ERR_CUDA;
    }
    return PHF_OK;
}

}  // namespace

void plan_destroyed() {
    std::lock_guard<std::mutex> lock(g_batch_mu);
    ++g_plan_epoch;
}

// All instances of a batch over concurrent branches: the first call for a set of plans and buffers launches them
// directly, the next one for the same set captures a CUDA graph, which later calls replay.  16 branches: 16
// instances of n = 16..96 take 23.8 ms direct and 23.6 replayed with 4, 8 or 16 (27.7 with one), 32 instances of
// n = 4..14 replay in 3.19, 2.79 and 2.66 ms and run directly in 4.3; capturing and timing the three counts for
// every set made two alternating sets cost 182 ms a call.
int plan_eval_batch(PlanImpl *const *plans, int count, const zc *const *d_c, zc *const *d_hs, zc *const *d_yg,
                    zc *const *d_yr, cudaStream_t st) {
    if (count <= 0) return PHF_OK;
    const int dev = plans[0]->device;
    for (int i = 0; i < count; ++i) {
        if (plans[i]->device != dev) {
            set_error(PHF_ERR_ARG, "phf_eval_batch: plans on different devices");
            return PHF_ERR_ARG;
        }
        if (plans[i]->cmplxconj == 2) {
            set_error(PHF_ERR_UNSUPPORTED, "phf_eval_batch: cmplxconj == 2 needs phf_plan_buildhsg");
            return PHF_ERR_UNSUPPORTED;
        }
    }
    PHF_CUDA(cudaSetDevice(dev));
    std::lock_guard<std::mutex> lock(g_batch_mu);
    if (g_prof.on) {  // kernel by kernel, one instance after another
        for (int i = 0; i < count; ++i) {
            PHF_TRY(eval_enqueue(*plans[i], d_c[i], d_hs[i], d_yg[i], d_yr[i], st, false));
            PHF_TRY(read_flag(*plans[i], st));
        }
        return PHF_OK;
    }
    std::vector<const void *> key;
    key.reserve(5 * (size_t)count);
    for (int i = 0; i < count; ++i) {
        key.push_back(plans[i]);
        key.push_back(d_c[i]);
        key.push_back(d_hs[i]);
        key.push_back(d_yg[i]);
        key.push_back(d_yr[i]);
    }
    BatchGraph &bg = g_batch;
    if (!(bg.key == key && bg.epoch == g_plan_epoch && bg.device == dev)) {
        // plans created with autotune are tuned (one direct evaluation each) before the batch is captured
        for (int i = 0; i < count; ++i)
            if (plans[i]->autotune && !plans[i]->tuned) {
                PHF_TRY(eval_enqueue(*plans[i], d_c[i], d_hs[i], d_yg[i], d_yr[i], st, false));
                PHF_TRY(read_flag(*plans[i], st));
            }
        bg.drop();
        PHF_TRY(batch_streams(dev));
        PHF_TRY(bg.reserve(count, dev));
        bg.h_ptrs.resize(2 * (size_t)count);
        for (int i = 0; i < count; ++i) {
            bg.h_ptrs[2 * i] = plans[i]->flag;
            bg.h_ptrs[2 * i + 1] = plans[i]->ozerr;
        }
        PHF_CUDA(cudaMemcpyAsync(bg.d_ptrs, bg.h_ptrs.data(), bg.h_ptrs.size() * sizeof(int *),
                                 cudaMemcpyHostToDevice, st));
        bg.branches = std::min(kMaxBranches, count);
        bg.h_flags.assign(2 * (size_t)count, 0);
        const int rc = enqueue_batch(plans, count, d_c, d_hs, d_yg, d_yr, bg.branches, bg.d_ptrs, bg.d_flags,
                                     st);
        if (rc != PHF_OK) {  // nothing of the batch is left running, whichever branch was not joined
            for (int b = 0; b < bg.branches; ++b) cudaStreamSynchronize(g_bs.br[b]);
            cudaStreamSynchronize(st);
            cudaGetLastError();
            return rc;
        }
        bg.key = std::move(key);
        bg.epoch = g_plan_epoch;
        bg.device = dev;
    } else {
        if (!bg.exec)
            PHF_TRY(capture_batch(plans, count, d_c, d_hs, d_yg, d_yr, bg.branches, bg.d_ptrs, bg.d_flags,
                                  &bg.exec, &bg.launches));
        PHF_CUDA(cudaGraphLaunch(bg.exec, st));
        g_launches += bg.launches;
    }
    PHF_CUDA(cudaMemcpyAsync(bg.h_flags.data(), bg.d_flags, bg.h_flags.size() * sizeof(int), cudaMemcpyDeviceToHost,
                             st));
    PHF_CUDA(cudaStreamSynchronize(st));
    for (int i = 0; i < count; ++i) {
        const int f = bg.h_flags[2 * i], oz = bg.h_flags[2 * i + 1];
        if (oz) {
            set_error(PHF_ERR_CUDA, "phf_eval_batch: instance " + std::to_string(i) +
                                        ": tensor-core GEMM pipeline wait timed out (code " + std::to_string(oz) + ")");
            return PHF_ERR_CUDA;
        }
        if (f & 1) {
            set_error(PHF_ERR_SINGULAR, "phf_eval_batch: instance " + std::to_string(i) + ": singular rotated overlap");
            return PHF_ERR_SINGULAR;
        }
        if (f & 2) {
            set_error(PHF_ERR_NONFINITE, "phf_eval_batch: instance " + std::to_string(i) + ": non-finite overlap");
            return PHF_ERR_NONFINITE;
        }
    }
    return PHF_OK;
}

int batch_branches() { return g_batch.branches; }

}  // namespace phf
