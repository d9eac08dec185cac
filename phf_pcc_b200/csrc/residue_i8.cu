// Exchange and Coulomb GEMMs on the tcgen05 int8 tensor cores through residues (an integer modular technique).
//
// A row a of one operand and a row b of the other are scaled by powers of two to integers of Euclidean
// norm at most 2^43, so that |a . b| <= 2^86 (Cauchy-Schwarz; rounding adds at most 2^-30 of that), which
// is less than half of P = 2^87.04, the product of eleven pairwise coprime moduli p_l <= 256.  Each integer is
// held as its eleven residues (one int8 plane per modulus); the tensor cores form the eleven products
// C_l = A_l B_l^T exactly in int32, and a . b is recovered from C_l mod p_l by the Chinese remainder
// theorem.  With the factor (P / p_l)^-1 mod p_l multiplied into the B residues beforehand,
//     (a . b) / P  =  sum_l (C_l mod p_l) / p_l   (mod 1),
// which is a sum of eleven 8-bit numbers times 64-bit fractions, the wrap-around of a 64-bit integer being
// the "mod 1" and its sign the sign of a . b; the fractions' rounding is 2^-52 of P.  The only error that
// matters is the rounding of the scaled integers: 2^-44 |a| |b| (rms), or about 2^-43.5 sqrt(k) of an entry
// of uncorrelated rows.  (Ozaki, Uchino, Imamura, "Ozaki Scheme II: A GEMM-oriented emulation of
// floating-point matrix multiplication using an integer modular technique", 2025.)
//
// Eleven int8 products replace the fifteen slice products of the five-digit form (ozaki_i8.cu), whose error
// on Gaussian data is 2.4e-11 of an entry (mostly the dropped products): 5e-12 here at k = 2080, 1.4e-11 at
// k = 20100.  Ten moduli would be sixteen times less exact, more than the digits allow.  Every tile here is a
// plain int8 product with one accumulator, so a CTA runs tiles of 256 x 256 (the digit form's five
// accumulators leave 128 x 96).
//
// The operands come in two parities (symmetric and antisymmetric halves of the exchange, see
// slice_density_sym_kernel in ozaki_i8.cu): plane = parity * 11 + l.  Both parities run over the pairs
// l <= j in row order (the antisymmetric operands hold zeros at l = j and in the rows i = k), so that one
// launch and one set of row and column indices serve both: 1 % more work than separate pair lists at n = 200.
//
// Operand layout: byte of (plane, row, k) at (plane rows_pad + row) kpad + k, kpad a multiple of 128.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "phf_internal.h"

namespace phf {

long long rz_pad_k(long long k);
long long rz_pad_rows(long long rows);

namespace {

constexpr int RZ_L = kRzModuli;          // moduli
constexpr int RZ_PLANES = 2 * RZ_L;      // two parities
constexpr int RZ_TILE = 256;             // output tile, rows and columns
constexpr int RZ_KPAD = 128;             // operand rows are padded to multiples of this
constexpr int RZ_BK = 64;                // k-block: one SWIZZLE_64B row
constexpr int RZ_STAGES = 7;
constexpr uint32_t RZ_OP = RZ_TILE * RZ_BK;             // 16 KB: one operand's rows of a stage
constexpr uint32_t RZ_STAGE = 2 * RZ_OP;
constexpr int RZ_EPI_WARPS = 8;
constexpr int RZ_THREADS = 64 + 32 * RZ_EPI_WARPS;      // producer, MMA issuer, epilogue
constexpr long long RZ_MAX_K = 65536;    // |C_l| < 2^30: int32 sums and the residue division stay exact
constexpr int RZ_NORM_BITS = 43;

struct RzTables {
    unsigned p[RZ_L];          // moduli
    int w[2][RZ_L];            // four signed bytes 2^{8 i} f mod p, i = 0..3 (f = 1, or the CRT factor)
    int c32[2][RZ_L];          // 2^32 f mod p, signed
    float pf[RZ_L], invf[RZ_L];  // p and 1 / p
    int inv38[RZ_L];           // ceil(2^38 / p)
    unsigned long long frac[RZ_L];  // round-down 2^64 / p
};

constexpr int rz_signed_mod(long long v, long long p) {  // representative in [-p/2, p/2], in int8
    long long r = ((v % p) + p) % p;
    if (2 * r >= p) r -= p;
    return (int)r;
}

constexpr RzTables rz_tables() {
    const unsigned ps[RZ_L] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223};
    RzTables t{};
    for (int l = 0; l < RZ_L; ++l) {
        const long long p = ps[l];
        long long q = 1;  // P / p mod p
        for (int m = 0; m < RZ_L; ++m)
            if (m != l) q = q * (long long)ps[m] % p;
        long long f = 1;
        while (q * f % p != 1) ++f;
        t.p[l] = ps[l];
        for (int s = 0; s < 2; ++s) {
            const long long g = s ? f : 1;
            long long pw = g % p;
            unsigned word = 0;
            for (int i = 0; i < 4; ++i) {
                word |= (unsigned)(rz_signed_mod(pw, p) & 0xff) << (8 * i);
                pw = pw * 256 % p;
            }
            t.w[s][l] = (int)word;
            t.c32[s][l] = rz_signed_mod(pw, p);
        }
        t.pf[l] = (float)p;
        t.invf[l] = 1.0f / (float)p;
        t.inv38[l] = (int)(((1LL << 38) + p - 1) / p);
        t.frac[l] = ~0ull / (unsigned long long)p + (~0ull % (unsigned long long)p == (unsigned long long)(p - 1));
    }
    return t;
}

__constant__ RzTables kRz = rz_tables();
constexpr double kRzUnit = 8635523.816796131;  // P / 2^64

// ------------------------------------------------------------------ scaling and residues
// Exponent s of a row with sum of squares ss and largest element mx over k elements: |row| 2^s <= 2^43.
// Squares that overflow or vanish are replaced by the bound mx sqrt(k).
__device__ __forceinline__ int rz_exponent(double ss, double mx, double k) {
    double norm = sqrt(ss);
    if (!(ss > 1e-280 && ss < 1e280)) norm = mx * sqrt(k);
    if (!(norm > 0.0) || !isfinite(norm)) return 0;
    int e;
    frexp(norm, &e);  // norm < 2^e
    return RZ_NORM_BITS - e;
}

struct RzScale {
    double f;   // 2^s when that is a normal double
    int s;
    bool fast;
};

__device__ __forceinline__ RzScale rz_scale(int s) {
    RzScale r;
    r.s = s;
    r.fast = s >= -1000 && s <= 1000;
    r.f = r.fast ? __hiloint2double((1023 + s) << 20, 0) : 1.0;
    return r;
}

// the integer rint(x 2^s) as a low 32-bit word (unsigned) and a high part (v = hi 2^32 + lo)
__device__ __forceinline__ void rz_integer(double x, const RzScale &sc, unsigned &lo, int &hi) {
    constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
    const double big = __dadd_rn(sc.fast ? x * sc.f : ldexp(x, sc.s), kRound);
    lo = (unsigned)__double2loint(big);
    hi = __double2hiint(big) - 0x43380000;
}

// residue of the integer for modulus l (side 0: the residue, side 1: times the CRT factor), an int8 in the
// low byte of the result.  The byte sum t = v f (mod p), |t| < 2^19 (|hi| <= 2^11, the low word's bytes times
// at most 127), is formed in the mantissa of 1.5 * 2^23 + t, and t - p rint(t / p) in FP32, exactly: the FP32
// pipe has twice the rate of the integer multiplies (with an integer high multiplication instead the
// density kernel took 1.07 ms against 0.89 for 800 points at n = 128).  t / p stays 1 / (2 p) away from a tie for odd p; for p = 256 either side
// of a tie is the same byte.
template <int SIDE>
__device__ __forceinline__ unsigned rz_byte(unsigned lo, int hi, int l) {
    constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
    int t = hi * kRz.c32[SIDE][l] + 0x4B400000;
    asm("dp4a.u32.s32 %0, %1, %2, %0;" : "+r"(t) : "r"(lo), "r"(kRz.w[SIDE][l]));
    const float m = __int_as_float(t), q = __fmaf_rn(m - kMagic, kRz.invf[l], kMagic) - kMagic;
    return (unsigned)__float_as_int(__fmaf_rn(-kRz.pf[l], q, m));
}

__device__ __forceinline__ unsigned rz_pack(unsigned b0, unsigned b1, unsigned b2, unsigned b3) {
    return __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
}

// ------------------------------------------------------------------ density operands
// Point w = blockIdx.y, element [r][q] of rho_w at rho[w ws + r rs + q] (rs, ws even), contraction index
// t = pair_le(l, j).  Blocks blockIdx.x = s = 0, 1: the exchange rows c = 8 w + 4 s + 2 t + part of both
// parities, the symmetric half (rho^{st}[l][j] + rho^{st}[j][l]) / 2 and the antisymmetric half, zero at l = j.
// Block 2: the Coulomb rows 2 w + part, the symmetric half of rho^{aa} + rho^{bb}.  Two passes: norms, then
// residues.  A thread takes two consecutive pairs and writes one 2-byte word per plane.  Spin rows are read
// as 32-byte loads (both t): a block per (s, t) with 16-byte loads moved twice the bytes and took 14.5 ms
// for 2432 points at n = 200, one block per point held 128 registers, two blocks an SM, and took 6 ms.
constexpr int RD_NT = 256;

__device__ __forceinline__ void ld_zc2(const zc *p, zc &a, zc &b) {  // two consecutive elements, 32 bytes
    asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(p));
}

// NV = 8: symmetric (t, part) 0..3 and antisymmetric 4..7 of spin row s; NV = 2: Coulomb (part)
template <int NV>
__device__ __forceinline__ void rd_values(const zc *R, long long rs, int s, int pr, double (&x)[NV]) {
    const int l = pr >> 16, j = pr & 0xffff;
    const zc *pv = R + (long long)(2 * l) * rs + 2 * j, *pu = R + (long long)(2 * j) * rs + 2 * l;
    zc v[2], u[2];
    if constexpr (NV == 8) {
        ld_zc2(pv + s * rs, v[0], v[1]);
        ld_zc2(pu + s * rs, u[0], u[1]);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            x[2 * t] = 0.5 * (v[t].x + u[t].x);
            x[2 * t + 1] = 0.5 * (v[t].y + u[t].y);
            x[4 + 2 * t] = 0.5 * (v[t].x - u[t].x);
            x[5 + 2 * t] = 0.5 * (v[t].y - u[t].y);
        }
    } else {
        const double2 a = __ldg(reinterpret_cast<const double2 *>(pv)), b = __ldg(reinterpret_cast<const double2 *>(pv + rs + 1));
        const double2 c = __ldg(reinterpret_cast<const double2 *>(pu)), d = __ldg(reinterpret_cast<const double2 *>(pu + rs + 1));
        x[0] = 0.5 * ((a.x + b.x) + (c.x + d.x));
        x[1] = 0.5 * ((a.y + b.y) + (c.y + d.y));
    }
}

// residue rows h at row0 + (h / 4) par + (h % 4) kpad, their exponents at es0[(h / 4) epar + h % 4]
template <int NV>
__device__ __forceinline__ void rd_block(int n, const int *__restrict__ pairs, const zc *R, long long rs, int s,
                                         long long kpad, long long plane, signed char *row0, long long par, int *es0,
                                         long long epar, double (*sh)[RD_NT / 32], int *exs) {
    const int kk = n * (n + 1) / 2, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double ss[NV];
#pragma unroll
    for (int h = 0; h < NV; ++h) ss[h] = 0.0;
    // two pairs in flight per thread, their table entries fetched one round ahead
    int p0 = __ldg(pairs + min((int)threadIdx.x, kk - 1)), p1 = __ldg(pairs + min((int)threadIdx.x + RD_NT, kk - 1));
    for (int e = threadIdx.x; e < kk; e += 2 * RD_NT) {
        double x[NV], y[NV];
        rd_values<NV>(R, rs, s, p0, x);
        rd_values<NV>(R, rs, s, p1, y);
        p0 = __ldg(pairs + min(e + 2 * RD_NT, kk - 1));
        p1 = __ldg(pairs + min(e + 3 * RD_NT, kk - 1));
        const double two = e + RD_NT < kk ? 1.0 : 0.0;
#pragma unroll
        for (int h = 0; h < NV; ++h) ss[h] = fma(x[h], x[h], fma(two * y[h], y[h], ss[h]));
    }
    bool odd = false;  // a sum of squares outside the normal range: the norms are bounded by the largest element
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        for (int o = 16; o > 0; o >>= 1) ss[h] += __shfl_xor_sync(0xffffffffu, ss[h], o);
        if (lane == 0) sh[h][wid] = ss[h];
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        double a = 0.0;
        for (int i = 0; i < RD_NT / 32; ++i) a += sh[h][i];
        ss[h] = a;
        odd = odd || !(a > 1e-280 && a < 1e280);
    }
    __syncthreads();
    if (odd) {  // the same decision in every thread
        double mx[NV];
#pragma unroll
        for (int h = 0; h < NV; ++h) mx[h] = 0.0;
        for (int e = threadIdx.x; e < kk; e += RD_NT) {
            double x[NV];
            rd_values<NV>(R, rs, s, __ldg(pairs + e), x);
#pragma unroll
            for (int h = 0; h < NV; ++h) mx[h] = fmax(mx[h], fabs(x[h]));
        }
#pragma unroll
        for (int h = 0; h < NV; ++h) {
            for (int o = 16; o > 0; o >>= 1) mx[h] = fmax(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], o));
            if (lane == 0) sh[h][wid] = mx[h];
        }
        __syncthreads();
    }
#pragma unroll
    for (int h = 0; h < NV; ++h)
        if (threadIdx.x == h) {
            double m = 0.0;
            for (int i = 0; i < RD_NT / 32 && odd; ++i) m = fmax(m, sh[h][i]);
            exs[h] = rz_exponent(ss[h], m, kk);
            es0[(h >> 2) * epar + (h & 3)] = exs[h];
        }
    __syncthreads();
    int q0 = __ldg(pairs + min(2 * (int)threadIdx.x, kk - 1)), q1 = __ldg(pairs + min(2 * (int)threadIdx.x + 1, kk - 1));
    for (int e0 = 2 * threadIdx.x; e0 < kpad; e0 += 2 * RD_NT) {
        double x[NV], y[NV];
        rd_values<NV>(R, rs, s, q0, x);
        rd_values<NV>(R, rs, s, q1, y);
        q0 = __ldg(pairs + min(e0 + 2 * RD_NT, kk - 1));
        q1 = __ldg(pairs + min(e0 + 2 * RD_NT + 1, kk - 1));
#pragma unroll
        for (int h = 0; h < NV; ++h) {
            const RzScale sc = rz_scale(exs[h]);
            unsigned lo0, lo1;
            int hi0, hi1;
            rz_integer(e0 < kk ? x[h] : 0.0, sc, lo0, hi0);
            rz_integer(e0 + 1 < kk ? y[h] : 0.0, sc, lo1, hi1);
            signed char *o = row0 + (h >> 2) * par + (h & 3) * kpad + e0;
#pragma unroll
            for (int l = 0; l < RZ_L; ++l, o += plane)
                *reinterpret_cast<unsigned short *>(o) =
                    (unsigned short)__byte_perm(rz_byte<0>(lo0, hi0, l), rz_byte<0>(lo1, hi1, l), 0x0040);
        }
    }
}

__global__ void __launch_bounds__(RD_NT, 3)
    residue_density_kernel(int n, const int *__restrict__ pairs, const zc *__restrict__ rho, long long rs,
                           long long ws, long long rows_k, long long rows_p, long long kpad, signed char *outk, int *ek,
                           signed char *outp, int *ep) {
    __shared__ double sh[8][RD_NT / 32];
    __shared__ int exs[8];
    const long long w = blockIdx.y, r = 8 * w + 4 * blockIdx.x;
    if (blockIdx.x < 2)
        rd_block<8>(n, pairs, rho + w * ws, rs, blockIdx.x, kpad, rows_k * kpad, outk + r * kpad, RZ_L * rows_k * kpad,
                    ek + r, rows_k, sh, exs);
    else
        rd_block<2>(n, pairs, rho + w * ws, rs, 0, kpad, rows_p * kpad, outp + 2 * w * kpad, 0, ep + 2 * w, 0, sh, exs);
}

// Rows of a real matrix (element (r, j) at A[r lda + j cs], j < k) as the CRT-side operand: a block per row.
__global__ void __launch_bounds__(RD_NT)
    residue_rows_kernel(int k, const double *__restrict__ A, long long lda, long long cs, long long rows_pad,
                        long long kpad, signed char *out, int *es) {
    __shared__ double sh[2][RD_NT / 32];
    const long long r = blockIdx.x;
    const double *a = A + r * lda;
    double ss = 0.0, mx = 0.0;
    for (int j = threadIdx.x; j < k; j += RD_NT) {
        const double x = a[j * cs];
        ss = fma(x, x, ss);
        mx = fmax(mx, fabs(x));
    }
    for (int o = 16; o > 0; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = ss;
        sh[1][threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    ss = mx = 0.0;
    for (int i = 0; i < RD_NT / 32; ++i) {
        ss += sh[0][i];
        mx = fmax(mx, sh[1][i]);
    }
    const int s = rz_exponent(ss, mx, k);
    if (threadIdx.x == 0) es[r] = s;
    const RzScale sc = rz_scale(s);
    const long long plane = rows_pad * kpad;
    for (long long j = threadIdx.x; j < kpad; j += RD_NT) {
        unsigned lo;
        int hi;
        rz_integer(j < k ? a[j * cs] : 0.0, sc, lo, hi);
#pragma unroll
        for (int l = 0; l < RZ_L; ++l) out[l * plane + r * kpad + j] = (signed char)rz_byte<1>(lo, hi, l);
    }
}

// ------------------------------------------------------------------ exchange rows
// Row r = pair (i, k) = pairs[t0 + r] of one panel from its Gram block, B[l][j] = G[(i - i0) n + l][(k - k0) n + j]:
// symmetric parity B[l][j] + B[j][l] (l < j), B[l][l] (l = j); antisymmetric parity B[l][j] - B[j][l] (zero
// at l = j, and in rows i = k), at contraction index pair_le(l, j).  The block goes through shared memory
// as 32 x 32 tile pairs, so that both B[l][j] and B[j][l] are read in rows, twice: norms, then residues.
constexpr int RE_NT = 256, RE_TP = 33;

__device__ __forceinline__ double rz_block_sum(double v, double *sh) {  // fixed order
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    for (int i = 0; i < RE_NT / 32; ++i) r += sh[i];
    __syncthreads();
    return r;
}
__device__ __forceinline__ double rz_block_max(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    for (int i = 0; i < RE_NT / 32; ++i) r = fmax(r, sh[i]);
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(RE_NT, 3)
    residue_ek_kernel(int n, int i0, int k0, const int *__restrict__ pairs, long long t0, const double *__restrict__ G,
                      long long ldg, long long rows_pad, long long kpad, signed char *out, int *es) {
    __shared__ double T1[32 * RE_TP], T2[32 * RE_TP];
    __shared__ double sh[RE_NT / 32];
    const long long r = blockIdx.x;
    const int pr = __ldg(pairs + t0 + r), i = pr >> 16, k = pr & 0xffff;
    const bool anti = i < k;
    const double *g = G + (long long)(i - i0) * n * ldg + (long long)(k - k0) * n;
    const int nt = (n + 31) / 32, lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const long long kk = (long long)n * (n + 1) / 2, plane = rows_pad * kpad;
    double ss = 0.0, sa = 0.0, ms = 0.0, ma = 0.0;
    RzScale scs = rz_scale(0), sca = rz_scale(0);
    signed char *os = out + r * kpad, *oa = os + RZ_L * plane;
    // the next tile pair's loads are in flight while a tile pair is worked on
    double f1[4], f2[4];
    auto fetch = [&](int lt, int jt) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int a = ty + 8 * q;
            const int l1 = lt * 32 + a, j1 = jt * 32 + lane, l2 = jt * 32 + a, j2 = lt * 32 + lane;
            f1[q] = (l1 < n && j1 < n) ? __ldg(g + (long long)l1 * ldg + j1) : 0.0;
            f2[q] = (jt != lt && l2 < n && j2 < n) ? __ldg(g + (long long)l2 * ldg + j2) : 0.0;
        }
    };
    fetch(0, 0);
    for (int pass = 0; pass < 2; ++pass) {
        for (int lt = 0; lt < nt; ++lt) {
            for (int jt = lt; jt < nt; ++jt) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int a = ty + 8 * q;
                    T1[a * RE_TP + lane] = f1[q];
                    T2[a * RE_TP + lane] = f2[q];
                }
                __syncthreads();
                if (jt + 1 < nt)
                    fetch(lt, jt + 1);
                else if (lt + 1 < nt)
                    fetch(lt + 1, lt + 1);
                else if (pass == 0)
                    fetch(0, 0);
                const double *U = (jt == lt) ? T1 : T2;  // U[b][a] = B[jt 32 + b][lt 32 + a]
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int a = ty + 8 * q, l = lt * 32 + a, j = jt * 32 + lane;
                    if (l <= j && j < n) {
                        const double x = T1[a * RE_TP + lane], y = U[lane * RE_TP + a];
                        const double sv = (l == j) ? x : x + y, av = anti ? x - y : 0.0;
                        if (pass == 0) {
                            ss = fma(sv, sv, ss);
                            sa = fma(av, av, sa);
                            ms = fmax(ms, fabs(sv));
                            ma = fmax(ma, fabs(av));
                        } else {
                            const long long t = (long long)l * n - (long long)l * (l - 1) / 2 + (j - l);
                            unsigned slo, alo;
                            int shi, ahi;
                            rz_integer(sv, scs, slo, shi);
                            rz_integer(av, sca, alo, ahi);
#pragma unroll
                            for (int m = 0; m < RZ_L; ++m) {
                                os[m * plane + t] = (signed char)rz_byte<1>(slo, shi, m);
                                oa[m * plane + t] = (signed char)rz_byte<1>(alo, ahi, m);
                            }
                        }
                    }
                }
                __syncthreads();
            }
        }
        if (pass == 0) {
            ss = rz_block_sum(ss, sh);
            sa = rz_block_sum(sa, sh);
            ms = rz_block_max(ms, sh);
            ma = rz_block_max(ma, sh);
            const int xs = rz_exponent(ss, ms, (double)kk), xa = rz_exponent(sa, ma, (double)kk);
            if (threadIdx.x == 0) {
                es[r] = xs;
                es[rows_pad + r] = xa;
            }
            scs = rz_scale(xs);
            sca = rz_scale(xa);
        }
    }
    for (long long e = kk + threadIdx.x; e < kpad; e += RE_NT) {
#pragma unroll
        for (int m = 0; m < RZ_L; ++m) os[m * plane + e] = oa[m * plane + e] = 0;
    }
}

// ------------------------------------------------------------------ GEMM
__device__ __forceinline__ uint32_t rz_smem(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void rz_mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(rz_smem(bar)), "r"(count));
}

__device__ __forceinline__ bool rz_mbar_try(uint32_t addr, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    return done != 0;
}

// Bounded wait (~2^31 cycles): false, with the code in *err, when it gives up.
__device__ __forceinline__ bool rz_wait(uint64_t *bar, uint32_t parity, int *err, int code) {
    const uint32_t addr = rz_smem(bar);
    if (rz_mbar_try(addr, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (rz_mbar_try(addr, parity)) return true;
        if (clock64() - t0 > (1LL << 31)) {
            atomicOr(err, code);
            return false;
        }
    }
}

__device__ __forceinline__ void rz_load(const CUtensorMap *map, uint64_t *bar, void *dst, int k, int row, int plane) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::
            "r"(rz_smem(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(rz_smem(bar)), "r"(k), "r"(row), "r"(plane)
        : "memory");
}

// K-major SWIZZLE_64B shared-memory matrix descriptor (8 rows x 64 B atoms)
__device__ __forceinline__ uint64_t rz_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

// D (128 x N in TMEM) += A B^T, int8 operands, one MMA of k = 32
__device__ __forceinline__ void rz_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

// one arrival once the MMAs issued so far complete
__device__ __forceinline__ void rz_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(rz_smem(bar)) : "memory");
}

__device__ __forceinline__ void rz_tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

struct RzArgs {
    int mt, nt, m, n;          // row and column tiles, rows and columns (rows of the B operand)
    int planes, kb, k32;       // planes, k-blocks, 32-element k-steps
    int group_m, a_row0, b_row0;  // raster group; first rows of the operands
    unsigned char *C;          // residues: (plane, row, column) at plane cplane + row ldc + column
    long long cplane, ldc;
    int *err;
};

// Tile t of the persistent loop: plane slowest, then column sweeps over groups of group_m row tiles (the
// tiles in flight share their operands in L2).
__device__ __forceinline__ void rz_tile(const RzArgs &a, int t, int &plane, int &m, int &n) {
    const int per = a.mt * a.nt;
    plane = t / per;
    const int L = t - plane * per, width = a.group_m * a.nt, first = (L / width) * a.group_m;
    const int gm = min(a.mt - first, a.group_m), rest = L % width;
    m = first + rest % gm;
    n = rest / gm;
}

// columns of the tile that starts at column c0, rounded up to a multiple of 32
__device__ __forceinline__ int rz_cols(int n, int c0) { return min(RZ_TILE, (n - c0 + 31) / 32 * 32); }

// C_l mod p_l (one byte, 0 .. p_l) of every plane.  One persistent CTA per SM runs tiles of 256 x 256: two
// 128 x 256 accumulators fill TMEM, k-blocks of 64 (16 KB of each operand) pass through a seven-stage ring,
// and each is two MMAs of 128 x 256 x 32 per row half.  At the full MMA rate operands would arrive at 64 B per
// cycle and SM (at 96 with 128 x 256 tiles).  Counters: tensor pipe 74 % active, operands read from DRAM once, L2 at
// 60 % of its throughput (n = 101, 312 points: 2496 rows x 5151 x k 5151 x 22, 2.77e15 operations per second);
// 58 % at k = 2080, where a tile's read-out is a larger part of it.  Epilogue:
// residues by one high multiplication, 8 warps; a row half is released as soon as it has been read, so the
// next tile's MMAs wait for half of the read-out (its loads are already in the ring).  A half that lies
// beyond the last row, and columns beyond the last one rounded up to 32, are not multiplied.  Measured: 3.0e15
// operations per second (n = 200, 7059 pair rows x 4864 density rows x k 20100: 10.1 ms; the digit form ran
// 2.8e15 and needs 15 / 11 of them).  CTA pairs (cta_group::2, 256 x 512 tiles, 48 B per cycle) took the same
// time, and hung beside other streams' kernels in a batch graph: one CTA per tile needs no cluster.
__global__ void __launch_bounds__(RZ_THREADS, 1)
    residue_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, RzArgs args) {
    extern __shared__ __align__(1024) unsigned char rz_raw[];
    unsigned char *smem = rz_raw;
    if ((rz_smem(rz_raw) & 1023u) != 0u) {  // the swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0) atomicOr(args.err, 16);
        return;
    }
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + RZ_STAGES * RZ_STAGE);
    uint64_t *empty = full + RZ_STAGES;
    uint64_t *acc_full = empty + RZ_STAGES;   // the tile's MMAs are complete
    uint64_t *acc_empty = acc_full + 1;       // [2] the epilogue has read row half h
    uint64_t *drained = acc_empty + 2;        // after a wait gave up: the MMAs issued are complete
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drained + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < RZ_STAGES; ++s) {
            rz_mbar_init(&full[s], 1);
            rz_mbar_init(&empty[s], 1);
        }
        rz_mbar_init(acc_full, 1);
        for (int h = 0; h < 2; ++h) rz_mbar_init(&acc_empty[h], RZ_EPI_WARPS);
        rz_mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(rz_smem(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const int ntile = args.mt * args.nt * args.planes;
    int loads = 0;  // k-blocks whose loads thread 0 has issued

    if (warp == 0) {
        if (lane == 0) {  // TMA producer
            int sg = 0;
            uint32_t ph = 1;  // the first lap finds every stage free
            for (int t = blockIdx.x; t < ntile && !*abort_flag; t += gridDim.x) {
                int plane, m, nn;
                rz_tile(args, t, plane, m, nn);
                const int arow = args.a_row0 + m * RZ_TILE, brow = args.b_row0 + nn * RZ_TILE;
                for (int kb = 0; kb < args.kb; ++kb) {
                    if (!rz_wait(&empty[sg], ph, args.err, 1)) {
                        *abort_flag = 1;
                        break;
                    }
                    unsigned char *dst = smem + sg * RZ_STAGE;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(rz_smem(&full[sg])),
                                 "r"(RZ_STAGE)
                                 : "memory");
                    rz_load(&tmA, &full[sg], dst, kb * RZ_BK, arow, plane);
                    rz_load(&tmB, &full[sg], dst + RZ_OP, kb * RZ_BK, brow, plane);
                    ++loads;
                    if (++sg == RZ_STAGES) {
                        sg = 0;
                        ph ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // MMA issuer
            int sg = 0, it = 0;
            uint32_t ph = 0;
            const uint32_t base = rz_smem(smem);
            for (int t = blockIdx.x; t < ntile && !*abort_flag; t += gridDim.x, ++it) {
                int plane, m, nn;
                rz_tile(args, t, plane, m, nn);
                // int32 accumulator, s8 operands, K-major, M = 128, N = columns
                const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) |
                                       ((uint32_t)(rz_cols(args.n, nn * RZ_TILE) >> 3) << 17) | (8u << 24);
                const bool low = args.m - m * RZ_TILE > 128;  // the tile has a second row half
                const uint32_t free_ph = (uint32_t)((it & 1) ^ 1);
                bool ok = rz_wait(&acc_empty[0], free_ph, args.err, 8);
                for (int kb = 0; kb < args.kb && ok; ++kb) {
                    ok = rz_wait(&full[sg], ph, args.err, 2);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t dA = rz_desc(base + sg * RZ_STAGE), dB = rz_desc(base + sg * RZ_STAGE + RZ_OP);
                    const bool two = args.k32 - 2 * kb > 1;
                    rz_mma(tmem, dA, dB, idesc, kb ? 1u : 0u);
                    if (two) rz_mma(tmem, dA + 2, dB + 2, idesc, 1u);
                    if (kb == 0) {  // the second half's previous tile has been read
                        ok = rz_wait(&acc_empty[1], free_ph, args.err, 8);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                    if (low) {
                        const uint64_t dA1 = rz_desc(base + sg * RZ_STAGE + RZ_OP / 2);
                        rz_mma(tmem + RZ_TILE, dA1, dB, idesc, kb ? 1u : 0u);
                        if (two) rz_mma(tmem + RZ_TILE, dA1 + 2, dB + 2, idesc, 1u);
                    }
                    rz_commit(&empty[sg]);
                    if (++sg == RZ_STAGES) {
                        sg = 0;
                        ph ^= 1u;
                    }
                }
                if (!ok) {
                    *abort_flag = 1;
                    break;
                }
                rz_commit(acc_full);
            }
        }
    } else {
        // epilogue: TMEM lane quarter warp % 4, every other 32 columns
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
        int it = 0;
        for (int t = blockIdx.x; t < ntile && !*abort_flag; t += gridDim.x, ++it) {
            int plane, m, nn;
            rz_tile(args, t, plane, m, nn);
            const int l = plane % RZ_L;
            if (!rz_wait(acc_full, it & 1, args.err, 4)) {
                *abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int p = (int)kRz.p[l], inv = kRz.inv38[l];
            const int ncol = rz_cols(args.n, nn * RZ_TILE), nh = args.m - m * RZ_TILE > 128 ? 2 : 1;
            unsigned char *row = args.C + plane * args.cplane +
                                 (long long)(m * RZ_TILE + quarter * 32 + lane) * args.ldc + nn * RZ_TILE;
#pragma unroll 1
            for (int h = 0; h < 2; ++h, row += 128 * args.ldc) {
#pragma unroll 1
                for (int c = half * 32; c < ncol && h < nh; c += 64) {
                    uint32_t v[32], o[8];
                    rz_tmem_ld32(lane_base + (uint32_t)(h * RZ_TILE + c), v);
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const int x = (int)v[j];
                        v[j] = (uint32_t)(x - (__mulhi(x, inv) >> 6) * p);  // x mod p in 0 .. p (|x| <= 2^30)
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        o[j] = __byte_perm(__byte_perm(v[4 * j], v[4 * j + 1], 0x0040),
                                           __byte_perm(v[4 * j + 2], v[4 * j + 3], 0x0040), 0x5410);
                    uint4 *d = reinterpret_cast<uint4 *>(row + c);
                    d[0] = make_uint4(o[0], o[1], o[2], o[3]);
                    d[1] = make_uint4(o[4], o[5], o[6], o[7]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(rz_smem(&acc_empty[h])) : "memory");
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag) {
        // a wait gave up: MMAs and loads may be in flight, and TMEM and shared memory must outlive them
        if (warp == 1 && lane == 0) {
            rz_commit(drained);
            rz_wait(drained, 0, args.err, 32);
        }
        if (threadIdx.x == 0)
            for (int s = 0; s < min(loads, RZ_STAGES); ++s)  // the last load into each stage
                rz_wait(&full[s], (uint32_t)((loads - 1 - s) / RZ_STAGES & 1), args.err, 32);
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

// ------------------------------------------------------------------ reconstruction into Gamma
// a 64-bit fraction of P as a double in units of P / 2^64
__device__ __forceinline__ double rz_double(unsigned long long y) {
    const double hi = __hiloint2double(0x43300000, (int)((unsigned)(y >> 32) ^ 0x80000000u)) - 4503601774854144.0;
    const double lo = __hiloint2double(0x43300000, (int)(unsigned)y) - 4503599627370496.0;
    return fma(hi, 4294967296.0, lo);
}

// NP products (consecutive bytes of plane 0 at src, planes `plane` apart; NP = 2 or 4) at scales 2^x
template <int NP>
__device__ __forceinline__ void rz_values(const unsigned char *src, long long plane, const int (&x)[NP], double (&d)[NP]) {
    unsigned word[RZ_L];
#pragma unroll
    for (int l = 0; l < RZ_L; ++l)
        word[l] = NP == 4 ? __ldg(reinterpret_cast<const unsigned *>(src + l * plane))
                          : (unsigned)__ldg(reinterpret_cast<const unsigned short *>(src + l * plane));
#pragma unroll
    for (int v = 0; v < NP; ++v) {
        unsigned long long y = 0;
#pragma unroll
        for (int l = 0; l < RZ_L; ++l) y += (unsigned long long)((word[l] >> (8 * v)) & 0xffu) * kRz.frac[l];
        const double u = rz_double(y) * kRzUnit;
        d[v] = (x[v] > -1000 && x[v] < 1000) ? u * __hiloint2double((1023 + x[v]) << 20, 0) : ldexp(u, x[v]);
    }
}

__device__ __forceinline__ void st_zc2(double2 *p, double a, double b, double c, double d) {  // 32-byte store
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// The Fock matrix of the panel's pairs (i, k) and points: F_w[2i + s][2k + t] = delta_st (J + h)_ik - (KS + KA),
// F_w[2k + s][2i + t] = delta_st (J + h)_ik - (KS - KA), from the residues of the exchange product C (row
// 8 wl + 4 s + 2 t + part of the wl-th point, column r = pair; parity planes) and of the Coulomb product CJ (row
// 2 wl + part).  A thread takes two consecutive pairs of one point and spin row s (a 2-byte word per plane and
// row); a pair's two values of t are one 32-byte store.  Bound: 198 residue bytes read and 128 bytes written
// per pair and point, and 45 instructions per value for the weighted sums; four pairs a thread needed 108
// registers and ran at 0.4 instructions per cycle and scheduler, waiting for loads.
constexpr int RG_NT = 256;
__global__ void __launch_bounds__(RG_NT, 3)
    residue_gamma_kernel(int n, int rows, const int *__restrict__ pairs, const unsigned char *__restrict__ C,
                         long long cplane, long long ldc, const unsigned char *__restrict__ CJ, long long jplane,
                         int npts, const int *__restrict__ ec, long long ec_par, const int *__restrict__ er,
                         long long er_par, const int *__restrict__ ed, const int *__restrict__ ej,
                         const double *__restrict__ h, zc *Gam) {
    const int lane = threadIdx.x & 31;
    const int r0 = (blockIdx.x * 32 + lane) * 2;
    const int ws = blockIdx.y * (RG_NT / 32) + (threadIdx.x >> 5), wl = ws >> 1, s = ws & 1;
    if (r0 >= rows || wl >= npts) return;
    const int M = 2 * n;
    double out[2][2][2][2];  // parity, t, part, pair
#pragma unroll
    for (int par = 0; par < 2; ++par)
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const int c = 8 * wl + 4 * s + 2 * t + part;
                const int e = __ldg(ec + par * ec_par + c);
                int x[2];
#pragma unroll
                for (int v = 0; v < 2; ++v) x[v] = -(e + __ldg(er + par * er_par + min(r0 + v, rows - 1)));
                rz_values<2>(C + par * RZ_L * cplane + (long long)c * ldc + r0, cplane, x, out[par][t][part]);
            }
    double jv[2][2];
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        const int e = __ldg(ed + 2 * wl + part);
        int x[2];
#pragma unroll
        for (int v = 0; v < 2; ++v) x[v] = -(e + __ldg(ej + min(r0 + v, rows - 1)));
        rz_values<2>(CJ + (long long)(2 * wl + part) * ldc + r0, jplane, x, jv[part]);
    }
    double2 *G = reinterpret_cast<double2 *>(Gam) + (long long)wl * M * M;
#pragma unroll
    for (int v = 0; v < 2; ++v) {
        if (r0 + v >= rows) break;
        const int pr = __ldg(pairs + r0 + v), i = pr >> 16, k = pr & 0xffff;
        const double jr = jv[0][v] + (h ? __ldg(h + (long long)i * n + k) : 0.0), ji = jv[1][v];
        const double dr[2] = {s == 0 ? jr : 0.0, s == 1 ? jr : 0.0}, di[2] = {s == 0 ? ji : 0.0, s == 1 ? ji : 0.0};
        double a[4], b[4];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const double sr = out[0][t][0][v], si = out[0][t][1][v], ar = out[1][t][0][v], ai = out[1][t][1][v];
            a[2 * t] = dr[t] - (sr + ar);
            a[2 * t + 1] = di[t] - (si + ai);
            b[2 * t] = dr[t] - (sr - ar);
            b[2 * t + 1] = di[t] - (si - ai);
        }
        st_zc2(G + (long long)(2 * i + s) * M + 2 * k, a[0], a[1], a[2], a[3]);
        if (i != k) st_zc2(G + (long long)(2 * k + s) * M + 2 * i, b[0], b[1], b[2], b[3]);
    }
}

// Row r = 2 w + part of d = (Cholesky operand) . P from its residues, as the plain-side operand of the
// Coulomb product (contraction over the Cholesky vectors): a block per row, the values computed once per pass.
__global__ void __launch_bounds__(RD_NT)
    residue_coulomb_kernel(int L, const unsigned char *__restrict__ C, long long cplane, long long ldc,
                           const int *__restrict__ ep, const int *__restrict__ eb, long long rows_pad, long long kpad,
                           signed char *out, int *es) {
    __shared__ double sh[2][RD_NT / 32];
    const long long r = blockIdx.x;
    const unsigned char *src = C + r * ldc;
    const int e = ep[r];
    auto value = [&](int j, double (&d)[4]) {  // j a multiple of 4
        int x[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) x[v] = -(e + __ldg(eb + min(j + v, L - 1)));
        rz_values<4>(src + j, cplane, x, d);
    };
    double ss = 0.0, mx = 0.0;
    for (int j = 4 * threadIdx.x; j < L; j += 4 * RD_NT) {
        double d[4];
        value(j, d);
#pragma unroll
        for (int v = 0; v < 4; ++v)
            if (j + v < L) {
                ss = fma(d[v], d[v], ss);
                mx = fmax(mx, fabs(d[v]));
            }
    }
    for (int o = 16; o > 0; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = ss;
        sh[1][threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    ss = mx = 0.0;
    for (int i = 0; i < RD_NT / 32; ++i) {
        ss += sh[0][i];
        mx = fmax(mx, sh[1][i]);
    }
    const int s = rz_exponent(ss, mx, L);
    if (threadIdx.x == 0) es[r] = s;
    const RzScale sc = rz_scale(s);
    const long long plane = rows_pad * kpad;
    for (int j = 4 * threadIdx.x; j < kpad; j += 4 * RD_NT) {
        double d[4] = {0.0, 0.0, 0.0, 0.0};
        if (j < L) value(j, d);
        unsigned lo[4];
        int hi[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) rz_integer(j + v < L ? d[v] : 0.0, sc, lo[v], hi[v]);
#pragma unroll
        for (int l = 0; l < RZ_L; ++l)
            *reinterpret_cast<unsigned *>(out + l * plane + r * kpad + j) =
                rz_pack(rz_byte<0>(lo[0], hi[0], l), rz_byte<0>(lo[1], hi[1], l), rz_byte<0>(lo[2], hi[2], l),
                        rz_byte<0>(lo[3], hi[3], l));
    }
}

// ------------------------------------------------------------------ host side
PFN_cuTensorMapEncodeTiled_v12000 rz_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// (k bytes, rows, planes) of an operand, boxes of one k-block x 256 rows
int rz_map(CUtensorMap *map, const signed char *base, long long kpad, long long rows_pad, int planes) {
    auto enc = rz_encoder();
    if (!enc) {
        set_error(PHF_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
        return PHF_ERR_CUDA;
    }
    cuuint64_t dims[3] = {(cuuint64_t)kpad, (cuuint64_t)rows_pad, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)kpad, (cuuint64_t)(kpad * rows_pad)};
    cuuint32_t box[3] = {(cuuint32_t)RZ_BK, (cuuint32_t)RZ_TILE, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<signed char *>(base), dims, strides, box,
                           estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error(PHF_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
        return PHF_ERR_CUDA;
    }
    return PHF_OK;
}

constexpr size_t kRzSmem = RZ_STAGES * RZ_STAGE + (2 * RZ_STAGES + 4) * 8 + 8;

// C_l mod p_l of A rows [a_row0, a_row0 + m) and B rows [b_row0, b_row0 + n) for every plane, contraction
// length k, into C (rz_pad_rows(m) rows of ldc = rz_pad_rows(n) bytes per plane).
int rz_gemm(long long m, long long n, long long k, int planes, const signed char *A, long long a_rows, int a_row0,
            const signed char *B, long long b_rows, int b_row0, unsigned char *C, int *err, int cls, cudaStream_t st) {
    const long long kpad = rz_pad_k(k);
    CUtensorMap ta, tb;
    PHF_TRY(rz_map(&ta, A, kpad, a_rows, planes));
    PHF_TRY(rz_map(&tb, B, kpad, b_rows, planes));
    RzArgs a;
    a.ldc = rz_pad_rows(n);
    a.mt = (int)(rz_pad_rows(m) / RZ_TILE);
    a.nt = (int)(a.ldc / RZ_TILE);
    a.m = (int)m;
    a.n = (int)n;
    a.planes = planes;
    a.kb = (int)((k + RZ_BK - 1) / RZ_BK);
    a.k32 = (int)((k + 31) / 32);
    a.group_m = 8;
    a.a_row0 = a_row0;
    a.b_row0 = b_row0;
    a.C = C;
    a.cplane = (long long)a.mt * RZ_TILE * a.ldc;
    a.err = err;
    PHF_CUDA(cudaFuncSetAttribute((const void *)residue_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kRzSmem));
    const long long tiles = (long long)a.mt * a.nt * a.planes;
    {
        ProfScope prof(st, cls);
        residue_gemm_kernel<<<(unsigned)std::min<long long>(tiles, 148), RZ_THREADS, kRzSmem, st>>>(ta, tb, a);
    }
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

}  // namespace

long long rz_pad_k(long long k) { return (k + RZ_KPAD - 1) / RZ_KPAD * RZ_KPAD; }
long long rz_pad_rows(long long rows) { return (rows + RZ_TILE - 1) / RZ_TILE * RZ_TILE; }
bool rz_ok(int n, int L) { return n >= 2 && L >= 1 && L <= RZ_MAX_K && (long long)n * (n + 1) / 2 <= RZ_MAX_K; }
size_t rz_operand_bytes(int planes, long long rows, long long k) {
    return (size_t)planes * (size_t)rows * (size_t)rz_pad_k(k);
}
size_t rz_product_bytes(int planes, long long a_rows, long long b_rows) {
    return (size_t)planes * (size_t)rz_pad_rows(a_rows) * (size_t)rz_pad_rows(b_rows);
}

int rz_density(int n, int bc, const int *pairs, const zc *rho, long long rs, long long ws, long long rows_k,
               signed char *outk, int *ek, long long rows_p, signed char *outp, int *ep, cudaStream_t st) {
    if (bc < 1 || bc > 65535 || 8LL * bc > rows_k || 2LL * bc > rows_p || (rs & 1) || (ws & 1)) {
        set_error(PHF_ERR_ARG, "rz_density: rows outside the operands");
        return PHF_ERR_ARG;
    }
    ProfScope prof(st, PROF_MEMORY);
    residue_density_kernel<<<dim3(3, (unsigned)bc), RD_NT, 0, st>>>(n, pairs, rho, rs, ws, rows_k, rows_p,
                                                                    rz_pad_k((long long)n * (n + 1) / 2), outk, ek,
                                                                    outp, ep);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int rz_rows(long long rows, int k, const double *A, long long lda, long long cs, signed char *out, int *es,
            cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    residue_rows_kernel<<<(unsigned)rows, RD_NT, 0, st>>>(k, A, lda, cs, rows, rz_pad_k(k), out, es);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int rz_exchange_rows(int n, int i0, int ipanel, int k0, const int *pairs, const double *G, long long ldg,
                     long long rows_pad, signed char *out, int *es, cudaStream_t st) {
    const long long nn = n, rows = ipanel * (nn - i0) - (long long)ipanel * (ipanel - 1) / 2;
    if (n < 2 || i0 < 0 || ipanel < 1 || i0 + ipanel > n || k0 < 0 || k0 > i0 || rows > rows_pad ||
        ldg < (nn - k0) * nn) {
        set_error(PHF_ERR_ARG, "rz_exchange_rows: panel rows outside the operand or a short Gram block");
        return PHF_ERR_ARG;
    }
    ProfScope prof(st, PROF_MEMORY);
    residue_ek_kernel<<<(unsigned)rows, RE_NT, 0, st>>>(n, i0, k0, pairs, i0 * nn - (long long)i0 * (i0 - 1) / 2, G,
                                                        ldg, rows_pad, rz_pad_k(nn * (nn + 1) / 2), out, es);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int rz_coulomb_d(int n, int L, int bc, const signed char *P, long long rows_p, const int *ep, const signed char *B1,
                 const int *e1, unsigned char *C, signed char *D, int *ed, int *err, cudaStream_t st) {
    if (!rz_ok(n, L) || bc < 1 || 2LL * bc > rows_p) {
        set_error(PHF_ERR_ARG, "rz_coulomb_d: rows outside the operands");
        return PHF_ERR_ARG;
    }
    PHF_TRY(rz_gemm(2LL * bc, L, (long long)n * (n + 1) / 2, RZ_L, P, rows_p, 0, B1, L, 0, C, err, PROF_JK, st));
    const long long ldc = rz_pad_rows(L);
    ProfScope prof(st, PROF_MEMORY);
    residue_coulomb_kernel<<<(unsigned)(2 * bc), RD_NT, 0, st>>>(L, C, rz_pad_rows(2LL * bc) * ldc, ldc, ep, e1, rows_p,
                                                                 rz_pad_k(L), D, ed);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int rz_fock(const RzFock &f, cudaStream_t st) {
    const long long kk = (long long)f.n * (f.n + 1) / 2;
    if (!rz_ok(f.n, f.L) || f.pts < 1 || f.rows < 1 || f.rows > f.e_rows || f.w0 < 0 ||
        8LL * (f.w0 + f.pts) > f.k_rows || 2LL * (f.w0 + f.pts) > f.d_rows || f.pair0 < 0 || f.pair0 + f.rows > kk) {
        set_error(PHF_ERR_ARG, "rz_fock: rows outside the operands");
        return PHF_ERR_ARG;
    }
    PHF_TRY(rz_gemm(2LL * f.pts, f.rows, f.L, RZ_L, f.D, f.d_rows, 2 * f.w0, f.B2, kk, f.pair0, f.CJ, f.err, PROF_JK, st));
    PHF_TRY(rz_gemm(8LL * f.pts, f.rows, kk, RZ_PLANES, f.K, f.k_rows, 8 * f.w0, f.E, f.e_rows, 0, f.C, f.err, PROF_JK,
                    st));
    const long long ldc = rz_pad_rows(f.rows);
    ProfScope prof(st, PROF_MEMORY);
    residue_gamma_kernel<<<dim3((unsigned)((f.rows + 63) / 64), (unsigned)((2 * f.pts + RG_NT / 32 - 1) / (RG_NT / 32))),
                           RG_NT, 0, st>>>(f.n, f.rows, f.pairs + f.pair0, f.C, rz_pad_rows(8LL * f.pts) * ldc, ldc,
                                           f.CJ, rz_pad_rows(2LL * f.pts) * ldc, f.pts, f.ek + 8LL * f.w0, f.k_rows,
                                           f.ee, f.e_rows, f.ed + 2LL * f.w0, f.e2 + f.pair0, f.h, f.Gam);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

}  // namespace phf
