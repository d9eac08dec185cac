// FP64 strided batched complex GEMM: the building block of the plain FP64 form.
//
// C[b] = alpha * A[b] * B[b] + beta * C[b] with every operand given as a strided view
// (row stride, column stride, two batch strides, optional per-batch offsets), so that
// transposes, conjugate transposes and the column-blocked layouts of the grid-point
// batches need no copies.  A may be real (real x complex products: Cholesky vectors and
// the one-electron matrix applied to complex orbitals).
//
// Tiling: BM x BN output tile per CTA of (BM / 32) (BN / 16) warps (64 x 64, 128 x 32 and 32 x 128 on
// 8 warps; 32 x 112 on 7 and 64 x 112 on 14 for products with 97..112 output columns, such as the
// per-point products with N = 100 orbitals; 32 x 32 on 2 for small products), k-step 16, the k-tiles
// staged by cp.async.
// The products run on the FP64 tensor cores (mma.sync m8n8k4 .f64; the larger shapes reach the same 37 TFLOP/s
// in isolation): each warp owns a 32 x 16 block of the tile as 4 x 2 blocks of 8 x 8, and a complex product
// is four real MMAs (re re, -im im, re im, im re), two for a real A.  Bound: the FP64 tensor pipe for long k
// (real 2080 x 2080 by complex 2080 x 3200: 2.19 -> 1.80 ms, 30.8 TFLOP/s, when the address arithmetic left
// the k loop), latency for the small products (n = 20, 112 points: GEMMs 230 -> 145 us of an evaluation, and 87 with
// the sums of small grids in groups).
#include <type_traits>

#include "phf_internal.h"

namespace phf {

namespace {

constexpr int BK = 16;

template <int BM, int BN>
__host__ __device__ constexpr int zg_threads() { return (BM / 32) * (BN / 16) * 32; }
template <int BM, int BN>
__host__ __device__ constexpr int zg_min_blocks() { return zg_threads<BM, BN>() <= 64 ? 6 : (zg_threads<BM, BN>() <= 128 ? 4 : (zg_threads<BM, BN>() <= 256 ? 2 : 1)); }

// Row pitches of the staged tiles (elements).  A 16-byte fragment load is served eight lanes at a time, and
// lanes (fk, fr) of such a group read row kk + fk, column c + fr: with a pitch of 2 mod 8 they land on distinct
// bank quadruples (one more than the tile, as before, made half of all shared-memory wavefronts conflicts).
// An 8-byte load is served sixteen lanes at a time: 4 mod 16.
template <bool AREAL>
__host__ __device__ constexpr int zg_pitch_a(int bm) { return AREAL ? bm + 4 : bm + 2; }
__host__ __device__ constexpr int zg_pitch_b(int bn) { return bn + 2; }

template <bool AREAL>
struct ATile {
    using T = typename std::conditional<AREAL, double, zc>::type;
};

// D (8 x 8) += A (8 x 4, row-major) B (4 x 8, column-major), FP64.  Lane l holds A[l/4][l%4],
// B[l%4][l/4] and D[l/4][2 (l%4) + {0, 1}].
__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async(uint32_t dst, const void *src, int bytes_valid, int size) {
    if (size == 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes_valid) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes_valid) : "memory");
}

// Shared-memory stages of the k loop (cp.async pipeline): three for the 64 x 64 and the 112-column
// tiles, two for the narrow tiles (their products are mostly k = 32, two k-tiles; two stages let two
// CTAs share an SM).
template <int BM, int BN>
__host__ __device__ constexpr int zg_stages() { return (BM == BN || BN == 112) ? 3 : 2; }

template <bool AREAL, int BM, int BN>
__host__ __device__ constexpr size_t zg_smem_bytes() {
    return (size_t)zg_stages<BM, BN>() * BK *
           (zg_pitch_a<AREAL>(BM) * (AREAL ? sizeof(double) : sizeof(zc)) + zg_pitch_b(BN) * sizeof(zc));
}

// BM x BN output tile, 256 threads = 8 warps of 32 x 16 (warp w: rows 32 (w / (BN/16)), columns
// 16 (w % (BN/16))).  64 x 64 serves general shapes; 128 x 32 the narrow per-point products
// (N <= 32 columns), 32 x 128 the N-row products bra^H Y and bra^H F X (m = N <= 32) over all
// points of a chunk.  Tiles of A and B reach shared memory by element-wise cp.async (16 bytes a
// complex element, 8 a real one; out-of-range elements are zero-filled) through zg_stages stages;
// conjugation is applied when fragments are read.  A real B (only the exchange-matrix build) is
// loaded with plain loads into the same stages.
//
// KS > 1: KS groups of such threads, each with its own stages, take consecutive ranges of k-tiles, and the groups'
// accumulators are added through shared memory in the groups' order.  For grids that leave the chip idle, where a
// tile's k loop is a chain of load and multiply latencies on one or two of the multiprocessor's four schedulers.
template <bool AREAL, int BM, int BN, int KS = 1>
__global__ void __launch_bounds__(KS *zg_threads<BM, BN>(), KS == 1 ? zg_min_blocks<BM, BN>() : 1)
    zgemm_kernel(int m, int n, int k, int nb0, int ntn, zc alpha, View A, View B, zc beta, OutView C,
                 const long long *__restrict__ offs) {
    using TA = typename ATile<AREAL>::T;
    constexpr int WARPS_N = BN / 16;
    constexpr int NT = zg_threads<BM, BN>();
    static_assert(BM % 32 == 0 && BN % 16 == 0, "tile/warp mismatch");
    // elements loaded per thread and k-tile (the last round partial when NT does not divide the tile)
    constexpr int LA = (BM * BK + NT - 1) / NT, LB = (BN * BK + NT - 1) / NT;
    constexpr int PA = zg_pitch_a<AREAL>(BM), PB = zg_pitch_b(BN);
    constexpr int ZG_STAGES = zg_stages<BM, BN>();
    extern __shared__ __align__(16) unsigned char zg_smem[];
    const int group = KS == 1 ? 0 : (int)threadIdx.x / NT;
    unsigned char *stages = zg_smem + (KS == 1 ? 0 : group * zg_smem_bytes<AREAL, BM, BN>());
    TA *As = reinterpret_cast<TA *>(stages);                                      // [stage][kk][i]
    zc *Bs = reinterpret_cast<zc *>(stages + (size_t)ZG_STAGES * BK * PA * sizeof(TA));  // [stage][kk][j]

    const int tid = threadIdx.x - group * NT, lane = tid & 31, warp = tid >> 5;
    const int wr = (warp / WARPS_N) * 32, wc = (warp % WARPS_N) * 16;  // warp block within the tile
    const int fr = lane >> 2, fk = lane & 3;                            // fragment row / k of this lane
    const long long bz = blockIdx.x / ntn;
    const int tn = blockIdx.x - bz * ntn;
    const int row0 = blockIdx.y * BM, col0 = tn * BN;
    const long long b0 = bz % nb0, b1 = bz / nb0;
    long long oa = b0 * A.bs0 + b1 * A.bs1, ob = b0 * B.bs0 + b1 * B.bs1, oc = b0 * C.bs0 + b1 * C.bs1;
    if (offs) {
        oa += offs[3 * bz];
        ob += offs[3 * bz + 1];
        oc += offs[3 * bz + 2];
    }
    const bool a_mfast = (A.rs == 1);  // element order of the A tile loads
    const bool b_nfast = (B.cs == 1);
    const int nkt_all = (k + BK - 1) / BK;
    const int per = (nkt_all + KS - 1) / KS, kt0 = group * per, nkt = max(0, min(per, nkt_all - kt0));
    // Each thread's r-th element of a tile is dA rows (or k's) and a fixed pointer and shared-memory step after
    // its first; the pointers advance by one k-tile per load_stage call (addresses from scratch for every
    // element were three of five instructions of the k loop).
    constexpr int RA = NT / BM, KA = NT / BK, RB = NT / BN;
    static_assert(NT % BM == 0 && NT % BN == 0 && NT % BK == 0, "tile loads");
    const int ai = a_mfast ? tid % BM : tid / BK, ak = a_mfast ? tid / BM : tid % BK;
    const int bj = b_nfast ? tid % BN : tid / BK, bk = b_nfast ? tid / BN : tid % BK;
    const int bsz = B.real ? (int)sizeof(double) : (int)sizeof(zc);
    const unsigned char *pa = reinterpret_cast<const unsigned char *>(A.p) +
                              (oa + (long long)(row0 + ai) * A.rs + (long long)(kt0 * BK + ak) * A.cs) *
                                  (long long)sizeof(TA);
    const unsigned char *pb = reinterpret_cast<const unsigned char *>(B.p) +
                              (ob + (long long)(kt0 * BK + bk) * B.rs + (long long)(col0 + bj) * B.cs) * bsz;
    const long long astep = (long long)(a_mfast ? RA * A.cs : KA * A.rs) * (long long)sizeof(TA),
                    bstep = (long long)(b_nfast ? RB * B.rs : KA * B.cs) * bsz;
    const uint32_t sa0 = (uint32_t)__cvta_generic_to_shared(As) + (uint32_t)((ak * PA + ai) * sizeof(TA)),
                   sar = (uint32_t)((a_mfast ? RA * PA : KA) * sizeof(TA));
    const uint32_t sb0 = (uint32_t)__cvta_generic_to_shared(Bs) + (uint32_t)((bk * PB + bj) * sizeof(zc)),
                   sbr = (uint32_t)((b_nfast ? RB * PB : KA) * sizeof(zc));
    // bit r: the r-th element's row (column) is inside the matrix
    unsigned amask = 0, bmask = 0;
#pragma unroll
    for (int r = 0; r < LA; ++r)
        if (row0 + ai + (a_mfast ? 0 : KA * r) < m && ((BM * BK) % NT == 0 || tid + NT * r < BM * BK)) amask |= 1u << r;
#pragma unroll
    for (int r = 0; r < LB; ++r)
        if (col0 + bj + (b_nfast ? 0 : KA * r) < n && ((BN * BK) % NT == 0 || tid + NT * r < BN * BK)) bmask |= 1u << r;

    auto load_stage = [&](int stage, int kt) {  // called for kt = kt0, kt0 + 1, ... in turn
        unsigned am = amask, bm = bmask;
        if ((kt + 1) * BK > k) {  // the last k-tile
            const int ka = k - kt * BK - ak, kb = k - kt * BK - bk;
#pragma unroll
            for (int r = 0; r < LA; ++r)
                if ((a_mfast ? RA * r : 0) >= ka) am &= ~(1u << r);
#pragma unroll
            for (int r = 0; r < LB; ++r)
                if ((b_nfast ? RB * r : 0) >= kb) bm &= ~(1u << r);
        }
#pragma unroll
        for (int r = 0; r < LA; ++r) {
            if ((BM * BK) % NT != 0 && r == LA - 1 && tid + NT * r >= BM * BK) break;
            const bool ok = (am >> r) & 1u;
            cp_async(sa0 + (uint32_t)(stage * BK * PA * (int)sizeof(TA)) + r * sar,
                     ok ? pa + r * astep : reinterpret_cast<const unsigned char *>(A.p), ok ? (int)sizeof(TA) : 0,
                     (int)sizeof(TA));
        }
#pragma unroll
        for (int r = 0; r < LB; ++r) {
            if ((BN * BK) % NT != 0 && r == LB - 1 && tid + NT * r >= BN * BK) break;
            const bool ok = (bm >> r) & 1u;
            const unsigned char *src = ok ? pb + r * bstep : reinterpret_cast<const unsigned char *>(B.p);
            const uint32_t dst = sb0 + (uint32_t)(stage * BK * PB * (int)sizeof(zc)) + r * sbr;
            if (B.real) {
                const double x = ok ? *reinterpret_cast<const double *>(src) : 0.0;
                asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(dst), "d"(x), "d"(0.0) : "memory");
            } else {
                cp_async(dst, src, ok ? 16 : 0, 16);
            }
        }
        pa += (long long)BK * A.cs * (long long)sizeof(TA);
        pb += (long long)BK * B.rs * bsz;
    };
    // Signs of the imaginary parts (conjugated views): with sa, sb = +-1, cr = sum ax bx - sa sb ay by, and ci is
    // accumulated as sb ci = sum ax by + sa sb ay bx, so that only A's fragments change sign.
    const int neg = ((!AREAL && A.conj) != (B.conj != 0)) ? (int)0x80000000u : 0;
    const auto flip = [](double x, int mask) { return __hiloint2double(__double2hiint(x) ^ mask, __double2loint(x)); };
    // 8 x 8 blocks of this warp inside the matrix: the others (padding) are not multiplied
    const int ni = min(4, (m - row0 - wr + 7) / 8), nj = min(2, (n - col0 - wc + 7) / 8);

    double cr[4][2][2], ci[4][2][2];  // 8 x 8 blocks (bi, bj): real and imaginary accumulators
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;

#pragma unroll
    for (int st = 0; st < ZG_STAGES - 1; ++st) {
        if (st < nkt) load_stage(st, kt0 + st);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int kt = 0; kt < nkt; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ZG_STAGES - 2) : "memory");
        // stage kt landed for every thread of the group; stage kt - 1 is no longer read
        if constexpr (KS == 1)
            __syncthreads();
        else
            asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(NT) : "memory");
        const int stage = kt % ZG_STAGES;
        const TA *At = As + (size_t)stage * BK * PA;
        const zc *Bt = Bs + (size_t)stage * BK * PB;
        // one k-step of four; FULL: every block of the warp is inside the matrix
        const auto step = [&](int kk, auto full) {
            constexpr bool FULL = decltype(full)::value;
            zc b[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) b[j] = Bt[(kk + fk) * PB + wc + 8 * j + fr];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (!FULL && i >= ni) break;
                const TA a = At[(kk + fk) * PA + wr + 8 * i + fr];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (!FULL && j == 1 && nj < 2) break;
                    if constexpr (AREAL) {
                        dmma884(cr[i][j], a, b[j].x);
                        dmma884(ci[i][j], a, b[j].y);
                    } else {
                        dmma884(cr[i][j], a.x, b[j].x);
                        dmma884(ci[i][j], a.x, b[j].y);
                        dmma884(cr[i][j], flip(a.y, neg ^ (int)0x80000000u), b[j].y);
                        dmma884(ci[i][j], flip(a.y, neg), b[j].x);
                    }
                }
            }
        };
        const int krem = k - (kt0 + kt) * BK;
        if (ni == 4 && nj == 2 && krem >= BK) {
#pragma unroll
            for (int kk = 0; kk < BK; kk += 4) step(kk, std::true_type{});
        } else if (nj > 0) {  // (warps, blocks and k-steps of padding alone are skipped)
#pragma unroll 1
            for (int kk = 0; kk < min(BK, krem); kk += 4) step(kk, std::false_type{});
        }
        const int kn = kt + ZG_STAGES - 1;  // refill the stage computed in the previous iteration
        if (kn < nkt) load_stage(kn % ZG_STAGES, kt0 + kn);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if constexpr (KS > 1) {
        // every group's accumulators to shared memory; group g then finishes row blocks g, g + KS, ..
        static_assert(KS * NT * 32 * sizeof(double) <= KS * zg_smem_bytes<AREAL, BM, BN>(), "reduction buffer");
        double *red = reinterpret_cast<double *>(zg_smem);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    red[((group * 4 + i) * 8 + j * 4 + h * 2) * NT + tid] = cr[i][j][h];
                    red[((group * 4 + i) * 8 + j * 4 + h * 2 + 1) * NT + tid] = ci[i][j][h];
                }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i % KS != group) continue;
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double *p = red + (i * 8 + j * 4 + h * 2) * NT + tid;
                    double x = p[0], y = p[NT];
#pragma unroll
                    for (int g = 1; g < KS; ++g) {
                        x += p[g * 32 * NT];
                        y += p[g * 32 * NT + NT];
                    }
                    cr[i][j][h] = x;
                    ci[i][j][h] = y;
                }
        }
    }
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (KS > 1 && i % KS != group) continue;
        const int gi = row0 + wr + 8 * i + fr;
        if (gi >= m) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int gj = col0 + wc + 8 * j + 2 * fk;
            if (gj >= n) continue;
            zc v[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) v[h] = alpha * zc{cr[i][j][h], B.conj ? -ci[i][j][h] : ci[i][j][h]};
            const long long off = oc + (long long)gi * C.rs + (long long)gj * C.cs;
            // consecutive columns side by side: one 32-byte store (a whole sector) instead of two halves
            if (!C.real && !use_beta && C.cs == 1 && gj + 1 < n && (reinterpret_cast<uintptr_t>(C.p + off) & 31) == 0) {
                asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(C.p + off), "d"(v[0].x), "d"(v[0].y),
                             "d"(v[1].x), "d"(v[1].y)
                             : "memory");
                continue;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (gj + h >= n) continue;
                const long long o = off + h * C.cs;
                if (C.real) {
                    double *cp = reinterpret_cast<double *>(C.p);
                    cp[o] = use_beta ? v[h].x + beta.x * cp[o] : v[h].x;
                } else {
                    C.p[o] = use_beta ? v[h] + beta * C.p[o] : v[h];
                }
            }
        }
    }
}

template <int BM, int BN, int KS = 1>
int launch_tile(int m, int n, int k, int nb0, int nb1, zc alpha, const View &A, const View &B, zc beta,
                const OutView &C, const long long *offs, cudaStream_t st) {
    const int ntn = (n + BN - 1) / BN, ntm = (m + BM - 1) / BM;
    const long long nbatch = (long long)nb0 * nb1;
    const long long gx = nbatch * ntn;
    if (gx > 2147483647LL || ntm > 65535) {
        set_error(PHF_ERR_ARG, "zgemm_strided: grid too large");
        return PHF_ERR_ARG;
    }
    dim3 grid((unsigned)gx, (unsigned)ntm, 1);
    if (A.real) {
        constexpr size_t smem = KS * zg_smem_bytes<true, BM, BN>();
        PHF_CUDA(cudaFuncSetAttribute(zgemm_kernel<true, BM, BN, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        ProfScope prof(st, -1);
        zgemm_kernel<true, BM, BN, KS><<<grid, KS * zg_threads<BM, BN>(), smem, st>>>(m, n, k, nb0, ntn, alpha, A, B,
                                                                                      beta, C, offs);
    } else {
        constexpr size_t smem = KS * zg_smem_bytes<false, BM, BN>();
        PHF_CUDA(cudaFuncSetAttribute(zgemm_kernel<false, BM, BN, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
        ProfScope prof(st, -1);
        zgemm_kernel<false, BM, BN, KS><<<grid, KS * zg_threads<BM, BN>(), smem, st>>>(m, n, k, nb0, ntn, alpha, A, B,
                                                                                       beta, C, offs);
    }
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

// Tile shape 0 = 64 x 64, 1 = 128 x 32, 2 = 32 x 128, 3 = 32 x 112, 4 = 64 x 112, 5 = 32 x 32,
// 6 = 32 x 64; 7 and 8 = 32 x 32 with k in four and two groups.
int launch_choice(int tile, int m, int n, int k, int nb0, int nb1, zc alpha, const View &A, const View &B, zc beta,
                  const OutView &C, const long long *offs, cudaStream_t st) {
    if (tile == 1) return launch_tile<128, 32>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    if (tile == 2) return launch_tile<32, 128>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    if (tile == 3) return launch_tile<32, 112>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    if (tile == 4) return launch_tile<64, 112>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    if (tile == 5) return launch_tile<32, 32>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    if (tile == 6) return launch_tile<32, 64>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    if (tile == 7) return launch_tile<32, 32, 4>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    if (tile == 8) return launch_tile<32, 32, 2>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    return launch_tile<64, 64>(m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
}

}  // namespace

// The tile comes from the launch tuner's table when the shape was tuned, else from rules set by
// measurements of the per-point products: 128 x 32 for at most 32 output columns and at least 96
// rows, 32 x 128 in the transposed case, 32 x 112 for 97..112 output columns (one column tile where
// 64 x 64 would pad 100 columns to 128), 64 x 64 otherwise.
int zgemm_strided(int m, int n, int k, int nb0, int nb1, zc alpha, const View &A, const View &B, zc beta,
                  const OutView &C, const long long *offs, cudaStream_t st) {
    if (m <= 0 || n <= 0 || nb0 <= 0 || nb1 <= 0) return PHF_OK;
    if (k <= 0) {
        set_error(PHF_ERR_ARG, "zgemm_strided: k <= 0");
        return PHF_ERR_ARG;
    }
    // Few 32 x 32 tiles over a long sum: the sum in groups of a block.  A tile's two warps use two of the four
    // schedulers and wait for every k-tile, so up to one block a multiprocessor takes four groups (16 tiles over k =
    // 400: 19.7 -> 10.3 us; 98 over 210: 20.1 -> 11.1; 35 over 40: 9.4 -> 6.8), up to two take two (195 over 96: 16.6
    // -> 14.5), and long sums take four groups up to three (200 over 1600: 175 -> 144 us, 325 real ones over 2080:
    // 173 -> 142; from four blocks a multiprocessor on, all schedulers are busy without).  The groups add in another
    // order than the other tiles, so such a shape has no other candidates.
    const long long tiles = (long long)nb0 * nb1 * ((m + 31) / 32) * ((n + 31) / 32);
    if (k > 2 * BK && tiles <= (k >= 16 * BK ? 444 : 296))
        return launch_choice(tiles <= 148 || k >= 16 * BK ? 7 : 8, m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
    const TuneKey key{0, (long long)m, (long long)n, (long long)k, (long long)nb0 * 65536 + nb1,
                      (long long)(A.real * 4 + B.real * 2 + C.real) * 2 + (offs != nullptr)};
    if (t_tune_record)
        t_tune_record->push_back({key, {0, 1, 2, 3, 4, 5, 6}, [=](int tile, cudaStream_t s) {
                                      return launch_choice(tile, m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, s);
                                  }});
    int tile = tuned_choice(key);
    if (tile < 0) {
        tile = (n <= 32 && m >= 96) ? 1 : ((m <= 32 && n >= 96) ? 2 : ((n > 96 && n <= 112) ? 3 : 0));
        // 32 x 32 tiles where the larger tile leaves multiprocessors idle or is mostly padding: the FP64 units of
        // one multiprocessor run at 64 multiply-adds a cycle whatever the tile, so the time goes with the
        // output elements per multiprocessor.  A quarter is allowed for the smaller tile's extra loads.
        constexpr int bm[4] = {64, 128, 32, 32}, bn[4] = {64, 32, 128, 112};
        const auto load = [&](int r, int c) {
            const long long ctas = (long long)nb0 * nb1 * ((m + r - 1) / r) * ((n + c - 1) / c);
            return (double)((ctas + 147) / 148) * r * c;
        };
        if (1.25 * load(32, 32) < load(bm[tile], bn[tile]) && (m + 31) / 32 <= 65535) tile = 5;
        // 32 x 64 instead of 64 x 64 for a short sum: a block is then mostly the first loads and the stores, and four
        // blocks on a multiprocessor overlap them where two leave it waiting (1600 x 1600 products over k = 30 and
        // 50 batches: 2.68 ms against 4.15; over k = 400 and more both measure the same, real ones 2 % worse).
        if (tile == 0 && k <= 64 && (m + 31) / 32 <= 65535) tile = 6;
    }
    return launch_choice(tile, m, n, k, nb0, nb1, alpha, A, B, beta, C, offs, st);
}

}  // namespace phf
