// FP64-accurate GEMM on the tcgen05 int8 tensor cores (Ozaki-style error-free slicing).
//
// D = A B with A (m x k) and B (k x n) given as FP64.  Each row of A is scaled by a power of
// two so that r = 127 a 2^-ea lies in (-127, 127) and cut into S balanced base-254 digits,
// r = sum_t d_t 254^{-t} (d_t in [-127, 127]); each column of B likewise with 2^eb.  Then
//     D_ij = 2^{ea_i + eb_j} / 127^2 sum_{g=2}^{S+1} 254^{2-g} sum_{t+u=g} (A_t B_u)_ij
// (slices numbered from 1) where every A_t B_u is an exact int8 x int8 -> int32 product on the
// tensor cores, the products of one group g share one int32 accumulator (exact while
// (g-1) k 127^2 < 2^31; longer k runs in several launches that add into D), and the S group sums
// are combined in FP64 in the epilogue.  Terms with t + u > S + 1 are dropped; the dropped terms
// and the digit remainder are of order 254^{-S} < 2^{-7S}: an entry's error is below about
// (S+1) k 2^{-7S} max|A_i.| max|B_.j| (random-sign errors grow like sqrt(k) in practice).
// (Ozaki, Ogita, Oishi, Rump, "Error-free transformations of matrix multiplication by using
// fast routines of matrix multiplication and its applications", Numer. Algorithms 59 (2012).)
//
// Slice layout in global memory (per operand, rows padded to 128, k to KB blocks of 32): slices
// 0..3 (group 0) interleaved per k-block so that one 128-byte row segment holds the same 32
// k-elements of four slices, byte (row KB + kb) 128 + t 32 + kk; then slices 4..S-1 (group 1) in
// 32-byte segments for S = 5, 64-byte segments for S = 6 or 128-byte segments for S = 7.  A TMA
// box of full segments (SWIZZLE_128B / 64B / 32B) carries several slices at once, and the MMA
// picks a slice by a +32-byte offset of its K-major descriptor.
//
// Kernel shape (one CTA per output tile, 6 warps); in launch order the CTAs sweep the column
// tiles in groups of eight row tiles, so that the A and B tiles in use fit in L2 together:
//   warp 0      TMA producer into a 224 KB shared-memory ring (full/empty mbarrier per slot): for
//               the single-pass formats (S <= 5, BF16X3, TF32) one packed stage per 32-element
//               k-block holding its A and B boxes (35 KB for S = 5, six stages); for S = 6, 7
//               fourteen 16 KB units, a k-block taking the A and B boxes of group 0 (a unit
//               each) and, in the second pass, group 1's boxes (one unit for S = 6, two for S = 7)
//   warp 1      TMEM allocation (512 columns) and the single-thread tcgen05.mma issuer.  S = 5
//               runs all five groups g = 2..6 in one pass over 128 x 96 tiles (five int32
//               accumulators, 480 columns); otherwise the tile is 128 x 128 and the groups run in
//               passes of four over the whole k range.  S <= 5 (the wide issue, the default):
//               per k-block one product per A slice t with the B slices 1 .. S + 1 - t laid side
//               by side, as MMAs of up to 256 columns (8 for S = 5); the narrow issue, kept for
//               comparison and used for S = 6, 7, makes every slice pair of the pass's groups one
//               128 x BN x 32 MMA (15 for S = 5).  At S = 5 the narrow issue ran at ~68 cycles per
//               128 x 96 x 32 MMA against 48 for the int8 rate, with the producer waiting on a
//               full ring (the operand reads of the narrow MMAs, not the loads, set the pace);
//               the wide issue reads 77 instead of 105 KB of shared memory per k-block
//   warps 2-5   epilogue after each pass: tcgen05.ld 32x32b.x32 of the pass's groups, int32 ->
//               FP64 with 254^{2-g} scaling.  For S = 6 the first pass's FP64 sums are parked in
//               TMEM (columns 0..255, where groups 2 and 3 were) and the second pass, accumulating
//               in columns 256..511, adds them before the single scaled store to D; for S = 7 the
//               second pass adds into D
// Every mbarrier wait gives up after ~2^31 clock cycles, sets *err and lets the CTA finish.
//
// The same kernel contracts two floating-point operand formats (slice-count codes OZ_FMT_BF16X3
// and OZ_FMT_TF32): a row (column) scaled by 2^-ea is held as BF16 high and low parts, or as one
// TF32 value, in one 128-byte segment per 32-element k-block; the MMAs are kind::f16 (BF16 x BF16)
// or kind::tf32 with FP32 accumulators in TMEM.  The k range runs in segments of args.kseg
// k-blocks that alternate between two FP32 accumulators (TMEM columns 0..127 and 128..255); the
// epilogue warps add each finished segment into FP64 sums parked in columns 256..511 (high and low
// words) while the MMAs fill the other accumulator, and store the FP64 total after the last one.
// The tensor core's FP32 accumulation rounds towards zero, so its error grows with the length of a
// same-sign sum; FP64 sums of short segments keep it at the level of one segment.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "phf_internal.h"

namespace phf {

namespace {

constexpr int OZ_BM = 128, OZ_BN = 128, OZ_BK = 32;  // tile rows, widest tile (row padding of B), k-block
constexpr int OZ_GP = 4;                             // slice groups per 128-byte row, accumulators per pass
constexpr int OZ_THREADS = 192;
constexpr int OZ_MAX_S = 7;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity) {
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

// Bounded wait on an mbarrier phase.  Returns false (and sets *err) after ~2^31 cycles.  The first
// probe takes no clock reading: the MMA issuer calls this once per k-block on its critical path.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *err, int code) {
    const uint32_t addr = smem_u32(bar);
    if (mbar_try(addr, parity)) return true;
    const long long t0 = clock64();
    while (true) {
        if (mbar_try(addr, parity)) return true;
        if (clock64() - t0 > (1LL << 31)) {
            atomicOr(err, code);
            return false;
        }
    }
}

__device__ __forceinline__ void tma_load_2d(const CUtensorMap *map, uint64_t *bar, void *dst, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}

// Shared-memory matrix descriptor: K-major, SWIZZLE_128B (8 rows x 128 B atoms, SBO = 1024 B).
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);          // start address
    d |= (uint64_t)1 << 16;                           // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                 // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                           // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                           // layout: SWIZZLE_128B
    return d;
}

// Shared-memory matrix descriptor: K-major, SWIZZLE_32B (8 rows x 32 B atoms, SBO = 256 B).
__device__ __forceinline__ uint64_t sdesc_sw32(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(256 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)6 << 61;                           // layout: SWIZZLE_32B
    return d;
}

// Shared-memory matrix descriptor: K-major, SWIZZLE_64B (8 rows x 64 B atoms, SBO = 512 B).
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;                           // layout: SWIZZLE_64B
    return d;
}

// Instruction descriptor: kind::i8, D = s32, A = B = s8, both K-major, M = 128, N = BN.
template <int BN>
__host__ __device__ constexpr uint32_t idesc_i8() {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);
}

// the same for an N known only as a value (a multiple of 16, at most 256)
__host__ __device__ constexpr uint32_t idesc_i8_n(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);
}

__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

// Instruction descriptors with FP32 accumulation, K-major A and B, M = 128, N = BN: kind::f16 with
// A = B = BF16, and kind::tf32.
template <int BN>
__host__ __device__ constexpr uint32_t idesc_bf16() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);
}
template <int BN>
__host__ __device__ constexpr uint32_t idesc_tf32() {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
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

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}

struct OzArgs {
    int m, n, kb0, kblocks, S;
    const int *ea, *eb;  // row / column exponents
    double *D;
    long long ldd;
    int accumulate;      // D += result instead of D = result
    int trans;           // write D^T: element (i, j) at D[j * ldd + i]
    long long dz;        // split-k: CTA z covers k-blocks [z kblocks, (z+1) kblocks) and writes D + z dz
    int kb_total;        // k-blocks of this launch over all splits
    int kseg;            // floating-point formats: k-blocks per FP32 accumulation segment (>= 1)
    int gamma_n;         // > 0: exchange-to-Gamma output (see store_row_chunk), n spatial orbitals
    int g_row0;          // exchange-to-Gamma output: global row of output row 0 (a panel of the exchange rows)
    int gamma_mode;      // exchange-to-Gamma rows: 0 full (i n + k), 1 symmetric pairs, 2 antisymmetric pairs
    const int *g_pairs;  // modes 1, 2: pair (i, k) of global row g packed as i << 16 | k
    int a_row0;          // A tiles are read from row a_row0 + m0 of the A slice buffer (a row range of it)
    int b_row0;          // B tiles are read from row b_row0 + n0 of the B slice buffer
    int group_m;         // row tiles per column sweep of the raster
    int batch = 0;       // 1: blockIdx.z is a batch index (one product per grid point) instead of a k split:
                         // its A rows start at z a_bs, its B rows at z b_bs (and their exponents likewise),
                         // its output at D + z dz
    long long a_bs = 0, b_bs = 0;
    int ct = 0;          // complex-transposed output: columns (2c, 2c + 1) of row r are the real and
                         // imaginary parts of complex element (c, r), stored at D[c ldd + 2 r] (doubles)
    int *err;
};

// Stores one epilogue thread's 32 consecutive columns col0 .. col0 + 31 of output row `row` (values
// acc * rowscale * cs): element (row, col) at D[row ldd + col], or D[col ldd + row] when args.trans,
// added to what is there when `add`.  Exchange-to-Gamma mode (args.gamma_n = n > 0): the product is
// K^T of the exchange GEMM, col = (4 w + 2 sigma + tau) 2 + part, and -K goes straight into the
// complex M x M matrix Gamma_w (D = Gamma as doubles); the Coulomb term is added to the diagonal spin
// blocks afterwards.  Rows by args.gamma_mode (g = args.g_row0 + row):
//   0: g = i n + k, -K_{sigma tau}[i][k] at [2i + sigma][2k + tau];
//   1: pair (i, k), i <= k, of g_pairs[g]: the symmetric-density part KS of K[i][k] and K[k][i]
//      (equal), -KS stored at [2i + sigma][2k + tau] and at [2k + sigma][2i + tau];
//   2: pair (i, k), i < k: the antisymmetric-density part KA (K[i][k] = KS + KA, K[k][i] = KS - KA),
//      -KA added at [2i + sigma][2k + tau] and +KA at [2k + sigma][2i + tau] (after mode 1's stores).
__device__ __forceinline__ void store_row_chunk(const OzArgs &args, double *Dz, int row, int col0,
                                                const double (&acc)[32], double rowscale, const double *cs,
                                                bool add) {
    if (args.gamma_n > 0) {
        const int gn = args.gamma_n, M = 2 * gn, grow = args.g_row0 + row;
        int i, k;
        if (args.gamma_mode == 0) {
            i = grow / gn;
            k = grow - i * gn;
        } else {
            const int pr = __ldg(args.g_pairs + grow);
            i = pr >> 16;
            k = pr & 0xffff;
        }
        const bool mirror = args.gamma_mode != 0 && i != k;
        const bool acc_both = add || args.gamma_mode == 2;
        double2 *const G2 = reinterpret_cast<double2 *>(Dz);
        // element (column pair q) of the chunk: Gamma_w[2i + sg][2k + tu] and its mirror [2k + sg][2i + tu]
        auto at = [&](int col, bool mir) {
            const int w = col >> 3, sg = (col >> 2) & 1, tu = (col >> 1) & 1;
            return mir ? G2 + ((long long)w * M + 2 * k + sg) * M + 2 * i + tu
                       : G2 + ((long long)w * M + 2 * i + sg) * M + 2 * k + tu;
        };
        // Accumulating stores read Gamma first: each batch of eight column pairs issues all its loads
        // before its stores (the addresses of distinct columns, and of an element and its mirror, never
        // coincide), so that the loads' latencies overlap instead of following one another.
#pragma unroll
        for (int jb = 0; jb < 32; jb += 16) {
            double2 og[8], oh[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int col = col0 + jb + 2 * q;
                og[q] = oh[q] = make_double2(0.0, 0.0);
                if (acc_both && col < args.n) {
                    og[q] = *at(col, false);
                    if (mirror) oh[q] = *at(col, true);
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int j = jb + 2 * q, col = col0 + j;
                if (col < args.n) {
                    const double2 u = make_double2(acc[j] * rowscale * cs[j], acc[j + 1] * rowscale * cs[j + 1]);
                    *at(col, false) = make_double2(og[q].x - u.x, og[q].y - u.y);
                    if (mirror)
                        *at(col, true) = args.gamma_mode == 2 ? make_double2(oh[q].x + u.x, oh[q].y + u.y)
                                                              : make_double2(oh[q].x - u.x, oh[q].y - u.y);
                }
            }
        }
        return;
    }
    if (args.ct) {  // (col0 and n are even: the chunk holds whole real/imaginary column pairs)
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
            const int col = col0 + j;
            if (col < args.n) {
                double2 *p = reinterpret_cast<double2 *>(Dz + (long long)(col >> 1) * args.ldd + 2LL * row);
                const double2 u = make_double2(acc[j] * rowscale * cs[j], acc[j + 1] * rowscale * cs[j + 1]);
                if (add) {
                    const double2 o = *p;
                    *p = make_double2(o.x + u.x, o.y + u.y);
                } else {
                    *p = u;
                }
            }
        }
        return;
    }
    double *drow = Dz + (args.trans ? (long long)row : (long long)row * args.ldd);
    const long long cstride = args.trans ? args.ldd : 1;
    double old[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const int col = col0 + j;
        old[j] = (add && col < args.n) ? drow[(long long)col * cstride] : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const int col = col0 + j;
        if (col < args.n) {
            const double val = acc[j] * rowscale * cs[j];
            drow[(long long)col * cstride] = add ? old[j] + val : val;
        }
    }
}

// floating-point operand formats (slice-count codes beyond the int8 range 1..7)
__host__ __device__ constexpr bool oz_float(int S) { return S == OZ_FMT_BF16X3 || S == OZ_FMT_TF32; }

// Slices per k-block row of group 1: one (32-byte rows) for S = 5, two (64-byte rows) for S = 6,
// four (128-byte rows) for S = 7; none for S <= 4 and the floating-point formats (one 128-byte
// segment per k-block).
__host__ __device__ constexpr int oz_g1_width(int S) {
    return (S <= OZ_GP || oz_float(S)) ? 0 : (S == 5 ? 1 : (S == 6 ? 2 : 4));
}

// Byte offset of element (row, k) of a floating-point-format operand (KB k-blocks of 32): the
// 128-byte segment of (row, k-block) holds, for BF16X3, the high parts of its 32 elements in bytes
// [0, 64) and the low parts in [64, 128) (part = 0, 1); for TF32 the 32 four-byte values.  Each
// 32-byte quarter is the K-chunk of one MMA (16 BF16 or 8 TF32 values).
__host__ __device__ __forceinline__ long long oz_float_offset(int part, long long row, long long k, long long KB,
                                                              int S) {
    const long long base = (row * KB + (k >> 5)) << 7, kk = k & 31;
    return S == OZ_FMT_BF16X3 ? base + 64 * part + 2 * kk : base + 4 * kk;
}

// Byte offset of slice t of element (row, k) in an operand's slice buffer with rows_pad rows and KB
// k-blocks of 32: group 0 in 128-byte k-block rows, then group 1 in (32 x width)-byte rows.
__host__ __device__ __forceinline__ long long oz_slice_offset(int t, long long row, long long k, long long rows_pad,
                                                              long long KB, int S) {
    const long long kb = k >> 5, kk = k & 31;
    if (t < OZ_GP) return ((row * KB + kb) << 7) + ((long long)t << 5) + kk;
    return rows_pad * KB * 128 + (row * KB + kb) * (32LL * oz_g1_width(S)) + ((long long)(t - OZ_GP) << 5) + kk;
}

// Shared-memory ring of OZ_UNITS units of 16 KB for the two-pass slice counts S = 6, 7: a k-block
// takes two units (A and B tiles of slice group 0), plus, in the second pass, one unit holding group
// 1's A and B boxes at 64-byte rows (S = 6) or two units (S = 7: group 1 at 128-byte rows).  The
// single-pass formats use the same bytes as a ring of packed k-block stages (oz_stage_bytes).
constexpr int OZ_UNITS = 14;
constexpr int OZ_GROUP_M = 8;  // row tiles per column sweep of the raster (default; the launch tuner may pick another)
constexpr int OZ_KSEG = 16;    // floating-point formats: k-blocks (512 k-elements) per FP32 accumulation segment

// Tile width and passes per slice count.  S = 5 runs its five groups g = 2..6 in one pass over
// 96-column tiles (5 x 96 of the 512 TMEM columns); the others use 128-column tiles and passes of
// up to four groups (S = 6, 7: groups 2..5, then the rest).
__host__ __device__ constexpr int oz_bn(int S) { return S == 5 ? 96 : 128; }
__host__ __device__ constexpr int oz_npass(int S) { return (S == 5 || oz_float(S)) ? 1 : (S + OZ_GP - 1) / OZ_GP; }
__host__ __device__ constexpr int oz_g0(int P) { return 2 + OZ_GP * P; }
__host__ __device__ constexpr int oz_g1(int S, int P) {
    return S == 5 ? 6 : ((1 + OZ_GP * (P + 1) < S + 1) ? 1 + OZ_GP * (P + 1) : S + 1);
}
// 16 KB ring units a k-block of pass P takes: A and B of group 0, plus group 1 when the pass uses
// slices beyond the fourth (one unit holding both 32- or 64-byte-row boxes, or one each for S = 7)
__host__ __device__ constexpr int oz_units(int S, int P) {
    return oz_float(S) ? 2 : (oz_g1(S, P) - 1 > OZ_GP ? (oz_g1_width(S) <= 2 ? 3 : 4) : 2);
}
// bytes the TMA delivers into unit j of a k-block
__host__ __device__ constexpr uint32_t oz_unit_bytes(int S, int j) {
    return j == 0 ? OZ_BM * 128u
                  : j == 1 ? (uint32_t)oz_bn(S) * 128u
                           : (oz_g1_width(S) <= 2 ? (OZ_BM + (uint32_t)oz_bn(S)) * 32u * (uint32_t)oz_g1_width(S)
                                                  : (j == 2 ? OZ_BM * 128u : (uint32_t)oz_bn(S) * 128u));
}

// 254^{-t}: group g = t + 2 of the balanced base-254 digit products
__constant__ double kPow254[7] = {1.0, 0.003937007874015748, 1.5500031000062e-05, 6.102374409473229e-08,
                                  2.40250961002883e-10, 9.458699252082008e-13, 3.723897343339373e-15};
constexpr uint32_t OZ_UNIT = 16384;

// Single-pass formats (S <= 5 and the floating-point formats) pack all boxes of one k-block into one
// stage of the ring instead of whole 16 KB units: A (BM x 128 B) at 0, B (BN x 128 B) at BM 128 and,
// for S = 5, the fifth slice's A (BM x 32 B) and B (BN x 32 B) behind them.  For S = 5 that is 35 KB
// per k-block (6 stages in flight instead of 4.7 k-blocks of three units); the ring's depth, not its
// bandwidth, is what keeps the MMAs fed.
__host__ __device__ constexpr bool oz_staged(int S) { return oz_npass(S) == 1; }
__host__ __device__ constexpr uint32_t oz_stage_bytes(int S) {
    return (OZ_BM + (uint32_t)oz_bn(S)) * 128u + (oz_g1_width(S) == 1 ? (OZ_BM + (uint32_t)oz_bn(S)) * 32u : 0u);
}
// stage footprint in the ring, a multiple of 1024 bytes (the SWIZZLE_128B atom)
__host__ __device__ constexpr uint32_t oz_stage_pitch(int S) { return (oz_stage_bytes(S) + 1023u) / 1024u * 1024u; }
__host__ __device__ constexpr int oz_stages(int S) { return (int)((OZ_UNITS * OZ_UNIT) / oz_stage_pitch(S)); }

// Wide issue (single-pass int8, S <= 5).  The products A_t B_u of one A slice t go to the groups
// g = t + u = t + 1 .. S + 1, whose accumulators sit side by side in TMEM (group g at columns
// (g - 2) BN); so when the stage holds the B slices one after another -- slice u at rows
// (u - 1) BN .. u BN - 1 of one 32-byte-row (SWIZZLE_32B) operand -- the products of A_t with
// B_1 .. B_{S+1-t} are ONE matrix product with an (S + 1 - t) BN-row B operand, written to TMEM
// columns (t - 1) BN onwards.  Per 32-element k-block that is S such products (split into MMAs of
// at most 256 columns: 8 MMAs for S = 5 instead of 15), and each A slice is read from shared
// memory once per MMA instead of once per slice pair: 77 KB of operand reads per k-block instead
// of 105 KB for S = 5.  The int32 sums are the same, so results are bitwise those of the narrow
// issue.  Stage: A's group-0 box (BM x 128 B, SWIZZLE_128B) at 0, the S B slices (S x BN x 32 B)
// at BM 128, the fifth A slice (BM x 32 B) behind them.
__host__ __device__ constexpr bool oz_wide_ok(int S) { return S >= 1 && S <= 5; }
__host__ __device__ constexpr uint32_t oz_wide_b_off() { return OZ_BM * 128u; }
__host__ __device__ constexpr uint32_t oz_wide_a1_off(int S) { return OZ_BM * 128u + (uint32_t)S * oz_bn(S) * 32u; }
__host__ __device__ constexpr uint32_t oz_wide_stage_bytes(int S) {
    return oz_wide_a1_off(S) + (oz_g1_width(S) == 1 ? OZ_BM * 32u : 0u);
}
__host__ __device__ constexpr uint32_t oz_wide_stage_pitch(int S) { return (oz_wide_stage_bytes(S) + 1023u) / 1024u * 1024u; }
__host__ __device__ constexpr int oz_wide_stages(int S) { return (int)((OZ_UNITS * OZ_UNIT) / oz_wide_stage_pitch(S)); }

// One k-block of pass P: every slice pair (t, g - t) of the pass's groups g is one MMA.  Unrolled,
// so that each descriptor is a tile's base descriptor plus a constant (+2 per 32 bytes): the
// single issuing thread runs barely ahead of the tensor core, and any latency between two MMAs
// is tensor-core idle time.  dA0/dB0: group-0 tiles, dA1/dB1: group-1 tiles.
template <int S, int P>
__device__ __forceinline__ void issue_kblock(uint32_t acc0, uint64_t dA0, uint64_t dB0, uint64_t dA1, uint64_t dB1,
                                             uint32_t acc_in) {
    constexpr int g0 = oz_g0(P), g1 = oz_g1(S, P), BN = oz_bn(S);
    constexpr uint32_t idesc = idesc_i8<BN>();
#pragma unroll
    for (int g = g0; g <= g1; ++g) {
#pragma unroll
        for (int t = 1; t < g; ++t) {
            const int u = g - t;
            const uint64_t a = (t > OZ_GP ? dA1 : dA0) + (uint64_t)(2 * ((t - 1) % OZ_GP));
            const uint64_t b = (u > OZ_GP ? dB1 : dB0) + (uint64_t)(2 * ((u - 1) % OZ_GP));
            mma_i8(acc0 + (uint32_t)(g - g0) * BN, a, b, idesc, t > 1 ? 1u : acc_in);
        }
    }
}

// One k-block of the wide issue: for each A slice t, its product with B slices 1 .. S + 1 - t
// as MMAs of at most 256 columns whose TMEM column offsets are multiples of 32 (480 = 256 + 224,
// 384 = 192 + 192, 288 = 160 + 128 for S = 5).  A_1's MMAs cover every group's columns, so with
// acc_in = 0 they start the accumulators of the tile's first k-block.
template <int S>
__device__ __forceinline__ void issue_kblock_wide(uint32_t acc0, uint64_t dA0, uint64_t dA1, uint32_t bbase,
                                                  uint32_t acc_in) {
    constexpr int BN = oz_bn(S);
#pragma unroll
    for (int t = 1; t <= S; ++t) {
        const uint64_t a = t > OZ_GP ? dA1 : dA0 + (uint64_t)(2 * (t - 1));
        const int nt = (S + 1 - t) * BN;
        const int parts = (nt + 255) / 256;
        const int w = ((nt + parts - 1) / parts + 31) / 32 * 32;
#pragma unroll
        for (int q = 0; q < parts; ++q) {
            const int r0 = q * w, np = min(w, nt - r0);
            mma_i8(acc0 + (uint32_t)((t - 1) * BN + r0), a, sdesc_sw32(bbase + (uint32_t)r0 * 32u), idesc_i8_n(np),
                   t > 1 ? 1u : acc_in);
        }
    }
}

// One k-block of a floating-point format (one 128-byte segment per operand row, +2 in a descriptor
// = +32 bytes = the next quarter), all into the accumulator acc0.  TF32: four K = 8 MMAs.  BF16X3
// (quarters 0, 1 = high parts of k 0..15 and 16..31, quarters 2, 3 = low parts): hi*hi, hi*lo and
// lo*hi of each half, six K = 16 MMAs.
template <int S>
__device__ __forceinline__ void issue_kblock_float(uint32_t acc0, uint64_t dA, uint64_t dB, uint32_t acc_in) {
    constexpr int BN = oz_bn(S);
    if constexpr (S == OZ_FMT_TF32) {
        constexpr uint32_t idesc = idesc_tf32<BN>();
#pragma unroll
        for (int q = 0; q < 4; ++q) mma_tf32(acc0, dA + 2 * q, dB + 2 * q, idesc, q > 0 ? 1u : acc_in);
    } else {
        constexpr uint32_t idesc = idesc_bf16<BN>();
#pragma unroll
        for (int h = 0; h < 2; ++h) mma_bf16(acc0, dA + 2 * h, dB + 2 * h, idesc, h > 0 ? 1u : acc_in);
#pragma unroll
        for (int h = 0; h < 2; ++h) mma_bf16(acc0, dA + 2 * h, dB + 4 + 2 * h, idesc, 1u);
#pragma unroll
        for (int h = 0; h < 2; ++h) mma_bf16(acc0, dA + 4 + 2 * h, dB + 2 * h, idesc, 1u);
    }
}

// The MMA issuer's k-block loop of pass P (u, ph: next ring unit -- or stage, for the single-pass
// formats -- and its full-barrier parity).
template <int S, int P, bool WIDE = false>
__device__ __forceinline__ bool mma_pass(uint32_t acc0, int KB, int &u, uint32_t &ph, uint32_t smem_base,
                                         uint64_t *full_bar, uint64_t *empty_bar, int *err) {
    if constexpr (WIDE) {
        constexpr int NS = oz_wide_stages(S);
        constexpr uint32_t PITCH = oz_wide_stage_pitch(S);
        for (int kb = 0; kb < KB; ++kb) {
            if (!mbar_wait(&full_bar[u], ph, err, 2)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t base = smem_base + (uint32_t)u * PITCH;
            const uint64_t dA1 = oz_g1_width(S) == 1 ? sdesc_sw32(base + oz_wide_a1_off(S)) : 0;
            issue_kblock_wide<S>(acc0, sdesc_sw128(base), dA1, base + oz_wide_b_off(), kb > 0 ? 1u : 0u);
            mma_commit(&empty_bar[u]);  // the stage is reusable once these MMAs have read it
            if (++u == NS) {
                u = 0;
                ph ^= 1u;
            }
        }
        return true;
    } else if constexpr (oz_staged(S)) {
        constexpr int NS = oz_stages(S), BN = oz_bn(S);
        constexpr uint32_t PITCH = oz_stage_pitch(S);
        for (int kb = 0; kb < KB; ++kb) {
            if (!mbar_wait(&full_bar[u], ph, err, 2)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t base = smem_base + (uint32_t)u * PITCH;
            const uint64_t dA0 = sdesc_sw128(base);
            const uint64_t dB0 = sdesc_sw128(base + OZ_BM * 128);
            if constexpr (oz_float(S)) {
                issue_kblock_float<S>(acc0, dA0, dB0, kb > 0 ? 1u : 0u);
            } else {
                uint64_t dA1 = 0, dB1 = 0;
                if constexpr (oz_g1_width(S) == 1) {
                    dA1 = sdesc_sw32(base + (OZ_BM + BN) * 128);
                    dB1 = sdesc_sw32(base + (OZ_BM + BN) * 128 + OZ_BM * 32);
                }
                issue_kblock<S, P>(acc0, dA0, dB0, dA1, dB1, kb > 0 ? 1u : 0u);
            }
            mma_commit(&empty_bar[u]);  // the stage is reusable once these MMAs have read it
            if (++u == NS) {
                u = 0;
                ph ^= 1u;
            }
        }
        return true;
    } else {
        constexpr int NU = oz_units(S, P);
        for (int kb = 0; kb < KB; ++kb) {
            int us[NU];
#pragma unroll
            for (int j = 0; j < NU; ++j) {
                us[j] = u;
                if (!mbar_wait(&full_bar[u], ph, err, 2)) return false;
                if (++u == OZ_UNITS) {
                    u = 0;
                    ph ^= 1u;
                }
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t dA0 = sdesc_sw128(smem_base + (uint32_t)us[0] * OZ_UNIT);
            const uint64_t dB0 = sdesc_sw128(smem_base + (uint32_t)us[1] * OZ_UNIT);
            uint64_t dA1 = 0, dB1 = 0;
            if constexpr (NU == 3) {  // S = 6: group 1 at 64-byte rows in one unit
                dA1 = sdesc_sw64(smem_base + (uint32_t)us[2] * OZ_UNIT);
                dB1 = sdesc_sw64(smem_base + (uint32_t)us[2] * OZ_UNIT + OZ_BM * 64);
            } else if constexpr (NU == 4) {
                dA1 = sdesc_sw128(smem_base + (uint32_t)us[2] * OZ_UNIT);
                dB1 = sdesc_sw128(smem_base + (uint32_t)us[3] * OZ_UNIT);
            }
            issue_kblock<S, P>(acc0, dA0, dB0, dA1, dB1, kb > 0 ? 1u : 0u);
#pragma unroll
            for (int j = 0; j < NU; ++j) mma_commit(&empty_bar[us[j]]);  // units reusable once these MMAs read them
        }
        return true;
    }
}

// tmBw: the B operand's group-0 slices as 32-byte boxes (the wide issue's per-slice B loads)
template <int S, bool WIDE = false>
__global__ void __launch_bounds__(OZ_THREADS, 1)
    ozaki_i8_gemm_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmB0,
                         const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1,
                         const __grid_constant__ CUtensorMap tmBw, OzArgs args) {
    static_assert(!WIDE || oz_wide_ok(S), "the wide issue takes single-pass int8 slices");
    extern __shared__ __align__(1024) unsigned char oz_smem_raw[];
    unsigned char *smem = oz_smem_raw;
    if ((smem_u32(oz_smem_raw) & 1023u) != 0u) {  // the swizzled tiles need a 1024-byte aligned base
        if (threadIdx.x == 0) atomicOr(args.err, 16);
        return;
    }
    constexpr int W1 = oz_g1_width(S), BN = oz_bn(S);
    constexpr double kUnit = oz_float(S) ? 1.0 : 1.0 / 127.0;  // value of one slice unit at exponent 0
    const int npass = oz_npass(S);  // pass p: groups oz_g0(p) .. oz_g1(S, p)
    // With two passes and at most two groups in the second, the first pass's FP64 partial sums stay
    // in TMEM columns [0, 256) (high words, then low words, per 32-column chunk) and the second
    // pass accumulates in columns [256, 512); otherwise the second pass adds into D.
    const bool keep = (npass == 2) && (S <= 6);
    uint64_t *full_bar = reinterpret_cast<uint64_t *>(smem + (size_t)OZ_UNITS * OZ_UNIT);
    uint64_t *empty_bar = full_bar + OZ_UNITS;
    uint64_t *pass_bar = empty_bar + OZ_UNITS;  // MMAs of a pass complete
    uint64_t *free_bar = pass_bar + 1;          // epilogue has read the pass's accumulators
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(free_bar + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    double *colscale = reinterpret_cast<double *>(free_bar + 2);  // 2^{eb} / 127 of the tile's columns
    // floating-point formats: accumulator b holds a finished segment (acc_full[b], one arrival by
    // the MMA commit) / has been drained by the epilogue (acc_empty[b], 128 arrivals)
    uint64_t *acc_full = reinterpret_cast<uint64_t *>(colscale + OZ_BN);
    uint64_t *acc_empty = acc_full + 2;
    const int kseg = max(1, args.kseg);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // grouped raster: CTAs in launch order sweep the column tiles in groups of args.group_m row tiles,
    // so that the A and B tiles the resident CTAs share fit in L2 together
    int m0, n0;
    {
        const int mt = gridDim.x, nt = gridDim.y;
        const int L = blockIdx.y * mt + blockIdx.x;
        const int G = args.group_m > 0 ? args.group_m : OZ_GROUP_M;
        const int width = G * nt;
        const int first = (L / width) * G;
        const int gm = min(mt - first, G);
        m0 = (first + (L % width) % gm) * OZ_BM;
        n0 = ((L % width) / gm) * BN;
    }
    const long long za = args.batch ? (long long)blockIdx.z * args.a_bs : 0;  // batch offsets of A and B rows
    const long long zb = args.batch ? (long long)blockIdx.z * args.b_bs : 0;
    const int am0 = (int)(m0 + args.a_row0 + za);  // first row of the A tile in the A slice buffer
    const int bn0 = (int)(n0 + args.b_row0 + zb);  // first row of the B tile in the B slice buffer
    const int kz0 = args.batch ? 0 : blockIdx.z * args.kblocks;  // first k-block of this split
    const int KB = max(0, min(args.kblocks, args.kb_total - kz0));
    double *const Dz = args.D + (long long)blockIdx.z * args.dz;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int s = 0; s < OZ_UNITS; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(pass_bar, 1);
        mbar_init(free_bar, 128);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 128);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA0)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(WIDE ? &tmBw : &tmB0)) : "memory");
        if (W1 > 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA1)) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB1)) : "memory");
        }
    }
    if (warp >= 2) {
        const int c = threadIdx.x - 64;
        colscale[c] = (c < BN && n0 + c < args.n) ? ldexp(kUnit, args.eb[zb + n0 + c]) : 0.0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0 && WIDE) {  // TMA producer, one wide stage per k-block
            constexpr int NS = oz_wide_stages(S);
            constexpr uint32_t PITCH = oz_wide_stage_pitch(S), BYTES = oz_wide_stage_bytes(S);
            constexpr int U0 = S < OZ_GP ? S : OZ_GP;  // B slices in the group-0 buffer
            int sg = 0;
            uint32_t eph = 0;
            bool wrapped = false;
            for (int kb = 0; kb < KB && !*abort_flag; ++kb) {
                const int kbg = args.kb0 + kz0 + kb;
                if (wrapped && !mbar_wait(&empty_bar[sg], eph, args.err, 1)) {
                    *abort_flag = 1;
                    break;
                }
                unsigned char *dst = smem + (size_t)sg * PITCH;
                unsigned char *bdst = dst + oz_wide_b_off();
                mbar_arrive_expect_tx(&full_bar[sg], BYTES);
                tma_load_2d(&tmA0, &full_bar[sg], dst, kbg * 128, am0);
#pragma unroll
                for (int u = 0; u < U0; ++u)  // slice u + 1 of B: 32 bytes of each 128-byte k-block row
                    tma_load_2d(&tmBw, &full_bar[sg], bdst + u * BN * 32, kbg * 128 + u * 32, bn0);
                if constexpr (W1 == 1) {
                    tma_load_2d(&tmB1, &full_bar[sg], bdst + OZ_GP * BN * 32, kbg * 32, bn0);
                    tma_load_2d(&tmA1, &full_bar[sg], dst + oz_wide_a1_off(S), kbg * 32, am0);
                }
                if (++sg == NS) {
                    sg = 0;
                    if (wrapped) eph ^= 1u;
                    wrapped = true;
                }
            }
        } else if (lane == 0 && oz_staged(S)) {  // TMA producer, one stage per k-block
            constexpr int NS = oz_stages(S);
            constexpr uint32_t PITCH = oz_stage_pitch(S), BYTES = oz_stage_bytes(S);
            int sg = 0;           // next stage
            uint32_t eph = 0;     // parity of the empty-barrier phase that frees it (after the first lap)
            bool wrapped = false;
            for (int kb = 0; kb < KB && !*abort_flag; ++kb) {
                const int kbg = args.kb0 + kz0 + kb;
                if (wrapped && !mbar_wait(&empty_bar[sg], eph, args.err, 1)) {
                    *abort_flag = 1;
                    break;
                }
                unsigned char *dst = smem + (size_t)sg * PITCH;
                mbar_arrive_expect_tx(&full_bar[sg], BYTES);
                tma_load_2d(&tmA0, &full_bar[sg], dst, kbg * 128, am0);
                tma_load_2d(&tmB0, &full_bar[sg], dst + OZ_BM * 128, kbg * 128, bn0);
                if constexpr (W1 == 1) {
                    tma_load_2d(&tmA1, &full_bar[sg], dst + (OZ_BM + BN) * 128, kbg * 32, am0);
                    tma_load_2d(&tmB1, &full_bar[sg], dst + (OZ_BM + BN) * 128 + OZ_BM * 32, kbg * 32, bn0);
                }
                if (++sg == NS) {
                    sg = 0;
                    if (wrapped) eph ^= 1u;
                    wrapped = true;
                }
            }
        } else if (lane == 0) {  // TMA producer: unit sequence = (pass, k-block, tile)
            int u = 0;            // next unit
            uint32_t eph = 0;     // parity of the empty-barrier phase that frees it (after the first lap)
            bool wrapped = false;
            for (int p = 0; p < npass && !*abort_flag; ++p) {
                const int nu = p == 0 ? oz_units(S, 0) : oz_units(S, 1);
                for (int kb = 0; kb < KB && !*abort_flag; ++kb) {
                    const int kbg = args.kb0 + kz0 + kb;
                    for (int j = 0; j < nu; ++j) {
                        if (wrapped && !mbar_wait(&empty_bar[u], eph, args.err, 1)) {
                            *abort_flag = 1;
                            break;
                        }
                        unsigned char *dst = smem + (size_t)u * OZ_UNIT;
                        const uint32_t ub = j == 0 ? oz_unit_bytes(S, 0)
                                                   : j == 1 ? oz_unit_bytes(S, 1)
                                                            : j == 2 ? oz_unit_bytes(S, 2) : oz_unit_bytes(S, 3);
                        mbar_arrive_expect_tx(&full_bar[u], ub);
                        if (j == 0) {
                            tma_load_2d(&tmA0, &full_bar[u], dst, kbg * 128, am0);
                        } else if (j == 1) {
                            tma_load_2d(&tmB0, &full_bar[u], dst, kbg * 128, bn0);
                        } else if (W1 <= 2) {  // j == 2: A and B of group 1 at 32- or 64-byte rows
                            tma_load_2d(&tmA1, &full_bar[u], dst, kbg * 32 * W1, am0);
                            tma_load_2d(&tmB1, &full_bar[u], dst + OZ_BM * 32 * W1, kbg * 32 * W1, bn0);
                        } else if (j == 2) {
                            tma_load_2d(&tmA1, &full_bar[u], dst, kbg * 128, am0);
                        } else {
                            tma_load_2d(&tmB1, &full_bar[u], dst, kbg * 128, bn0);
                        }
                        if (++u == OZ_UNITS) {
                            u = 0;
                            if (wrapped) eph ^= 1u;
                            wrapped = true;
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // MMA issuer
            int u = 0;         // next unit
            uint32_t ph = 0;   // parity of its full-barrier phase
            bool ok = true;
            const uint32_t smem_base = smem_u32(smem);
            if constexpr (oz_float(S)) {  // segments s into accumulator s & 1
                const int nseg = max(1, (KB + kseg - 1) / kseg);
                for (int sg = 0; sg < nseg && ok; ++sg) {
                    const int b = sg & 1;
                    if (sg >= 2) {  // wait until the epilogue has drained segment sg - 2
                        if (!mbar_wait(&acc_empty[b], ((sg >> 1) - 1) & 1, args.err, 8)) {
                            *abort_flag = 1;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                    const int nkb = max(0, min(kseg, KB - sg * kseg));
                    ok = mma_pass<S, 0>(tmem_base + (uint32_t)b * BN, nkb, u, ph, smem_base, full_bar, empty_bar,
                                        args.err);
                    if (!ok) *abort_flag = 1;
                    mma_commit(&acc_full[b]);
                }
            }
            for (int p = 0; p < npass && ok && !oz_float(S); ++p) {
                if (p > 0) {  // accumulators drained by the epilogue
                    if (!mbar_wait(free_bar, (p - 1) & 1, args.err, 8)) {
                        *abort_flag = 1;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                const uint32_t acc0 = tmem_base + ((p > 0 && keep) ? 256u : 0u);
                if (p == 0)
                    ok = mma_pass<S, 0, WIDE>(acc0, KB, u, ph, smem_base, full_bar, empty_bar, args.err);
                else if constexpr (oz_npass(S) > 1)
                    ok = mma_pass<S, 1>(acc0, KB, u, ph, smem_base, full_bar, empty_bar, args.err);
                if (!ok) *abort_flag = 1;
                mma_commit(pass_bar);  // the pass's accumulators are final once its MMAs complete
            }
        }
    } else {
        // epilogue warps 2..5 cover TMEM lane quarters (warp % 4)
        const int quarter = warp & 3;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const int row = m0 + quarter * 32 + lane;
        const bool row_ok = row < args.m;
        const double rowscale = row_ok ? ldexp(kUnit, args.ea[za + row]) : 0.0;
        if constexpr (oz_float(S)) {
            // segment sums: FP32 accumulator -> FP64, added to the parked sums (columns 256 + c 32
            // high words, 384 + c 32 low words), stored to D after the last segment
            const int nseg = max(1, (KB + kseg - 1) / kseg);
            for (int sg = 0; sg < nseg; ++sg) {
                const int b = sg & 1;
                const bool ok = mbar_wait(&acc_full[b], (sg >> 1) & 1, args.err, 4);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (!ok || *abort_flag) break;
                const bool filled = sg * kseg < KB, last = (sg + 1 == nseg);
#pragma unroll 1
                for (int c = 0; c < BN / 32; ++c) {
                    double acc[32];
                    uint32_t v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[j] = 0.0;
                    if (filled) {
                        tmem_ld32(lane_base + (uint32_t)b * BN + c * 32, v);
#pragma unroll
                        for (int j = 0; j < 32; ++j) acc[j] = (double)__uint_as_float(v[j]);
                    }
                    if (sg > 0) {
                        uint32_t hi[32], lo[32];
                        tmem_ld32(lane_base + 256 + c * 32, hi);
                        tmem_ld32(lane_base + 384 + c * 32, lo);
#pragma unroll
                        for (int j = 0; j < 32; ++j) acc[j] += __hiloint2double((int)hi[j], (int)lo[j]);
                    }
                    if (!last) {
                        uint32_t hi[32], lo[32];
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            hi[j] = (uint32_t)__double2hiint(acc[j]);
                            lo[j] = (uint32_t)__double2loint(acc[j]);
                        }
                        tmem_st32(lane_base + 256 + c * 32, hi);
                        tmem_st32(lane_base + 384 + c * 32, lo);
                    } else if (row_ok) {
                        store_row_chunk(args, Dz, row, n0 + c * 32, acc, rowscale, colscale + c * 32,
                                        args.accumulate != 0);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(&acc_empty[b]);  // accumulator b may take segment sg + 2
            }
        }
        // Single-pass int8 tiles with a plain row-major D: the scaled tile goes through shared memory (the
        // ring, idle once the last MMA has completed) and out as whole rows, so that a warp's stores are
        // 32 consecutive doubles instead of one double in each of 32 rows.  Same values, same order of
        // operations as store_row_chunk; for short k (a few k-blocks) the store is most of the tile's time.
        constexpr bool kStageable = oz_npass(S) == 1 && !oz_float(S);
        const bool staged = kStageable && args.gamma_n == 0 && !args.trans && !args.ct;
        if (staged) {
            const bool ok = mbar_wait(pass_bar, 0, args.err, 4);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool go = ok && !*abort_flag;
            constexpr int TP = BN + 1;  // row pitch in doubles: a warp's column-j writes hit distinct banks
            double *T = reinterpret_cast<double *>(smem);
            const int rl = quarter * 32 + lane;
            if (go) {
#pragma unroll 1
                for (int c = 0; c < BN / 32; ++c) {
                    double acc[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[j] = 0.0;
#pragma unroll 1
                    for (int g = oz_g1(S, 0); g >= oz_g0(0) && KB > 0; --g) {
                        uint32_t v[32];
                        tmem_ld32(lane_base + (uint32_t)(g - oz_g0(0)) * BN + c * 32, v);
                        const double sc = kPow254[g - 2];
#pragma unroll
                        for (int j = 0; j < 32; ++j) acc[j] = fma((double)(int)v[j], sc, acc[j]);
                    }
                    const double *cs = colscale + c * 32;
#pragma unroll
                    for (int j = 0; j < 32; ++j) T[rl * TP + c * 32 + j] = acc[j] * rowscale * cs[j];
                }
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");  // the four epilogue warps
            if (go) {
                const bool add = args.accumulate != 0;
#pragma unroll 1
                for (int r = quarter * 32; r < quarter * 32 + 32; ++r) {
                    const int grow = m0 + r;
                    if (grow >= args.m) break;
                    double *drow = Dz + (long long)grow * args.ldd + n0;
                    const double *trow = T + r * TP;
#pragma unroll
                    for (int c = lane; c < BN; c += 32) {
                        if (n0 + c < args.n) drow[c] = add ? drow[c] + trow[c] : trow[c];
                    }
                }
            }
        }
        for (int p = 0; p < npass && !oz_float(S) && !staged; ++p) {
            const bool ok = mbar_wait(pass_bar, p & 1, args.err, 4);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (!ok || *abort_flag) break;
            const int g0 = p == 0 ? oz_g0(0) : oz_g0(1), g1 = p == 0 ? oz_g1(S, 0) : oz_g1(S, 1);
            const uint32_t acc0 = lane_base + ((p > 0 && keep) ? 256u : 0u);
            const bool last = (p + 1 == npass);
#pragma unroll 1
            for (int c = 0; c < BN / 32; ++c) {
                double acc[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) acc[j] = 0.0;
#pragma unroll 1
                for (int g = g1; g >= g0 && KB > 0; --g) {  // an empty k range contributes zero
                    uint32_t v[32];
                    tmem_ld32(acc0 + (uint32_t)(g - g0) * BN + c * 32, v);
                    const double sc = kPow254[g - 2];
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[j] = fma((double)(int)v[j], sc, acc[j]);
                }
                if (keep && p == 1) {  // add the first pass's partial sums
                    uint32_t hi[32], lo[32];
                    tmem_ld32(lane_base + c * 32, hi);
                    tmem_ld32(lane_base + 128 + c * 32, lo);
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[j] += __hiloint2double((int)hi[j], (int)lo[j]);
                }
                if (keep && !last) {  // park the partial sums over groups 2 and 3's chunk c (already read)
                    uint32_t hi[32], lo[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        hi[j] = (uint32_t)__double2hiint(acc[j]);
                        lo[j] = (uint32_t)__double2loint(acc[j]);
                    }
                    tmem_st32(lane_base + c * 32, hi);
                    tmem_st32(lane_base + 128 + c * 32, lo);
                } else if (row_ok) {
                    store_row_chunk(args, Dz, row, n0 + c * 32, acc, rowscale, colscale + c * 32,
                                    (p > 0 && !keep) || args.accumulate);
                }
            }
            if (!last) {
                if (keep) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(free_bar);  // this thread's reads of the pass's accumulators are done
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base));
    }
}

// ------------------------------------------------------------------ slicing kernels
__device__ __forceinline__ int exp_of_max(double mx) {
    if (!(mx > 0.0) || !isfinite(mx)) return 0;
    int e;
    frexp(mx, &e);  // mx = f 2^e, f in [0.5, 1): |x| 2^-e < 1
    return e;
}

// Slicing of one value (balanced base-254 digits): with r = 127 x 2^-e (|r| < 127), slice t is
//     d_t = rint(r_t),  r_{t+1} = 254 (r_t - d_t),   r_0 = r,
// so every digit lies in [-127, 127] (|r_t - d_t| <= 1/2) and carries log2(254) ~ 8 bits:
//     x = 2^e / 127 * sum_t d_t 254^{-t} + O(2^e 254^{-S}).
// rint is the round-to-nearest addition of 1.5 * 2^52, whose low mantissa word is the digit as a
// 32-bit two's-complement integer -- plain FP64 adds, no integer/floating conversions (those are
// long-latency and dominated the slicing).  r_t - d_t is exact; 254 (r_t - d_t) rounds once.
struct SliceScale {
    double p1;  // 2^-e
    int e;
    bool fast;  // 2^-e is a normal double: one exact multiplication instead of ldexp
};

__device__ __forceinline__ double pow2_normal(int k) {  // 2^k for -1022 <= k <= 1023
    return __hiloint2double((1023 + k) << 20, 0);
}

__device__ __forceinline__ SliceScale slice_scale(int e, int S) {
    (void)S;
    SliceScale sc;
    sc.e = e;
    sc.fast = (e >= -1000 && e <= 1000);
    sc.p1 = sc.fast ? pow2_normal(-e) : 1.0;
    return sc;
}

__device__ __forceinline__ void slice_digits(double x, const SliceScale &sc, int S, int (&d)[OZ_MAX_S]) {
    constexpr double kRound = 6755399441055744.0;  // 1.5 * 2^52
    double r = (sc.fast ? x * sc.p1 : ldexp(x, -sc.e)) * 127.0;
#pragma unroll
    for (int t = 0; t < OZ_MAX_S; ++t) {
        if (t < S) {
            const double big = __dadd_rn(r, kRound);  // 1.5 * 2^52 + rint(r)
            d[t] = __double2loint(big);
            r = (r - (big - kRound)) * 254.0;
        } else {
            d[t] = 0;
        }
    }
}

// Floating-point formats of r = x 2^-e (|r| < 1).  BF16X3: hi = the BF16 nearest to (float) r,
// lo = the BF16 nearest to r - hi (exact in FP64), so that r - hi - lo = O(2^-17 |r|).  TF32: the
// FP32 value of r rounded to 10 fraction bits, ties away from zero (cvt.rna.tf32.f32), whose
// low 13 bits are zero.  Returned as raw bits: hi | lo << 16, or the TF32 word.
__device__ __forceinline__ uint32_t float_format_bits(double x, const SliceScale &sc, int S) {
    const double r = sc.fast ? x * sc.p1 : ldexp(x, -sc.e);
    if (S == OZ_FMT_TF32) {
        uint32_t t;
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(t) : "f"((float)r));
        return t;
    }
    const __nv_bfloat16 hi = __float2bfloat16_rn((float)r);
    const __nv_bfloat16 lo = __float2bfloat16_rn((float)(r - (double)__bfloat162float(hi)));
    return (uint32_t)__bfloat16_as_ushort(hi) | ((uint32_t)__bfloat16_as_ushort(lo) << 16);
}

// Slices of x for element k of row `row` of an operand slice buffer (rows_pad rows, KB k-blocks).
__device__ __forceinline__ void slice_value(double x, const SliceScale &sc, int S, signed char *out, long long row,
                                            long long rows_pad, long long KB, long long k) {
    if (oz_float(S)) {
        const uint32_t bits = float_format_bits(x, sc, S);
        if (S == OZ_FMT_TF32) {
            *reinterpret_cast<uint32_t *>(out + oz_float_offset(0, row, k, KB, S)) = bits;
        } else {
            *reinterpret_cast<unsigned short *>(out + oz_float_offset(0, row, k, KB, S)) = (unsigned short)bits;
            *reinterpret_cast<unsigned short *>(out + oz_float_offset(1, row, k, KB, S)) = (unsigned short)(bits >> 16);
        }
        return;
    }
    int d[OZ_MAX_S];
    slice_digits(x, sc, S, d);
#pragma unroll
    for (int t = 0; t < OZ_MAX_S; ++t)
        if (t < S) out[oz_slice_offset(t, row, k, rows_pad, KB, S)] = (signed char)d[t];
}

constexpr int SL_NT = 256;

__device__ double block_max(double v, double *sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + s]);
        __syncthreads();
    }
    double r = sh[0];
    __syncthreads();
    return r;
}

// Rows of a real matrix A (element (i, j) at A[i lda + j cs]) -> slices [S][mpad][kpad] and ea[m].
__global__ void __launch_bounds__(SL_NT) slice_rows_kernel(int m, int k, const double *A, long long lda, long long cs,
                                                           int S, long long mpad, long long kpad, signed char *out,
                                                           int *ea) {
    __shared__ double sh[SL_NT];
    const long long row = blockIdx.x;
    const double *a = A + row * lda;
    double mx = 0.0;
    for (int j = threadIdx.x; j < k; j += SL_NT) mx = fmax(mx, fabs(a[(long long)j * cs]));
    mx = block_max(mx, sh);
    const int e = exp_of_max(mx);
    if (threadIdx.x == 0) ea[row] = e;
    const SliceScale sc = slice_scale(e, S);
    for (long long j = threadIdx.x; j < kpad; j += SL_NT) {
        double x = (j < k) ? a[j * cs] : 0.0;
        slice_value(x, sc, S, out, row, mpad, kpad >> 5, j);
    }
}

// The same for short rows (kpad <= 1024): one warp per row, eight rows per CTA, the row maximum by
// warp shuffles (one CTA per row leaves most of a 256-thread block idle when k is a few hundred).
// Row r is row (r % inner) istride + r / inner of A (inner = 0: row r).
constexpr int SLW_ROWS = 8;
__global__ void __launch_bounds__(32 * SLW_ROWS) slice_rows_warp_kernel(int m, int k, const double *A, long long lda,
                                                                        long long cs, int S, long long mpad,
                                                                        long long kpad, signed char *out, int *ea,
                                                                        int inner, long long istride) {
    const long long row = (long long)blockIdx.x * SLW_ROWS + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= m) return;
    const double *a = A + (inner ? (row % inner) * istride + row / inner : row) * lda;
    double mx = 0.0;
    for (int j = lane; j < k; j += 32) mx = fmax(mx, fabs(a[(long long)j * cs]));
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const int e = exp_of_max(mx);
    if (lane == 0) ea[row] = e;
    const SliceScale sc = slice_scale(e, S);
    for (long long j = lane; j < kpad; j += 32) {
        double x = (j < k) ? a[j * cs] : 0.0;
        slice_value(x, sc, S, out, row, mpad, kpad >> 5, j);
    }
}

// Both density operands of one grid point w, from rho_w (M x M complex, interleaved spin order;
// element [r][q] at rho[w ws + r rs + q]) in two passes over it (column maxima, then digits):
//   exchange columns c = (4 w + 2 sigma + tau) 2 + part: part(rho_w[2l + sigma][2j + tau]) at k = l n + j;
//   Coulomb columns c = 2 w + part: part(P_w[l][j]), P_w = rho_aa + rho_bb (the spin-summed density).
// Thread-iteration (l, j) reads the 2 x 2 spin block of rho_w at rows 2l, 2l + 1, columns 2j, 2j + 1 as
// two 32-byte pieces, so consecutive j are consecutive 32-byte segments of the two rows; the ten
// values it yields (8 exchange, 2 Coulomb) keep ten running maxima.  rs and ws are even.
constexpr int SD_NT = 256;
__global__ void __launch_bounds__(SD_NT, 3) slice_density_kernel(int n, const zc *__restrict__ rho, long long rs,
                                                              long long ws, int S, long long npadK, long long npadP,
                                                              long long kpad, signed char *Ksl, int *eK,
                                                              signed char *Psl, int *eP) {
    __shared__ double sh[10][SD_NT / 32];
    const long long w = blockIdx.x;
    const zc *R = rho + w * ws;
    const int k = n * n;
    const long long KB = kpad >> 5;
    // the 2 x 2 block (l, j): v[2 sigma + tau] = rho_w[2l + sigma][2j + tau]
    auto block = [&](int e, zc (&v)[4]) {
        const int l = e / n, j = e - l * n;
        const double2 *r0 = reinterpret_cast<const double2 *>(R + (long long)(2 * l) * rs + 2 * j), *r1 = r0 + rs;
        const double2 a0 = __ldg(r0), a1 = __ldg(r0 + 1), b0 = __ldg(r1), b1 = __ldg(r1 + 1);
        v[0] = mkz(a0.x, a0.y);
        v[1] = mkz(a1.x, a1.y);
        v[2] = mkz(b0.x, b0.y);
        v[3] = mkz(b1.x, b1.y);
    };
    double mx[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) mx[q] = 0.0;
    for (int e = threadIdx.x; e < k; e += SD_NT) {
        zc v[4];
        block(e, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            mx[2 * q] = fmax(mx[2 * q], fabs(v[q].x));
            mx[2 * q + 1] = fmax(mx[2 * q + 1], fabs(v[q].y));
        }
        mx[8] = fmax(mx[8], fabs(v[0].x + v[3].x));
        mx[9] = fmax(mx[9], fabs(v[0].y + v[3].y));
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 10; ++q) {
        double m = mx[q];
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) sh[q][wid] = m;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 10; ++q) {
        double m = 0.0;
        for (int i = 0; i < SD_NT / 32; ++i) m = fmax(m, sh[q][i]);
        mx[q] = m;
    }
    SliceScale sc[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) sc[q] = slice_scale(exp_of_max(mx[q]), S);
#pragma unroll
    for (int q = 0; q < 8; ++q)
        if (threadIdx.x == q) eK[8 * w + q] = sc[q].e;
    if (threadIdx.x == 8) eP[2 * w] = sc[8].e;
    if (threadIdx.x == 9) eP[2 * w + 1] = sc[9].e;
    for (long long e = threadIdx.x; e < kpad; e += SD_NT) {
        zc v[4] = {mkz(0.0), mkz(0.0), mkz(0.0), mkz(0.0)};
        if (e < k) block((int)e, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            slice_value(v[q].x, sc[2 * q], S, Ksl, 8 * w + 2 * q, npadK, KB, e);
            slice_value(v[q].y, sc[2 * q + 1], S, Ksl, 8 * w + 2 * q + 1, npadK, KB, e);
        }
        slice_value(v[0].x + v[3].x, sc[8], S, Psl, 2 * w, npadP, KB, e);
        slice_value(v[0].y + v[3].y, sc[9], S, Psl, 2 * w + 1, npadP, KB, e);
    }
}

// Rows of one panel of the exchange matrix, EK[(i, k), (l, j)] = (il|kj) for i in [i0, i0 + I),
// from the panel's Gram block G[(i - i0) n + l][k n + j] = sum_L B_L[i][l] B_L[k][j] (row stride ldg):
// slice row r = (i - i0) n + k holds EK[(i, k), (l, j)] at k-index l n + j.  For fixed l the n
// values j are contiguous in G, so the reads run in coalesced segments of n doubles.
__global__ void __launch_bounds__(SL_NT) slice_ek_panel_kernel(int n, const double *G, long long ldg, int S,
                                                               long long rows_pad, long long kpad, signed char *out,
                                                               int *ea) {
    __shared__ double sh[SL_NT];
    const long long r = blockIdx.x;
    const int il = (int)(r / n), k = (int)(r - (long long)il * n);
    const double *g = G + (long long)il * n * ldg + (long long)k * n;  // + l ldg + j
    const int kk = n * n;
    double mx = 0.0;
    for (int e = threadIdx.x; e < kk; e += SL_NT) {
        const int l = e / n, j = e - l * n;
        mx = fmax(mx, fabs(g[(long long)l * ldg + j]));
    }
    mx = block_max(mx, sh);
    const int ex = exp_of_max(mx);
    if (threadIdx.x == 0) ea[r] = ex;
    const SliceScale sc = slice_scale(ex, S);
    for (long long e = threadIdx.x; e < kpad; e += SL_NT) {
        double x = 0.0;
        if (e < kk) {
            const int l = (int)(e / n), j = (int)(e - (long long)l * n);
            x = g[(long long)l * ldg + j];
        }
        slice_value(x, sc, S, out, r, rows_pad, kpad >> 5, e);
    }
}

// Symmetric exchange form.  For real integrals K(rho^T) = K(rho)^T, so with rho = rho_s + rho_a (its
// symmetric and antisymmetric halves) and the pairs (i <= k), resp. (i < k), of the index pairs:
//   K[i][k] = KS(i, k) + KA(i, k),  K[k][i] = KS(i, k) - KA(i, k),
//   KS(i, k) = sum_{l <= j} EKS[(i, k)][(l, j)] rho_s[l][j],  EKS = (il|kj) + (ij|kl) (l < j), (il|kl) (l = j),
//   KA(i, k) = sum_{l < j}  EKA[(i, k)][(l, j)] rho_a[l][j],  EKA = (il|kj) - (ij|kl),
// half the rows and half the contraction length of the full exchange matrix (KA(i, i) = 0).  Pairs are
// numbered in row order: pair_le(l, j) = l n - l (l - 1) / 2 + (j - l), pair_lt(l, j) = l (n - 1) - l (l - 1) / 2
// + (j - l - 1); the same numbering indexes the exchange rows and the contraction (k) elements.
__host__ __device__ __forceinline__ long long pair_le(long long n, long long l, long long j) {
    return l * n - l * (l - 1) / 2 + (j - l);
}
__host__ __device__ __forceinline__ long long pair_lt(long long n, long long l, long long j) {
    return l * (n - 1) - l * (l - 1) / 2 + (j - l - 1);
}

// Symmetric and antisymmetric exchange rows of one panel from its Gram block: pair (i, k), i <= k, of
// symmetric panel row r = pairs[t0 + r] (t0 = pair_le(i0, i0)) reads the n x n block
// B[l][j] = G[(i - i0) n + l][(k - k0) n + j] = (il|kj) (row stride ldg) and writes symmetric row r
// (EKS at k-index pair_le(l, j)) and, when i < k, antisymmetric row ra = r - (i - i0) - 1 (EKA at
// pair_lt(l, j); the panel's diagonal pairs precede it).  The block goes through shared memory as the
// 32 x 32 tile pairs B[lt][jt], B[jt][lt] (lt <= jt), so that B[l][j] and B[j][l] are both read in
// coalesced rows, twice: row maxima, then slices.  Exponents e_s[r], e_a[ra].
constexpr int EKS_TP = 33;  // tile pitch (doubles): row and column reads of a warp hit distinct banks
__global__ void __launch_bounds__(SL_NT) slice_ek_sym_panel_kernel(int n, int i0, int k0, const int *__restrict__ pairs,
                                                                   long long t0, const double *__restrict__ G,
                                                                   long long ldg, int S, long long rows_pad_s,
                                                                   long long kpad_s, signed char *out_s, int *e_s,
                                                                   long long rows_pad_a, long long kpad_a,
                                                                   signed char *out_a, int *e_a) {
    __shared__ double T1[32 * EKS_TP], T2[32 * EKS_TP];
    __shared__ double sh[SL_NT];
    const long long r = blockIdx.x;
    const int pr = __ldg(pairs + t0 + r), i = pr >> 16, k = pr & 0xffff;
    const bool anti = i < k;
    const long long ra = r - (i - i0) - 1;
    const double *g = G + (long long)(i - i0) * n * ldg + (long long)(k - k0) * n;
    const int nt = (n + 31) / 32, lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const long long kks = (long long)n * (n + 1) / 2, kka = (long long)n * (n - 1) / 2;
    double mxs = 0.0, mxa = 0.0;
    SliceScale scs = slice_scale(0, S), sca = slice_scale(0, S);
    for (int pass = 0; pass < 2; ++pass) {
        for (int lt = 0; lt < nt; ++lt) {
            for (int jt = lt; jt < nt; ++jt) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int a = ty + 8 * q;
                    const int l1 = lt * 32 + a, j1 = jt * 32 + lane;
                    T1[a * EKS_TP + lane] = (l1 < n && j1 < n) ? g[(long long)l1 * ldg + j1] : 0.0;
                    if (jt != lt) {
                        const int l2 = jt * 32 + a, j2 = lt * 32 + lane;
                        T2[a * EKS_TP + lane] = (l2 < n && j2 < n) ? g[(long long)l2 * ldg + j2] : 0.0;
                    }
                }
                __syncthreads();
                const double *U = (jt == lt) ? T1 : T2;  // U[b][a] = B[jt 32 + b][lt 32 + a]
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int a = ty + 8 * q, l = lt * 32 + a, j = jt * 32 + lane;
                    if (l <= j && j < n) {
                        const double x = T1[a * EKS_TP + lane], y = U[lane * EKS_TP + a];
                        const double sv = (l == j) ? x : x + y, av = x - y;
                        if (pass == 0) {
                            mxs = fmax(mxs, fabs(sv));
                            if (l < j) mxa = fmax(mxa, fabs(av));
                        } else {
                            slice_value(sv, scs, S, out_s, r, rows_pad_s, kpad_s >> 5, pair_le(n, l, j));
                            if (anti && l < j) slice_value(av, sca, S, out_a, ra, rows_pad_a, kpad_a >> 5, pair_lt(n, l, j));
                        }
                    }
                }
                __syncthreads();
            }
        }
        if (pass == 0) {
            mxs = block_max(mxs, sh);
            mxa = block_max(mxa, sh);
            const int es = exp_of_max(mxs), ea = exp_of_max(mxa);
            if (threadIdx.x == 0) {
                e_s[r] = es;
                if (anti) e_a[ra] = ea;
            }
            scs = slice_scale(es, S);
            sca = slice_scale(ea, S);
        }
    }
    for (long long e = kks + threadIdx.x; e < kpad_s; e += SL_NT) slice_value(0.0, scs, S, out_s, r, rows_pad_s, kpad_s >> 5, e);
    if (anti)
        for (long long e = kka + threadIdx.x; e < kpad_a; e += SL_NT)
            slice_value(0.0, sca, S, out_a, ra, rows_pad_a, kpad_a >> 5, e);
}

// Density operands of one grid point w in the symmetric exchange form, from rho_w (element [r][q] at
// rho[w ws + r rs + q], as slice_density_kernel), rho^{st}[l][j] = rho_w[2l + s][2j + t], over the pairs
// l <= j (pairs[t] = l << 16 | j, t = pair_le(l, j)):
//   symmetric exchange columns c = (4w + 2s + t) 2 + part at k-index t: part of rho_s^{st}[l][j] =
//     (rho^{st}[l][j] + rho^{st}[j][l]) / 2;
//   antisymmetric exchange columns (same c) at k-index pair_lt(l, j), l < j: part of rho_a^{st}[l][j] =
//     (rho^{st}[l][j] - rho^{st}[j][l]) / 2;
//   Coulomb columns c = 2w + part at k-index t: part of the symmetric half of P = rho^{aa} + rho^{bb} (the
//     Cholesky operand holds B_L[l][j] (2 - delta_lj) there: sum_lj B_L[l][j] P[l][j] with B_L symmetric).
// Each pair reads the 2 x 2 spin blocks (l, j) and (j, l) as two 32-byte pieces each; 18 running
// maxima, then the slices.
constexpr int SDS_NT = 256;
__global__ void __launch_bounds__(SDS_NT, 2) slice_density_sym_kernel(int n, const int *__restrict__ pairs,
                                                                     const zc *__restrict__ rho, long long rs,
                                                                     long long ws, int S, long long npadK,
                                                                     long long kpad_s, long long kpad_a,
                                                                     signed char *Ks, int *eKs, signed char *Ka,
                                                                     int *eKa, long long npadP, signed char *Psl,
                                                                     int *eP) {
    __shared__ double sh[18][SDS_NT / 32];
    __shared__ int exs[18];
    const long long w = blockIdx.x;
    const zc *R = rho + w * ws;
    const long long kks = (long long)n * (n + 1) / 2, kka = (long long)n * (n - 1) / 2;
    auto block = [&](int l, int j, zc (&v)[4]) {
        const double2 *r0 = reinterpret_cast<const double2 *>(R + (long long)(2 * l) * rs + 2 * j), *r1 = r0 + rs;
        const double2 a0 = __ldg(r0), a1 = __ldg(r0 + 1), b0 = __ldg(r1), b1 = __ldg(r1 + 1);
        v[0] = mkz(a0.x, a0.y);
        v[1] = mkz(a1.x, a1.y);
        v[2] = mkz(b0.x, b0.y);
        v[3] = mkz(b1.x, b1.y);
    };
    // halves of pair t: sv (symmetric), av (antisymmetric, zero for l = j)
    auto halves = [&](long long t, zc (&sv)[4], zc (&av)[4], int &l, int &j) {
        const int pr = __ldg(pairs + t);
        l = pr >> 16;
        j = pr & 0xffff;
        zc v[4];
        block(l, j, v);
        if (l == j) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                sv[q] = v[q];
                av[q] = mkz(0.0);
            }
        } else {
            zc u[4];
            block(j, l, u);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                sv[q] = mkz(0.5 * (v[q].x + u[q].x), 0.5 * (v[q].y + u[q].y));
                av[q] = mkz(0.5 * (v[q].x - u[q].x), 0.5 * (v[q].y - u[q].y));
            }
        }
    };
    {
        double mx[18];
#pragma unroll
        for (int q = 0; q < 18; ++q) mx[q] = 0.0;
        for (long long t = threadIdx.x; t < kks; t += SDS_NT) {
            zc sv[4], av[4];
            int l, j;
            halves(t, sv, av, l, j);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                mx[2 * q] = fmax(mx[2 * q], fabs(sv[q].x));
                mx[2 * q + 1] = fmax(mx[2 * q + 1], fabs(sv[q].y));
                mx[8 + 2 * q] = fmax(mx[8 + 2 * q], fabs(av[q].x));
                mx[9 + 2 * q] = fmax(mx[9 + 2 * q], fabs(av[q].y));
            }
            mx[16] = fmax(mx[16], fabs(sv[0].x + sv[3].x));
            mx[17] = fmax(mx[17], fabs(sv[0].y + sv[3].y));
        }
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            double m = mx[q];
            for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0) sh[q][wid] = m;
        }
        __syncthreads();
        if (threadIdx.x < 18) {
            double m = 0.0;
            for (int i = 0; i < SDS_NT / 32; ++i) m = fmax(m, sh[threadIdx.x][i]);
            const int e = exp_of_max(m);
            exs[threadIdx.x] = e;
            if (threadIdx.x < 8) eKs[8 * w + threadIdx.x] = e;
            else if (threadIdx.x < 16) eKa[8 * w + threadIdx.x - 8] = e;
            else eP[2 * w + threadIdx.x - 16] = e;
        }
        __syncthreads();
    }
    const long long KBs = kpad_s >> 5, KBa = kpad_a >> 5;
    for (long long t = threadIdx.x; t < kpad_s; t += SDS_NT) {
        zc sv[4] = {mkz(0.0), mkz(0.0), mkz(0.0), mkz(0.0)}, av[4] = {mkz(0.0), mkz(0.0), mkz(0.0), mkz(0.0)};
        int l = 0, j = 0;
        if (t < kks) halves(t, sv, av, l, j);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            slice_value(sv[q].x, slice_scale(exs[2 * q], S), S, Ks, 8 * w + 2 * q, npadK, KBs, t);
            slice_value(sv[q].y, slice_scale(exs[2 * q + 1], S), S, Ks, 8 * w + 2 * q + 1, npadK, KBs, t);
        }
        slice_value(sv[0].x + sv[3].x, slice_scale(exs[16], S), S, Psl, 2 * w, npadP, KBs, t);
        slice_value(sv[0].y + sv[3].y, slice_scale(exs[17], S), S, Psl, 2 * w + 1, npadP, KBs, t);
        if (t < kks && l < j) {
            const long long u = pair_lt(n, l, j);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                slice_value(av[q].x, slice_scale(exs[8 + 2 * q], S), S, Ka, 8 * w + 2 * q, npadK, KBa, u);
                slice_value(av[q].y, slice_scale(exs[9 + 2 * q], S), S, Ka, 8 * w + 2 * q + 1, npadK, KBa, u);
            }
        }
    }
    for (long long u = kka + threadIdx.x; u < kpad_a; u += SDS_NT) {
#pragma unroll
        for (int q = 0; q < 8; ++q) slice_value(0.0, slice_scale(exs[8 + q], S), S, Ka, 8 * w + q, npadK, KBa, u);
    }
}

// Operands of the batched product F_w X_w (one per grid point w; F = H1 + J - K, M x M complex; X, M x N)
// as int8 slices, with (F X)[c][j] = sum_i F[c][i] X[i][j] written as real dot products over k = 2i + part:
//   orbital rows  r = w N + j:        (Re X[i][j], Im X[i][j])       at k = 2i, 2i + 1
//   Fock rows     r = w 2M + 2c:      (Re F[c][i], -Im F[c][i])      -> Re (F X)[c][j]
//                 r = w 2M + 2c + 1:  (Im F[c][i],  Re F[c][i])      -> Im (F X)[c][j]
// Each row takes the exponent of its largest |Re| or |Im| (one exponent for both Fock rows of c).
//
// Fock rows: a warp per complex row c of F_w (at F + w fs + c M, contiguous), a lane per two elements
// i, i + 1.  The digits of Re and Im are formed once (those of -x are the negated digits of x: rint is
// symmetric) and each row's four bytes k = 2i .. 2i + 3 are one 4-byte store per slice.
__global__ void __launch_bounds__(32 * SLW_ROWS) slice_fock_rows_kernel(int M, long long nrows, const zc *F,
                                                                        long long fs, int S, long long rows_pad,
                                                                        long long kpad, signed char *out, int *eb) {
    const long long q = (long long)blockIdx.x * SLW_ROWS + (threadIdx.x >> 5);  // q = w M + c
    const int lane = threadIdx.x & 31;
    if (q >= nrows) return;
    const long long w = q / M, c = q - w * M;
    const double2 *f = reinterpret_cast<const double2 *>(F + w * fs + c * M);
    double mx = 0.0;
    for (int i = lane; i < M; i += 32) {
        const double2 v = f[i];
        mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
    }
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const int e = exp_of_max(mx);
    const long long r = 2 * q;
    if (lane == 0) {
        eb[r] = e;
        eb[r + 1] = e;
    }
    const SliceScale sc = slice_scale(e, S);
    const long long KB = kpad >> 5;
    for (long long i = 2 * lane; 2 * i < kpad; i += 64) {  // kpad is a multiple of 32: k = 2i .. 2i + 3 < kpad
        unsigned int u0[OZ_MAX_S], u1[OZ_MAX_S];
#pragma unroll
        for (int t = 0; t < OZ_MAX_S; ++t) u0[t] = u1[t] = 0u;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double re = 0.0, im = 0.0;
            if (i + h < M) {
                const double2 v = f[i + h];
                re = v.x;
                im = v.y;
            }
            int dr[OZ_MAX_S], di[OZ_MAX_S];
            slice_digits(re, sc, S, dr);
            slice_digits(im, sc, S, di);
#pragma unroll
            for (int t = 0; t < OZ_MAX_S; ++t) {
                // row r: (Re, -Im); row r + 1: (Im, Re) -- little-endian: the lowest k in the low byte
                u0[t] |= (unsigned int)((dr[t] & 0xff) | ((-di[t] & 0xff) << 8)) << (16 * h);
                u1[t] |= (unsigned int)((di[t] & 0xff) | ((dr[t] & 0xff) << 8)) << (16 * h);
            }
        }
#pragma unroll
        for (int t = 0; t < OZ_MAX_S; ++t)
            if (t < S) {
                *reinterpret_cast<unsigned int *>(out + oz_slice_offset(t, r, 2 * i, rows_pad, KB, S)) = u0[t];
                *reinterpret_cast<unsigned int *>(out + oz_slice_offset(t, r + 1, 2 * i, rows_pad, KB, S)) = u1[t];
            }
    }
}

// Orbital rows: a CTA per 32 columns j0 .. j0 + 31 of one point's X_w (X_w[i][j] at X + i ld + w N + j).
// The maxima come from coalesced reads of X's rows; the slices go through 32 x 32 tiles of X in shared
// memory, each of the CTA's 256 threads taking 4 consecutive elements i of one row per tile: 8
// consecutive k (Re, Im interleaved) written as one 8-byte store per slice.  The tiles cover k up to the
// next multiple of 64 past 2M; the stores stop at kpad (zeros beyond 2M are the padding).
constexpr int SXC_NT = 256;
__global__ void __launch_bounds__(SXC_NT) slice_xcols_kernel(int M, int N, const zc *__restrict__ X, long long ld,
                                                             int S, long long rows_pad, long long kpad,
                                                             signed char *out, int *ea) {
    __shared__ zc T[32][33];
    __shared__ double smx[SXC_NT / 32][32];
    __shared__ int sexp[32];
    const long long w = blockIdx.x;
    const int j0 = blockIdx.y * 32;
    const int tid = threadIdx.x, jj = tid & 31, ii = tid >> 5;
    const bool jok = j0 + jj < N;
    const zc *Xw = X + w * N + j0;
    double mx = 0.0;
    if (jok)
        for (int i = ii; i < M; i += SXC_NT / 32) {
            const zc v = Xw[(long long)i * ld + jj];
            mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
        }
    smx[ii][jj] = mx;
    __syncthreads();
    if (tid < 32) {
        double m = 0.0;
        for (int q = 0; q < SXC_NT / 32; ++q) m = fmax(m, smx[q][tid]);
        const int e = exp_of_max(m);
        sexp[tid] = e;
        if (j0 + tid < N) ea[w * N + j0 + tid] = e;
    }
    __syncthreads();
    const int jr = tid >> 3, seg = tid & 7;
    const bool rok = j0 + jr < N;
    const SliceScale sc = slice_scale(sexp[jr], S);
    const long long row = w * N + j0 + jr, KB = kpad >> 5;
    for (int i0 = 0; i0 < M; i0 += 32) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = i0 + ii + 8 * q;
            T[ii + 8 * q][jj] = (jok && i < M) ? Xw[(long long)i * ld + jj] : mkz(0.0);
        }
        __syncthreads();
        const long long k0 = 2LL * (i0 + 4 * seg);  // a multiple of 8: the 8 bytes lie in one 32-byte k-block
        if (rok && k0 < kpad) {
            unsigned long long word[OZ_MAX_S];
#pragma unroll
            for (int t = 0; t < OZ_MAX_S; ++t) word[t] = 0ull;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const zc v = T[4 * seg + q][jr];
                int dr[OZ_MAX_S], di[OZ_MAX_S];
                slice_digits(v.x, sc, S, dr);
                slice_digits(v.y, sc, S, di);
#pragma unroll
                for (int t = 0; t < OZ_MAX_S; ++t)
                    word[t] |= ((unsigned long long)(dr[t] & 0xff) << (16 * q)) |
                               ((unsigned long long)(di[t] & 0xff) << (16 * q + 8));
            }
#pragma unroll
            for (int t = 0; t < OZ_MAX_S; ++t)
                if (t < S) *reinterpret_cast<unsigned long long *>(out + oz_slice_offset(t, row, k0, rows_pad, KB, S)) =
                               word[t];
        }
        __syncthreads();
    }
}

// Rows of the Cholesky operand of the symmetric Coulomb contraction: row L holds B_L[l][j] (2 - delta_lj)
// (off = 2, or B_L[l][j] with off = 1) at k-index pair_le(l, j) (B_L[l][j] = Bst[L n^2 + l n + j]), as FP64 rows of length n (n + 1) / 2.
__global__ void cholesky_pairs_kernel(int n, int L, const double *__restrict__ Bst, const int *__restrict__ pairs,
                                      double *out, double off) {
    const long long kks = (long long)n * (n + 1) / 2, tot = kks * L, n2 = (long long)n * n;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot;
         e += (long long)gridDim.x * blockDim.x) {
        const long long row = e / kks, t = e - row * kks;
        const int pr = pairs[t], l = pr >> 16, j = pr & 0xffff;
        const double b = Bst[row * n2 + (long long)l * n + j];
        out[e] = l == j ? b : off * b;
    }
}

// ------------------------------------------------------------------ fused density + operand slicing
// D (8 x 8) += A (8 x 4, row-major) B (4 x 8, column-major), FP64 tensor cores.
__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// ERI form with n <= 64: the exchange (K) and Coulomb (P) operand columns straight from X_w and
// bra, without writing the M x M density to HBM.  CTA (w, pair): pair 0 forms rho_aa, rho_bb and
// P = rho_aa + rho_bb, pair 1 forms rho_ab and rho_ba, each as
//     rho_st[l][j] = sum_m X_w[2l+s][m] conj(bra[2j+t][m])
// with the tensor-core MMA sequence of zgemm_kernel (m ascending in steps of four), so every
// column, its exponent and its slices are those of the density GEMM followed by slice_rho_cols /
// slice_p_cols.  A cluster of two CTAs shares each (w, pair): CTA rank r forms rows
// l in [32 r, 32 r + 32) and slices that part of every column; the column maxima (one exponent per
// column) are combined through distributed shared memory.  Two such CTAs fit on an SM, so one
// CTA's FP64 MMAs overlap another's slicing.
// threads, m-chunk, padded row pitch (complex).  A 16-byte fragment load is served eight lanes at a
// time; lanes (fk, fr) of one such group read row kk + fk, column c + fr, so with a pitch of 2 mod 8
// (complex) the eight land on distinct bank quadruples.
constexpr int RS_NT = 256, RS_MC = 16, RS_P = 66;
constexpr int RS_WI = 2;     // 8-row fragments per warp: 8 warps of 16 x 16 cover 32 rows x 64 columns
constexpr int RS_ROWS = 32;  // density rows l per CTA: the two CTAs of a cluster take l < 32 and l >= 32

// operand staging (2 x 2 x RS_MC x RS_P complex), reused for two half density columns (2 x 32 x 64
// doubles)
size_t rs_smem_bytes() {
    return std::max((size_t)2 * 2 * RS_MC * RS_P * sizeof(zc), (size_t)2 * RS_ROWS * 64 * sizeof(double));
}

// Slices of four consecutive k-elements e0..e0+3 (one 32-element block) of a column, packed four
// to a 32-bit word (byte v = element e0 + v), one store per slice; for the floating-point formats
// one 16-byte store (TF32) or two 8-byte stores (BF16 high parts, low parts).
template <int S>
__device__ __forceinline__ void slice_pack4(const double (&x)[4], const SliceScale &sc, signed char *out, long long row,
                                            long long rows_pad, long long KB, long long e0) {
    if constexpr (oz_float(S)) {
        uint32_t b[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) b[v] = float_format_bits(x[v], sc, S);
        if constexpr (S == OZ_FMT_TF32) {
            *reinterpret_cast<uint4 *>(out + oz_float_offset(0, row, e0, KB, S)) = make_uint4(b[0], b[1], b[2], b[3]);
        } else {
            *reinterpret_cast<uint2 *>(out + oz_float_offset(0, row, e0, KB, S)) =
                make_uint2((b[0] & 0xFFFFu) | (b[1] << 16), (b[2] & 0xFFFFu) | (b[3] << 16));
            *reinterpret_cast<uint2 *>(out + oz_float_offset(1, row, e0, KB, S)) =
                make_uint2((b[0] >> 16) | (b[1] & 0xFFFF0000u), (b[2] >> 16) | (b[3] & 0xFFFF0000u));
        }
    } else {
        uint32_t wd[S];
#pragma unroll
        for (int t = 0; t < S; ++t) wd[t] = 0u;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            int d[OZ_MAX_S];
            slice_digits(x[v], sc, S, d);
#pragma unroll
            for (int t = 0; t < S; ++t) wd[t] |= ((uint32_t)d[t] & 0xFFu) << (8 * v);
        }
#pragma unroll
        for (int t = 0; t < S; ++t)
            *reinterpret_cast<uint32_t *>(out + oz_slice_offset(t, row, e0, rows_pad, KB, S)) = wd[t];
    }
}

template <int S>
__global__ void __launch_bounds__(RS_NT, 2) rho_slice_kernel(int n, int N, const zc *__restrict__ Xs, long long ld,
                                                             const zc *__restrict__ bra, long long npadK,
                                                             long long npadP, long long kpad, signed char *outK,
                                                             int *ebK, signed char *outP, int *ebP) {
    extern __shared__ __align__(16) unsigned char rs_smem[];
    zc *xs = reinterpret_cast<zc *>(rs_smem);  // [s][mm][l - r0]: X_w[2l+s][m0+mm] at (s RS_MC + mm) RS_P + l - r0
    zc *bs = xs + 2 * RS_MC * RS_P;            // [t][mm][j]: bra[2j+t][m0+mm]
    double *stage = reinterpret_cast<double *>(rs_smem);  // this CTA's part of two columns after the products
    __shared__ double red[6 * (RS_NT / 32)];
    __shared__ double cmax[6];  // this CTA's column maxima, read by the other CTA of the cluster
    const int tid = threadIdx.x;
    uint32_t rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const long long w = blockIdx.x >> 2;
    const int pair = (int)((blockIdx.x >> 1) & 1);
    const int r0 = (int)rank * RS_ROWS;  // first density row of this CTA
    // warp tile: rows r0 + wr + 8 bi + fr, columns wc + 8 bj + 2 fk + h of both spin blocks q = 0, 1,
    // as FP64 tensor-core products (mma.sync m8n8k4: lane l holds A[l/4][l%4], B[l%4][l/4],
    // D[l/4][2 (l%4) + h]), four real MMAs per complex step in the order of zgemm_kernel
    const int lane = tid & 31, warp = tid >> 5;
    const int wr = (warp >> 2) * (8 * RS_WI), wc = (warp & 3) * 16, fr = lane >> 2, fk = lane & 3;
    double cr[2][RS_WI][2][2], ci[2][RS_WI][2][2];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < RS_WI; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) cr[q][i][j][0] = cr[q][i][j][1] = ci[q][i][j][0] = ci[q][i][j][1] = 0.0;

    for (int m0 = 0; m0 < N; m0 += RS_MC) {
        const int mc = min(RS_MC, N - m0);
        __syncthreads();
        for (int idx = tid; idx < 2 * 64 * RS_MC; idx += RS_NT) {  // mm fastest: 256-byte row runs
            const int mm = idx % RS_MC, l = (idx / RS_MC) & 63, sp = idx / (RS_MC * 64);
            zc bv = {0.0, 0.0};
            if (l < n && mm < mc) bv = bra[(long long)(2 * l + sp) * N + m0 + mm];
            bs[(sp * RS_MC + mm) * RS_P + l] = bv;
        }
        for (int idx = tid; idx < 2 * RS_ROWS * RS_MC; idx += RS_NT) {
            const int mm = idx % RS_MC, ll = (idx / RS_MC) % RS_ROWS, sp = idx / (RS_MC * RS_ROWS);
            const int l = r0 + ll;
            zc xv = {0.0, 0.0};
            if (l < n && mm < mc) xv = Xs[(long long)(2 * l + sp) * ld + w * N + m0 + mm];
            xs[(sp * RS_MC + mm) * RS_P + ll] = xv;
        }
        __syncthreads();
        for (int kk = 0; kk < mc; kk += 4) {  // zero-padded beyond mc
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int sg = q, tu = pair ? 1 - q : q;
                zc b[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    b[j] = bs[(tu * RS_MC + kk + fk) * RS_P + wc + 8 * j + fr];
                    b[j].y = -b[j].y;  // conj(bra)
                }
#pragma unroll
                for (int i = 0; i < RS_WI; ++i) {
                    const zc a = xs[(sg * RS_MC + kk + fk) * RS_P + wr + 8 * i + fr];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        dmma884(cr[q][i][j], a.x, b[j].x);
                        dmma884(cr[q][i][j], -a.y, b[j].y);
                        dmma884(ci[q][i][j], a.x, b[j].y);
                        dmma884(ci[q][i][j], a.y, b[j].x);
                    }
                }
            }
        }
    }

    // columns of this CTA: K (q, part) for q = 0, 1; for pair 0 also P (part)
    const int ncol = pair == 0 ? 6 : 4;
    const int nn = n * n;
    auto value = [&](int col, int i, int j, int h) -> double {
        const int part = col & 1;
        if (col < 2) return part ? ci[0][i][j][h] : cr[0][i][j][h];
        if (col < 4) return part ? ci[1][i][j][h] : cr[1][i][j][h];
        return part ? ci[0][i][j][h] + ci[1][i][j][h] : cr[0][i][j][h] + cr[1][i][j][h];
    };
    // column maxima over this CTA's rows: warp shuffles, then the 8 warps through shared memory
    double mx[6];
#pragma unroll
    for (int col = 0; col < 6; ++col) mx[col] = 0.0;
#pragma unroll
    for (int i = 0; i < RS_WI; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if ((r0 + wr + 8 * i + fr < n) && (wc + 8 * j + 2 * fk + h < n)) {
#pragma unroll
                    for (int col = 0; col < 6; ++col)
                        if (col < ncol) mx[col] = fmax(mx[col], fabs(value(col, i, j, h)));
                }
#pragma unroll
    for (int col = 0; col < 6; ++col) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx[col] = fmax(mx[col], __shfl_xor_sync(0xffffffffu, mx[col], off));
        if (lane == 0) red[col * (RS_NT / 32) + warp] = mx[col];
    }
    __syncthreads();  // also orders the last reads of xs / bs before the stage writes
    if (tid < 6) {
        double m = 0.0;
#pragma unroll
        for (int wv = 0; wv < RS_NT / 32; ++wv) m = fmax(m, red[tid * (RS_NT / 32) + wv]);
        cmax[tid] = m;
    }
    // exchange the maxima with the other CTA of the cluster (every thread of both CTAs arrives)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    uint32_t peer_cmax;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer_cmax) : "r"(smem_u32(cmax)), "r"(rank ^ 1u));
    long long cidx[6];
    int ex[6];
#pragma unroll
    for (int col = 0; col < 6; ++col) {
        double other;
        asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(other) : "r"(peer_cmax + 8u * col) : "memory");
        ex[col] = exp_of_max(fmax(cmax[col], other));
        const int part = col & 1;
        if (col < 4) {
            const int q = col >> 1, sg = q, tu = pair ? 1 - q : q;
            cidx[col] = (w * 4 + sg * 2 + tu) * 2 + part;
        } else {
            cidx[col] = 2 * w + part;
        }
    }
    // the peer's maxima have been read: neither CTA leaves (or reuses cmax) before both have
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (rank == 0 && tid < ncol) {
#pragma unroll
        for (int col = 0; col < 6; ++col)
            if (col == tid) (col < 4 ? ebK : ebP)[cidx[col]] = ex[col];
    }
    // this CTA slices elements [e_lo, e_hi) of every column (element e = l n + c); rows l >= 32 and the
    // zero padding up to kpad belong to rank 1 unless n <= 32, when rank 0 covers the whole column
    const long long split = (RS_ROWS * n >= nn) ? kpad : (long long)RS_ROWS * n;
    const long long e_lo = rank ? split : 0, e_hi = rank ? kpad : split;
    const long long part_len = (long long)RS_ROWS * n;  // stage pitch of one column part
    // two columns per round through the stage, sliced four k-elements per store
#pragma unroll
    for (int c0 = 0; c0 < 6; c0 += 2) {
        if (c0 >= ncol) break;
#pragma unroll
        for (int i = 0; i < RS_WI; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ll = wr + 8 * i + fr, c = wc + 8 * j + 2 * fk + h;
                    if (r0 + ll < n && c < n) {
                        stage[ll * n + c] = value(c0, i, j, h);
                        stage[part_len + ll * n + c] = value(c0 + 1, i, j, h);
                    }
                }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int col = c0 + h;
            const bool isK = col < 4;
            const SliceScale sc = slice_scale(ex[col], S);
            const double *src = stage + h * part_len - (long long)r0 * n;  // indexed by the element e
            const bool pairs = (reinterpret_cast<uintptr_t>(stage + h * part_len) & 15u) == 0;  // 16-byte loads
            for (long long e0 = e_lo + 4LL * tid; e0 < e_hi; e0 += 4LL * RS_NT) {
                double x[4];
                if (pairs && e0 + 3 < nn) {
                    const double2 a = *reinterpret_cast<const double2 *>(src + e0);
                    const double2 b = *reinterpret_cast<const double2 *>(src + e0 + 2);
                    x[0] = a.x;
                    x[1] = a.y;
                    x[2] = b.x;
                    x[3] = b.y;
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) x[u] = (e0 + u < nn) ? src[e0 + u] : 0.0;
                }
                slice_pack4<S>(x, sc, isK ? outK : outP, cidx[col], isK ? npadK : npadP, kpad >> 5, e0);
            }
        }
        __syncthreads();  // the stage is rewritten by the next round
    }
}

// ------------------------------------------------------------------ host side
PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
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

// 2-D map over one slice group of an operand: dimension 0 = bytes of a row (KB k-block segments of
// seg_bytes), dimension 1 = rows; a box is box_bytes (default: one k-block segment) of box_rows rows,
// swizzled at its own width.
int make_group_map(CUtensorMap *map, const signed char *base, long long KB, int seg_bytes, long long rows_pad,
                   int box_rows, int box_bytes = 0) {
    if (box_bytes <= 0) box_bytes = seg_bytes;
    auto enc = get_encode();
    if (!enc) {
        set_error(PHF_ERR_CUDA, "cuTensorMapEncodeTiled entry point unavailable");
        return PHF_ERR_CUDA;
    }
    const long long rowb = KB * seg_bytes;
    cuuint64_t dims[2] = {(cuuint64_t)rowb, (cuuint64_t)rows_pad};
    cuuint64_t strides[1] = {(cuuint64_t)rowb};
    cuuint32_t box[2] = {(cuuint32_t)box_bytes, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<signed char *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE,
                     box_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                      : (box_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B),
                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error(PHF_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
        return PHF_ERR_CUDA;
    }
    return PHF_OK;
}

// Group-0 and group-1 maps of an operand's slice buffer (group 1 = group 0 when S <= 4: unused).
int make_slice_maps(CUtensorMap *g0, CUtensorMap *g1, const signed char *base, long long kpad, long long rows_pad,
                    int S, int box_rows) {
    const long long KB = kpad / OZ_BK;
    PHF_TRY(make_group_map(g0, base, KB, 128, rows_pad, box_rows));
    const int w = oz_g1_width(S);
    if (w == 0) {
        *g1 = *g0;
        return PHF_OK;
    }
    return make_group_map(g1, base + rows_pad * KB * 128, KB, 32 * w, rows_pad, box_rows);
}

// The wide issue's map of an operand's group-0 slices: one slice (32 bytes of a 128-byte k-block row)
// of box_rows rows per box, SWIZZLE_32B.
int make_wide_map(CUtensorMap *map, const signed char *base, long long kpad, long long rows_pad, int box_rows) {
    return make_group_map(map, base, kpad / OZ_BK, 128, rows_pad, box_rows, 32);
}

}  // namespace

long long oz_pad_rows(long long m) { return (m + OZ_BM - 1) / OZ_BM * OZ_BM; }
long long oz_pad_cols(long long n) { return (n + OZ_BN - 1) / OZ_BN * OZ_BN; }
long long oz_pad_k(long long k) { return (k + OZ_BK - 1) / OZ_BK * OZ_BK; }

int oz_slice_rows(int m, int k, const double *A, long long lda, int S, long long rows_pad, signed char *out, int *ea,
                  cudaStream_t st) {
    return oz_slice_rows_strided(m, k, A, lda, 1, S, rows_pad, out, ea, st);
}

int oz_slice_rows_strided(int m, int k, const double *A, long long lda, long long cs, int S, long long rows_pad,
                          signed char *out, int *ea, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    if (oz_pad_k(k) <= 1024)
        slice_rows_warp_kernel<<<(unsigned)((m + SLW_ROWS - 1) / SLW_ROWS), 32 * SLW_ROWS, 0, st>>>(
            m, k, A, lda, cs, S, rows_pad, oz_pad_k(k), out, ea, 0, 0);
    else
        slice_rows_kernel<<<m, SL_NT, 0, st>>>(m, k, A, lda, cs, S, rows_pad, oz_pad_k(k), out, ea);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_slice_point_rows(int M, int b, int bc, int k, const double *A, long long lda, int S, long long rows_pad,
                        signed char *out, int *ea, cudaStream_t st) {
    const long long m = (long long)M * bc;
    if (M < 1 || b < bc || m > rows_pad || m > 2147483647LL || !oz_format_ok(S)) {
        set_error(PHF_ERR_ARG, "oz_slice_point_rows: rows outside the slice buffer");
        return PHF_ERR_ARG;
    }
    ProfScope prof(st, PROF_MEMORY);
    slice_rows_warp_kernel<<<(unsigned)((m + SLW_ROWS - 1) / SLW_ROWS), 32 * SLW_ROWS, 0, st>>>(
        (int)m, k, A, lda, 1, S, rows_pad, oz_pad_k(k), out, ea, M, b);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_slice_density(int n, int bc, const zc *rho, long long rs, long long ws, int S, signed char *Ksl, int *eK,
                     long long npadK, signed char *Psl, int *eP, long long npadP, cudaStream_t st) {
    if (n < 1 || bc < 1 || 8LL * bc > npadK || 2LL * bc > npadP || !oz_format_ok(S) || (rs & 1) || (ws & 1)) {
        set_error(PHF_ERR_ARG, "oz_slice_density: columns outside the slice buffers or odd strides");
        return PHF_ERR_ARG;
    }
    ProfScope prof(st, PROF_MEMORY);
    slice_density_kernel<<<(unsigned)bc, SD_NT, 0, st>>>(n, rho, rs, ws, S, npadK, npadP, oz_pad_k((long long)n * n),
                                                          Ksl, eK, Psl, eP);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_slice_ek_panel(int n, int ipanel, const double *G, long long ldg, int S, long long rows_pad, signed char *out,
                      int *ea, cudaStream_t st) {
    const long long rows = (long long)ipanel * n;
    if (rows <= 0 || rows > rows_pad) {
        set_error(PHF_ERR_ARG, "oz_slice_ek_panel: panel rows outside the slice buffer");
        return PHF_ERR_ARG;
    }
    ProfScope prof(st, PROF_MEMORY);
    slice_ek_panel_kernel<<<(unsigned)rows, SL_NT, 0, st>>>(n, G, ldg, S, rows_pad, oz_pad_k((long long)n * n), out,
                                                            ea);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_slice_ek_sym_panel(int n, int i0, int ipanel, int k0, const int *pairs, const double *G, long long ldg, int S,
                          long long rows_pad_s, signed char *out_s, int *e_s, long long rows_pad_a, signed char *out_a,
                          int *e_a, cudaStream_t st) {
    const long long nn = n;
    // sum_{i = i0}^{i0 + ipanel - 1} (n - i) pairs (i, k >= i), of which ipanel are diagonal
    const long long rows_s = ipanel * (nn - i0) - (long long)ipanel * (ipanel - 1) / 2;
    const long long rows_a = rows_s - ipanel;
    if (n < 1 || n > 65535 || i0 < 0 || ipanel < 1 || i0 + ipanel > n || k0 < 0 || k0 > i0 || rows_s > rows_pad_s ||
        rows_a > rows_pad_a || ldg < (nn - k0) * nn) {
        set_error(PHF_ERR_ARG, "oz_slice_ek_sym_panel: panel rows outside the slice buffers or a short Gram block");
        return PHF_ERR_ARG;
    }
    ProfScope prof(st, PROF_MEMORY);
    slice_ek_sym_panel_kernel<<<(unsigned)rows_s, SL_NT, 0, st>>>(
        n, i0, k0, pairs, pair_le(nn, i0, i0), G, ldg, S, rows_pad_s, oz_pad_k(nn * (nn + 1) / 2), out_s, e_s,
        rows_pad_a, oz_pad_k(nn * (nn - 1) / 2), out_a, e_a);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_slice_density_sym(int n, int bc, const int *pairs, const zc *rho, long long rs, long long ws, int S,
                         signed char *Ks, int *eKs, signed char *Ka, int *eKa, long long npadK, signed char *Psl,
                         int *eP, long long npadP, cudaStream_t st) {
    if (n < 2 || n > 65535 || bc < 1 || 8LL * bc > npadK || 2LL * bc > npadP || !oz_format_ok(S) || (rs & 1) ||
        (ws & 1)) {
        set_error(PHF_ERR_ARG, "oz_slice_density_sym: columns outside the slice buffers or odd strides");
        return PHF_ERR_ARG;
    }
    const long long nn = n;
    ProfScope prof(st, PROF_MEMORY);
    slice_density_sym_kernel<<<(unsigned)bc, SDS_NT, 0, st>>>(n, pairs, rho, rs, ws, S, npadK,
                                                             oz_pad_k(nn * (nn + 1) / 2), oz_pad_k(nn * (nn - 1) / 2),
                                                             Ks, eKs, Ka, eKa, npadP, Psl, eP);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_slice_fock_rows(int M, int batch, const zc *F, long long fs, int S, long long rows_pad, signed char *out,
                       int *eb, cudaStream_t st) {
    const long long nrows = (long long)batch * M;
    if (M < 1 || batch < 1 || 2 * nrows > rows_pad || !oz_format_ok(S) || oz_float(S)) {
        set_error(PHF_ERR_ARG, "oz_slice_fock_rows: rows outside the slice buffer or a non-int8 format");
        return PHF_ERR_ARG;
    }
    ProfScope prof(st, PROF_MEMORY);
    slice_fock_rows_kernel<<<(unsigned)((nrows + SLW_ROWS - 1) / SLW_ROWS), 32 * SLW_ROWS, 0, st>>>(
        M, nrows, F, fs, S, rows_pad, oz_pad_k(2LL * M), out, eb);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_slice_xcols(int M, int N, int batch, const zc *X, long long ld, int S, long long rows_pad, signed char *out,
                   int *ea, cudaStream_t st) {
    if (M < 1 || N < 1 || batch < 1 || (long long)batch * N > rows_pad || !oz_format_ok(S) || oz_float(S)) {
        set_error(PHF_ERR_ARG, "oz_slice_xcols: rows outside the slice buffer or a non-int8 format");
        return PHF_ERR_ARG;
    }
    ProfScope prof(st, PROF_MEMORY);
    slice_xcols_kernel<<<dim3((unsigned)batch, (unsigned)((N + 31) / 32)), SXC_NT, 0, st>>>(
        M, N, X, ld, S, rows_pad, oz_pad_k(2LL * M), out, ea);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_cholesky_pairs(int n, int L, const double *Bst, const int *pairs, double *out, cudaStream_t st, double off) {
    ProfScope prof(st, PROF_MEMORY);
    cholesky_pairs_kernel<<<148 * 8, 256, 0, st>>>(n, L, Bst, pairs, out, off);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

bool oz_rho_slice_ok(int n) { return n >= 1 && n <= 64; }

int oz_rho_slice(int n, int N, int bc, const zc *Xs, long long ld, const zc *bra, int S, signed char *Ksl, int *eK,
                 signed char *Psl, int *eP, cudaStream_t st) {
    if (!oz_rho_slice_ok(n) || !oz_format_ok(S) || N < 1) {
        set_error(PHF_ERR_UNSUPPORTED, "oz_rho_slice: needs 1 <= n <= 64 and a valid operand format");
        return PHF_ERR_UNSUPPORTED;
    }
    using RsFn = void (*)(int, int, const zc *, long long, const zc *, long long, long long, long long, signed char *,
                          int *, signed char *, int *);
    RsFn fn = nullptr;
    switch (S) {
        case 1: fn = rho_slice_kernel<1>; break;
        case 2: fn = rho_slice_kernel<2>; break;
        case 3: fn = rho_slice_kernel<3>; break;
        case 4: fn = rho_slice_kernel<4>; break;
        case 5: fn = rho_slice_kernel<5>; break;
        case 6: fn = rho_slice_kernel<6>; break;
        case 7: fn = rho_slice_kernel<7>; break;
        case OZ_FMT_BF16X3: fn = rho_slice_kernel<OZ_FMT_BF16X3>; break;
        default: fn = rho_slice_kernel<OZ_FMT_TF32>; break;
    }
    const size_t smem = rs_smem_bytes();
    PHF_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // one cluster of two CTAs per (grid point, spin-block pair)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(4LL * bc), 1, 1);
    cfg.blockDim = dim3(RS_NT, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const long long npadK = oz_pad_cols(8LL * bc), npadP = oz_pad_cols(2LL * bc), kpad = oz_pad_k((long long)n * n);
    ProfScope prof(st, PROF_MEMORY);
    PHF_CUDA(cudaLaunchKernelEx(&cfg, fn, n, N, Xs, ld, bra, npadK, npadP, kpad, Ksl, eK, Psl, eP));
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

bool oz_format_ok(int S) { return (S >= 1 && S <= OZ_MAX_S) || oz_float(S); }

int oz_slots(int S) { return OZ_GP + oz_g1_width(S); }

size_t oz_slice_bytes(long long rows_pad, long long k, int S) {
    return (size_t)(OZ_GP + oz_g1_width(S)) * (size_t)rows_pad * (size_t)oz_pad_k(k);
}

// the unit ring, 2 OZ_UNITS + 2 mbarriers, the TMEM address and abort flag, the column scales, the
// four accumulator mbarriers of the floating-point formats
size_t oz_smem_bytes() { return (size_t)OZ_UNITS * OZ_UNIT + (2 * OZ_UNITS + 2) * 8 + 8 + OZ_BN * 8 + 4 * 8; }

// D (m x n, ldd) (+)= A_slices (S x mpad x kpad) * B_slices (S x npad x kpad)^T with exponents ea, eb.
// k is split into passes short enough for exact int32 group sums; later passes add into D.
int oz_gemm(int m, int n, int k, int S, const signed char *Asl, const int *ea, const signed char *Bsl, const int *eb,
            double *D, long long ldd, int accumulate, int *err, cudaStream_t st) {
    return oz_gemm_t(m, n, k, S, Asl, ea, Bsl, eb, D, ldd, accumulate, 0, err, st);
}

namespace {
using OzKernelFn = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap,
                            const CUtensorMap, OzArgs);

OzKernelFn oz_wide_kernel_for(int S) {
    switch (S) {
        case 1: return ozaki_i8_gemm_kernel<1, true>;
        case 2: return ozaki_i8_gemm_kernel<2, true>;
        case 3: return ozaki_i8_gemm_kernel<3, true>;
        case 4: return ozaki_i8_gemm_kernel<4, true>;
        case 5: return ozaki_i8_gemm_kernel<5, true>;
        default: return nullptr;
    }
}

OzKernelFn oz_kernel_for(int S) {
    switch (S) {
        case 1: return ozaki_i8_gemm_kernel<1>;
        case 2: return ozaki_i8_gemm_kernel<2>;
        case 3: return ozaki_i8_gemm_kernel<3>;
        case 4: return ozaki_i8_gemm_kernel<4>;
        case 5: return ozaki_i8_gemm_kernel<5>;
        case 6: return ozaki_i8_gemm_kernel<6>;
        case 7: return ozaki_i8_gemm_kernel<7>;
        case OZ_FMT_BF16X3: return ozaki_i8_gemm_kernel<OZ_FMT_BF16X3>;
        case OZ_FMT_TF32: return ozaki_i8_gemm_kernel<OZ_FMT_TF32>;
        default: return nullptr;
    }
}

// k-blocks one launch may accumulate: int8 group sums stay exact while S kpass 127^2 < 2^31; the
// FP32 accumulators of the floating-point formats take the whole k range.
long long oz_kb_pass(int S) {
    if (oz_float(S)) return 1LL << 40;
    const long long kb = (long long)(2147483647.0 / ((double)S * 127.0 * 127.0)) / OZ_BK;
    return kb < 1 ? 1 : kb;
}

__global__ void sum_splits_kernel(long long count, int nsplit, long long dz, const double *part, double *D) {
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < count; i += (long long)gridDim.x * 256)
    {
        double s = 0.0;
        for (int z = 0; z < nsplit; ++z) s += part[z * dz + i];
        D[i] = s;
    }
}
}  // namespace

// Split-k variant for small outputs with long k: nsplit CTAs per output tile write partial
// results to part (nsplit x (rows of D) x ldd), summed in split order into D.
int oz_gemm_splitk(int m, int n, int k, int S, const signed char *Asl, const int *ea, const signed char *Bsl,
                   const int *eb, double *D, long long ldd, int trans, int nsplit, double *part, int *err,
                   cudaStream_t st) {
    const long long kpad = oz_pad_k(k), kb_total = kpad / OZ_BK;
    if (nsplit <= 1 || kb_total > oz_kb_pass(S) || kb_total < 2 * nsplit)
        return oz_gemm_t(m, n, k, S, Asl, ea, Bsl, eb, D, ldd, 0, trans, err, st);
    CUtensorMap ta0, ta1, tb0, tb1, tbw;
    const long long mpad = oz_pad_rows(m), npad = oz_pad_cols(n);
    PHF_TRY(make_slice_maps(&ta0, &ta1, Asl, kpad, mpad, S, OZ_BM));
    PHF_TRY(make_slice_maps(&tb0, &tb1, Bsl, kpad, npad, S, oz_bn(S)));
    const bool wide = oz_wide_ok(S) && !g_narrow_mma;
    if (wide) PHF_TRY(make_wide_map(&tbw, Bsl, kpad, npad, oz_bn(S)));
    else tbw = tb0;
    const long long rows = trans ? n : m;
    const long long dz = rows * ldd;
    OzArgs a;
    a.m = m;
    a.n = n;
    a.kb0 = 0;
    a.kblocks = (int)((kb_total + nsplit - 1) / nsplit);
    a.kb_total = (int)kb_total;
    a.kseg = OZ_KSEG;
    a.gamma_n = 0;
    a.g_row0 = 0;
    a.gamma_mode = 0;
    a.g_pairs = nullptr;
    a.a_row0 = 0;
    a.b_row0 = 0;
    a.group_m = OZ_GROUP_M;
    a.S = S;
    a.ea = ea;
    a.eb = eb;
    a.D = part;
    a.ldd = ldd;
    a.accumulate = 0;
    a.trans = trans;
    a.dz = dz;
    a.err = err;
    const size_t smem = oz_smem_bytes();
    const OzKernelFn kern = wide ? oz_wide_kernel_for(S) : oz_kernel_for(S);
    if (!kern) {
        set_error(PHF_ERR_ARG, "oz_gemm: slices out of range");
        return PHF_ERR_ARG;
    }
    PHF_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((unsigned)(mpad / OZ_BM), (unsigned)((npad + oz_bn(S) - 1) / oz_bn(S)), (unsigned)nsplit);
    {
        ProfScope prof(st, PROF_JK);
        kern<<<grid, OZ_THREADS, smem, st>>>(ta0, tb0, ta1, tb1, tbw, a);
    }
    ++g_launches;
    PHF_CHECK_LAUNCH();
    {
        ProfScope prof(st, PROF_MEMORY);
        sum_splits_kernel<<<148 * 4, 256, 0, st>>>(dz, nsplit, dz, part, D);
    }
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

namespace {
int oz_gemm_launch(OzKernelFn kern, dim3 grid, size_t smem, const CUtensorMap &ta0, const CUtensorMap &tb0,
                   const CUtensorMap &ta1, const CUtensorMap &tb1, const CUtensorMap &tbw, int m, int n, int S,
                   const int *ea, const int *eb, double *D, long long ldd, int accumulate, int trans, int *err,
                   cudaStream_t st, int gamma_n, int g_row0, int a_row0, const OzEx &ex, long long kb_total,
                   long long kb_pass, int group_m);
}  // namespace

int oz_gemm_t(int m, int n, int k, int S, const signed char *Asl, const int *ea, const signed char *Bsl, const int *eb,
              double *D, long long ldd, int accumulate, int trans, int *err, cudaStream_t st, int gamma_n) {
    return oz_gemm_ex(m, n, k, S, Asl, oz_pad_rows(m), 0, ea, Bsl, eb, D, ldd, accumulate, trans, err, st, gamma_n, 0);
}

bool oz_fx_ok(int M, int S) {
    return M >= 1 && oz_format_ok(S) && !oz_float(S) && oz_npass(S) == 1 && oz_pad_k(2LL * M) / OZ_BK <= oz_kb_pass(S);
}

int oz_gemm_fx(int M, int N, int batch, int S, const signed char *Asl, long long a_rows_pad, const int *ea,
               const signed char *Bsl, long long b_rows_pad, const int *eb, zc *GX, long long ld, int *err,
               cudaStream_t st) {
    const long long kpad = oz_pad_k(2LL * M), kb_total = kpad / OZ_BK;
    if (M < 1 || N < 1 || batch < 1 || batch > 65535 || (long long)batch * N > a_rows_pad ||
        2LL * M * batch > b_rows_pad || !oz_format_ok(S) || oz_float(S) || oz_npass(S) != 1 ||
        kb_total > oz_kb_pass(S)) {
        set_error(PHF_ERR_ARG, "oz_gemm_fx: rows outside the slice buffers, too many points or an unsupported format");
        return PHF_ERR_ARG;
    }
    CUtensorMap ta0, ta1, tb0, tb1, tbw;
    PHF_TRY(make_slice_maps(&ta0, &ta1, Asl, kpad, a_rows_pad, S, OZ_BM));
    PHF_TRY(make_slice_maps(&tb0, &tb1, Bsl, kpad, b_rows_pad, S, oz_bn(S)));
    const bool wide = oz_wide_ok(S) && !g_narrow_mma;
    if (wide) PHF_TRY(make_wide_map(&tbw, Bsl, kpad, b_rows_pad, oz_bn(S)));
    else tbw = tb0;
    OzArgs a;
    a.m = N;  // rows j of one point (tiles reach into the next point's rows, which are not stored)
    a.n = 2 * M;
    a.kb0 = 0;
    a.kblocks = (int)kb_total;
    a.kb_total = (int)kb_total;
    a.kseg = OZ_KSEG;
    a.gamma_n = 0;
    a.g_row0 = 0;
    a.gamma_mode = 0;
    a.g_pairs = nullptr;
    a.a_row0 = 0;
    a.b_row0 = 0;
    a.group_m = OZ_GROUP_M;
    a.S = S;
    a.ea = ea;
    a.eb = eb;
    a.D = reinterpret_cast<double *>(GX);
    a.ldd = 2 * ld;     // doubles per row c of GX
    a.accumulate = 0;
    a.trans = 0;
    a.dz = 2LL * N;     // point w's columns start at GX + w N
    a.batch = 1;
    a.a_bs = N;
    a.b_bs = 2LL * M;
    a.ct = 1;
    a.err = err;
    const size_t smem = oz_smem_bytes();
    const OzKernelFn kern = wide ? oz_wide_kernel_for(S) : oz_kernel_for(S);
    if (!kern) {
        set_error(PHF_ERR_ARG, "oz_gemm_fx: slices out of range");
        return PHF_ERR_ARG;
    }
    PHF_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((unsigned)(oz_pad_rows(N) / OZ_BM), (unsigned)((2LL * M + oz_bn(S) - 1) / oz_bn(S)),
                    (unsigned)batch);
    {
        ProfScope prof(st, PROF_GEMM);
        kern<<<grid, OZ_THREADS, smem, st>>>(ta0, tb0, ta1, tb1, tbw, a);
    }
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int oz_gemm_ex(int m, int n, int k, int S, const signed char *Asl, long long a_rows_pad, int a_row0, const int *ea,
               const signed char *Bsl, const int *eb, double *D, long long ldd, int accumulate, int trans, int *err,
               cudaStream_t st, int gamma_n, int g_row0, const OzEx &ex) {
    if (gamma_n > 0) {
        const long long gn = gamma_n;
        const long long grows = ex.gamma_mode == 0 ? gn * gn : (ex.gamma_mode == 1 ? gn * (gn + 1) / 2 : gn * (gn - 1) / 2);
        if (ex.gamma_mode < 0 || ex.gamma_mode > 2 || (ex.gamma_mode != 0 && (!ex.g_pairs || gamma_n > 65535)) ||
            g_row0 < 0 || (long long)g_row0 + m > grows || n % 8 != 0 || trans) {
            set_error(PHF_ERR_ARG, "oz_gemm: the Gamma output needs rows within its exchange rows (n^2, or the "
                                   "n(n+1)/2 or n(n-1)/2 pairs with their table) and 8 columns per point");
            return PHF_ERR_ARG;
        }
    }
    if (a_row0 < 0 || (long long)a_row0 + m > a_rows_pad) {
        set_error(PHF_ERR_ARG, "oz_gemm: A row range outside its slice buffer");
        return PHF_ERR_ARG;
    }
    const long long b_rows_pad = ex.b_rows_pad > 0 ? ex.b_rows_pad : oz_pad_cols(n);
    // (the last column tile may reach past the buffer: TMA fills rows beyond the map's extent with zeros,
    // and the epilogue stores only columns < n)
    if (ex.b_row0 < 0 || (long long)ex.b_row0 + n > b_rows_pad || b_rows_pad % OZ_BN != 0) {
        set_error(PHF_ERR_ARG, "oz_gemm: B row range outside its slice buffer");
        return PHF_ERR_ARG;
    }
    if (!oz_format_ok(S)) {
        set_error(PHF_ERR_ARG, "oz_gemm: slices out of range");
        return PHF_ERR_ARG;
    }
    CUtensorMap ta0, ta1, tb0, tb1, tbw;
    const long long mpad = oz_pad_rows(m), npad = oz_pad_cols(n), kpad = oz_pad_k(k);
    PHF_TRY(make_slice_maps(&ta0, &ta1, Asl, kpad, a_rows_pad, S, OZ_BM));
    PHF_TRY(make_slice_maps(&tb0, &tb1, Bsl, kpad, b_rows_pad, S, oz_bn(S)));
    const bool wide = oz_wide_ok(S) && !g_narrow_mma;  // single-pass int8: the wide issue
    if (wide) PHF_TRY(make_wide_map(&tbw, Bsl, kpad, b_rows_pad, oz_bn(S)));
    else tbw = tb0;
    const long long kb_pass = oz_kb_pass(S);
    const long long kb_total = kpad / OZ_BK;
    const size_t smem = oz_smem_bytes();
    const OzKernelFn kern = wide ? oz_wide_kernel_for(S) : oz_kernel_for(S);
    if (!kern) {
        set_error(PHF_ERR_ARG, "oz_gemm: slices out of range");
        return PHF_ERR_ARG;
    }
    PHF_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((unsigned)(mpad / OZ_BM), (unsigned)((npad + oz_bn(S) - 1) / oz_bn(S)), 1);  // grouped raster
    const TuneKey key{1, m, n, k, (long long)S * 16 + ex.gamma_mode * 4 + (gamma_n > 0) * 2 + trans, accumulate};
    int group_m = tuned_choice(key);
    if (t_tune_record) {
        // the tuner repeats the launch; an accumulating launch then adds several times, which is harmless:
        // the tuning evaluation's outputs are discarded and recomputed by the evaluation that follows
        t_tune_record->push_back({key, {4, 8, 16}, [=](int g, cudaStream_t s) {
                                      return oz_gemm_launch(kern, grid, smem, ta0, tb0, ta1, tb1, tbw, m, n, S,
                                                            ea + a_row0, eb + ex.b_row0, D, ldd, accumulate, trans,
                                                            err, s, gamma_n, g_row0, a_row0, ex, kb_total, kb_pass, g);
                                  }});
    }
    if (group_m < 0) group_m = OZ_GROUP_M;
    return oz_gemm_launch(kern, grid, smem, ta0, tb0, ta1, tb1, tbw, m, n, S, ea + a_row0, eb + ex.b_row0, D, ldd,
                          accumulate, trans, err, st, gamma_n, g_row0, a_row0, ex, kb_total, kb_pass, group_m);
}

namespace {
// the k passes of one oz_gemm_ex call with the given raster group
int oz_gemm_launch(OzKernelFn kern, dim3 grid, size_t smem, const CUtensorMap &ta0, const CUtensorMap &tb0,
                   const CUtensorMap &ta1, const CUtensorMap &tb1, const CUtensorMap &tbw, int m, int n, int S,
                   const int *ea, const int *eb, double *D, long long ldd, int accumulate, int trans, int *err,
                   cudaStream_t st, int gamma_n, int g_row0, int a_row0, const OzEx &ex, long long kb_total,
                   long long kb_pass, int group_m) {
    for (long long kb0 = 0; kb0 < kb_total; kb0 += kb_pass) {
        OzArgs a;
        a.m = m;
        a.n = n;
        a.kb0 = (int)kb0;
        a.kblocks = (int)std::min(kb_pass, kb_total - kb0);
        a.S = S;
        a.ea = ea;
        a.eb = eb;
        a.D = D;
        a.ldd = ldd;
        a.accumulate = (kb0 > 0) ? 1 : accumulate;
        a.trans = trans;
        a.dz = 0;
        a.kb_total = a.kblocks;
        a.kseg = OZ_KSEG;
        a.gamma_n = gamma_n;
        a.g_row0 = g_row0;
        a.gamma_mode = ex.gamma_mode;
        a.g_pairs = ex.g_pairs;
        a.a_row0 = a_row0;
        a.b_row0 = ex.b_row0;
        a.group_m = group_m;
        a.err = err;
        {
            ProfScope prof(st, PROF_JK);
            kern<<<grid, OZ_THREADS, smem, st>>>(ta0, tb0, ta1, tb1, tbw, a);
        }
        ++g_launches;
        PHF_CHECK_LAUNCH();
    }
    return PHF_OK;
}
}  // namespace

}  // namespace phf

namespace phf {
namespace {
// Slices both operands into freshly allocated scratch, multiplies and frees (synchronous on st).
int tc_dgemm(const char *who, int m, int n, int k, int S, const double *dA, long long lda, const double *dBt,
             long long ldb, double *dD, long long ldd, cudaStream_t st) {
    const long long mp = oz_pad_rows(m), np = oz_pad_cols(n);
    signed char *As = nullptr, *Bs = nullptr;
    int *ea = nullptr, *eb = nullptr, *err = nullptr;
    int status = PHF_OK;
    auto al = [&](void **p, size_t bytes) {
        if (status != PHF_OK) return;
        if (cudaMalloc(p, bytes) != cudaSuccess) {
            cudaGetLastError();
            set_error(PHF_ERR_OOM, std::string(who) + ": cudaMalloc failed");
            status = PHF_ERR_OOM;
        }
    };
    const size_t asz = oz_slice_bytes(mp, k, S), bsz = oz_slice_bytes(np, k, S);
    al((void **)&As, asz);
    al((void **)&Bs, bsz);
    al((void **)&ea, mp * sizeof(int));
    al((void **)&eb, np * sizeof(int));
    al((void **)&err, sizeof(int));
    if (status == PHF_OK) {
        cudaMemsetAsync(As, 0, asz, st);
        cudaMemsetAsync(Bs, 0, bsz, st);
        cudaMemsetAsync(err, 0, sizeof(int), st);
        status = oz_slice_rows(m, k, dA, lda, S, mp, As, ea, st);
        if (status == PHF_OK) status = oz_slice_rows(n, k, dBt, ldb, S, np, Bs, eb, st);
        if (status == PHF_OK) status = oz_gemm(m, n, k, S, As, ea, Bs, eb, dD, ldd, 0, err, st);
        int herr = 0;
        if (status == PHF_OK) {
            cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st);
            if (cudaStreamSynchronize(st) != cudaSuccess) {
                set_error(PHF_ERR_CUDA, std::string(who) + ": stream synchronize failed");
                status = PHF_ERR_CUDA;
            } else if (herr) {
                set_error(PHF_ERR_CUDA, std::string(who) + ": pipeline wait timed out");
                status = PHF_ERR_CUDA;
            }
        }
    }
    cudaStreamSynchronize(st);
    cudaFree(As);
    cudaFree(Bs);
    cudaFree(ea);
    cudaFree(eb);
    cudaFree(err);
    return status;
}

bool gemm_args_ok(const char *who, int m, int n, int k, const double *dA, long long lda, const double *dBt,
                  long long ldb, double *dD, long long ldd) {
    if (m <= 0 || n <= 0 || k <= 0 || !dA || !dBt || !dD || lda < k || ldb < k || ldd < n) {
        set_error(PHF_ERR_ARG, std::string(who) + ": bad sizes or null pointer");
        return false;
    }
    return true;
}
}  // namespace
}  // namespace phf

extern "C" int phf_ozaki_dgemm(int m, int n, int k, int slices, const double *dA, long long lda, const double *dBt,
                               long long ldb, double *dD, long long ldd, void *stream) {
    using namespace phf;
    set_error(PHF_OK, "");
    if (!gemm_args_ok("phf_ozaki_dgemm", m, n, k, dA, lda, dBt, ldb, dD, ldd)) return PHF_ERR_ARG;
    if (slices < 1 || slices > OZ_MAX_S) {
        set_error(PHF_ERR_ARG, "phf_ozaki_dgemm: slices must be 1..7");
        return PHF_ERR_ARG;
    }
    return tc_dgemm("phf_ozaki_dgemm", m, n, k, slices, dA, lda, dBt, ldb, dD, ldd,
                    reinterpret_cast<cudaStream_t>(stream));
}

extern "C" int phf_tc_dgemm(int m, int n, int k, int precision, int slices, const double *dA, long long lda,
                            const double *dBt, long long ldb, double *dD, long long ldd, void *stream) {
    using namespace phf;
    set_error(PHF_OK, "");
    if (!gemm_args_ok("phf_tc_dgemm", m, n, k, dA, lda, dBt, ldb, dD, ldd)) return PHF_ERR_ARG;
    int S = 0;
    if (precision == PHF_PREC_OZAKI_I8) {
        S = slices == 0 ? 5 : slices;
        if (S < 1 || S > OZ_MAX_S) {
            set_error(PHF_ERR_ARG, "phf_tc_dgemm: slices must be 0..7");
            return PHF_ERR_ARG;
        }
    } else if (precision == PHF_PREC_BF16X3) {
        S = OZ_FMT_BF16X3;
    } else if (precision == PHF_PREC_TF32) {
        S = OZ_FMT_TF32;
    } else {
        set_error(PHF_ERR_ARG, "phf_tc_dgemm: precision must be PHF_PREC_OZAKI_I8, PHF_PREC_BF16X3 or PHF_PREC_TF32");
        return PHF_ERR_ARG;
    }
    return tc_dgemm("phf_tc_dgemm", m, n, k, S, dA, lda, dBt, ldb, dD, ldd, reinterpret_cast<cudaStream_t>(stream));
}
