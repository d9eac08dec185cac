// Batched FP64 complex inverse, determinant and log-determinant of the rotated overlaps
// S_w = bra^H R_w ket (N x N): one warp per grid point for N <= 32, one CTA with the matrix in registers
// for N <= 100, else one CTA of 32 x 32 threads with the matrix in shared memory.
//
// Replaces InvertC (ZGETRF + ZGETRI) and determinantC (ZGETRF) of PHF_fort/Wrappers.f90:195-336
// as called from RDM (PHF_fort/PHFTools.f90:259-260).  Algorithm: in-place Gauss-Jordan
// elimination with partial (row) pivoting -- the pivot is the first row of maximal |re| + |im|
// in the column, the choice LAPACK's izamax makes -- followed by the column interchanges
// in reverse order.  The pivots are those of LU with partial pivoting, so
//   det S = (-1)^{#interchanges} * prod(pivots),
//   log det S = sum log|pivot| + i (sum arg(pivot) + pi #interchanges).
// A zero pivot is reported as status 1 (the reference STOPs "Error in ZGetRF"); a
// non-finite entry as status 2.  Both are OR-ed into *flag and the outputs of that grid
// point are zeroed.
#include <type_traits>

#include "phf_common.cuh"

namespace phf {

namespace {

// x - c r, two fused multiply-adds a component
__device__ __forceinline__ zc submul(zc x, zc c, zc r) {
    return mkz(fma(c.y, r.y, fma(-c.x, r.x, x.x)), fma(-c.y, r.x, fma(-c.x, r.y, x.y)));
}

// det = (-1)^{#interchanges} prod(pivots) and log det from log|pivot| and arg(pivot) (plog), the product and the sums
// taken in pivot order by one thread
__device__ void write_det(int N, const zc *pivs, const zc *plog, int nswap, zc *det, zc *logdet) {
    zc d = mkz(1.0, 0.0);
    double logabs = 0.0, phase = 0.0;
    for (int k = 0; k < N; ++k) {
        d = d * pivs[k];
        logabs += plog[k].x;
        phase += plog[k].y;
    }
    if (nswap & 1) d = mkz(-d.x, -d.y);
    *det = d;
    const double pi = 3.14159265358979323846;
    double ph = fmod(phase + pi * (nswap & 1), 2.0 * pi);
    if (ph > pi) ph -= 2.0 * pi;
    if (ph <= -pi) ph += 2.0 * pi;
    *logdet = mkz(logabs, ph);
}

// One CTA of 32 x 32 threads per grid point (N > 100): thread (ty, tx) updates the elements of rows
// ty + 32 m and columns tx + 32 q, so a Gauss-Jordan step is four barriers -- the pivot search is one
// warp's shuffle arg-max -- and no index division.
constexpr int GJ_T = 32;  // threads per row and per column of the CTA

__global__ void __launch_bounds__(GJ_T *GJ_T) gj_inverse_kernel(int N, const zc *__restrict__ S, long long s_rs,
                                                                 long long s_bs, zc *__restrict__ Sinv, long long i_rs,
                                                                 long long i_bs, zc *__restrict__ det,
                                                                 zc *__restrict__ logdet, int *__restrict__ flag) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    zc *A = reinterpret_cast<zc *>(smem_raw);                 // N*N, row-major
    zc *rowk = A + (size_t)N * N;                             // N
    zc *colk = rowk + N;                                      // N
    int *perm = reinterpret_cast<int *>(colk + N);            // N
    __shared__ int s_bad, s_piv;
    __shared__ double s_pv;

    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * GJ_T + tx;
    constexpr int NTH = GJ_T * GJ_T;
    const long long b = blockIdx.x;
    const zc *Sb = S + b * s_bs;
    if (tid == 0) s_bad = 0;
    __syncthreads();
    for (int i = ty; i < N; i += GJ_T)
        for (int j = tx; j < N; j += GJ_T) {
            const zc v = Sb[(long long)i * s_rs + j];
            if (!isfinite(v.x) || !isfinite(v.y)) s_bad = 2;
            A[i * N + j] = v;
        }
    __syncthreads();

    double logabs = 0.0, phase = 0.0;  // kept by thread 0
    zc d = mkz(1.0, 0.0);
    int nswap = 0;
    for (int k = 0; k < N && s_bad == 0; ++k) {
        // pivot search (warp 0): first index of the maximal |re| + |im| in rows k..N-1 of column k
        if (ty == 0) {
            double best = -1.0;
            int bi = N;
            for (int i = k + tx; i < N; i += GJ_T) {
                const double a = abs1(A[i * N + k]);
                if (a > best) {
                    best = a;
                    bi = i;
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const double ov = __shfl_down_sync(0xffffffffu, best, off);
                const int oi = __shfl_down_sync(0xffffffffu, bi, off);
                if (ov > best || (ov == best && oi < bi)) {
                    best = ov;
                    bi = oi;
                }
            }
            if (tx == 0) {
                s_piv = bi;
                s_pv = best;
            }
        }
        __syncthreads();
        const int p = s_piv;
        const double pv = s_pv;
        if (!(pv > 0.0)) {  // exactly singular (or NaN pivot)
            if (tid == 0) s_bad = (pv == 0.0) ? 1 : 2;
            __syncthreads();
            break;
        }
        if (p != k && tid < N) {
            const zc t = A[k * N + tid];
            A[k * N + tid] = A[p * N + tid];
            A[p * N + tid] = t;
        }
        if (tid == 0) perm[k] = p;
        __syncthreads();
        const zc piv = A[k * N + k];
        if (tid == 0) {  // running determinant and log-determinant
            d = d * piv;
            logabs += log(hypot(piv.x, piv.y));
            phase += atan2(piv.y, piv.x);
            if (p != k) {
                d = mkz(-d.x, -d.y);
                ++nswap;
            }
        }
        const zc inv = divz(mkz(1.0, 0.0), piv);
        // scaled pivot row (with 1/piv in column k) and the saved column k
        if (tid < N) rowk[tid] = (tid == k) ? inv : A[k * N + tid] * inv;
        else if (tid < 2 * N && tid - N < NTH) colk[tid - N] = A[(tid - N) * N + k];
        __syncthreads();
        for (int i = ty; i < N; i += GJ_T) {
            const zc ci = colk[i];
            for (int j = tx; j < N; j += GJ_T) {
                const int e = i * N + j;
                if (i == k) {
                    A[e] = rowk[j];
                } else {
                    const zc a = (j == k) ? mkz(0.0, 0.0) : A[e];
                    A[e] = a - ci * rowk[j];
                }
            }
        }
        __syncthreads();
    }
    const int bad = s_bad;
    if (bad == 0) {
        // undo the row interchanges as column interchanges, in reverse order
        for (int k = N - 1; k >= 0; --k) {
            const int p = perm[k];
            if (p != k && tid < N) {
                const zc t = A[tid * N + k];
                A[tid * N + k] = A[tid * N + p];
                A[tid * N + p] = t;
            }
            __syncthreads();
        }
    }
    zc *Ib = Sinv + b * i_bs;
    for (int i = ty; i < N; i += GJ_T)
        for (int j = tx; j < N; j += GJ_T) Ib[(long long)i * i_rs + j] = bad ? mkz(0.0, 0.0) : A[i * N + j];
    if (tid == 0) {
        if (bad) {
            det[b] = mkz(0.0, 0.0);
            logdet[b] = mkz(-INFINITY, 0.0);
            atomicOr(flag, bad);
        } else {
            det[b] = d;
            const double pi = 3.14159265358979323846;
            double ph = fmod(phase + pi * (nswap & 1), 2.0 * pi);
            if (ph > pi) ph -= 2.0 * pi;
            if (ph <= -pi) ph += 2.0 * pi;
            logdet[b] = mkz(logabs, ph);
        }
    }
}

// 32 < N <= 100: the matrix held in registers.  A CTA of R x C threads (R = ceil(N / MR),
// C = ceil(N / MC)) per grid point; thread (r, c) keeps the MR x MC elements of rows r + R m and
// columns c + C q for the whole elimination, so a step reads and writes no matrix element through
// shared memory: only the pivot column (N values) and the scaled pivot row (N values) pass through
// it, with two barriers per step.
//
// Rows are not interchanged.  Step k takes as pivot the eligible row p (not pivoted before) of
// maximal |re| + |im| in column k; ties go to the row that the interchanging form would hold at the
// lowest position, so the pivot sequence and the interchange count are those of gj_inverse_kernel
// (every warp tracks the positions in its lanes' registers).  With p_k the pivot row of step k, the
// stored result E satisfies E[p_j][k] = inv(S)[j][p_k], which the write-out undoes: element (row, col)
// goes to inv(S)[step_of_row[row]][piv_row[col]].
// Bound: the serial chain of a step (publish, search, division, row, update).  The search is three warp
// reductions over the published column in every warp, the update is four multiply-adds an element without
// selects (the owners clear column k and row p beforehand), log and atan2 of the pivots are taken in parallel:
// 800 matrices of N = 100 in 1.40 ms against 2.40 with candidates through shared memory, a shuffle search and
// selects in the update; N = 64, 312 of them 0.22 against 0.38; N = 40, 56 of them 69 against 119 us.
constexpr int GR_NMAX = 128;  // bound of the shared pivot arrays

template <int MR, int MC, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    gj_inverse_reg_kernel(int N, int R, int C, const zc *__restrict__ S, long long s_rs, long long s_bs,
                          zc *__restrict__ Sinv, long long i_rs, long long i_bs, zc *__restrict__ det,
                          zc *__restrict__ logdet, int *__restrict__ flag) {
    // The thread grid covers rows 0 .. R MR - 1 and columns 0 .. C MC - 1; the entries outside the
    // N x N matrix are zero and stay zero (their column entries and pivot-row entries are zero in
    // every step before step N), are never taken as pivots before step N (value 0, and positions
    // above every row of the matrix), and are not written out.  So no update needs a bounds test.
    // colk alternates between two buffers by step parity: step k's column is still read in the update
    // phase after the second barrier, while the owners of column k + 1 may already publish theirs
    __shared__ zc rowk[GR_NMAX], colk2[2][GR_NMAX], pivs[GR_NMAX];
    __shared__ int step_of_row[GR_NMAX], piv_row[GR_NMAX];
    __shared__ int s_bad;

    const int tid = threadIdx.x, lane = tid & 31;
    const bool own = tid < R * C;
    const int r = own ? tid / C : 0, c = own ? tid - (tid / C) * C : 0;
    const long long b = blockIdx.x;
    const zc *Sb = S + b * s_bs;
    if (tid == 0) s_bad = 0;
    for (int i = tid; i < GR_NMAX; i += blockDim.x) colk2[0][i] = colk2[1][i] = mkz(0.0, 0.0);
    int pos[GR_NMAX / 32];  // position of row lane + 32 u, kept alike by every warp
#pragma unroll
    for (int u = 0; u < GR_NMAX / 32; ++u) pos[u] = lane + 32 * u;
    __syncthreads();
    zc a[MR][MC];
#pragma unroll
    for (int m = 0; m < MR; ++m)
#pragma unroll
        for (int q = 0; q < MC; ++q) {
            const int row = r + R * m, col = c + C * q;
            zc v = mkz(0.0, 0.0);
            if (own && row < N && col < N) {
                v = Sb[(long long)row * s_rs + col];
                if (!isfinite(v.x) || !isfinite(v.y)) s_bad = 2;
            }
            a[m][q] = v;
        }
    __syncthreads();

    int nswap = 0;  // kept by thread 0
    const int bad0 = s_bad;
    for (int k = 0; k < N && bad0 == 0; ++k) {
        zc *colk = colk2[k & 1];
        // (A) the owners of column k (slot q with c + C q == k: one q at most) publish it and clear their copy, so
        // that the update below is the same for every column
#pragma unroll
        for (int q = 0; q < MC; ++q)
            if (own && c + C * q == k) {
#pragma unroll
                for (int m = 0; m < MR; ++m) {
                    colk[r + R * m] = a[m][q];
                    a[m][q] = mkz(0.0, 0.0);
                }
            }
        __syncthreads();
        // (B) every warp searches the column: maximal value (a non-negative double orders like its bits), then
        // lowest position
        unsigned long long best = 0;
        unsigned at = ~0u;  // position and row of the lane's best candidate
#pragma unroll
        for (int u = 0; u < GR_NMAX / 32; ++u) {
            const double v = abs1(colk[lane + 32 * u]);
            const unsigned long long key = (unsigned long long)__double_as_longlong(v);
            const unsigned pr = (unsigned)pos[u] * GR_NMAX + lane + 32 * u;
            if (pos[u] >= k && lane + 32 * u < N && v == v && (at == ~0u || key > best || (key == best && pr < at))) {
                best = key;
                at = pr;
            }
        }
        const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32));
        const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32) == hi ? (unsigned)best : 0u);
        at = __reduce_min_sync(0xffffffffu, best == ((unsigned long long)hi << 32 | lo) ? at : ~0u);
        if ((hi | lo) == 0) {  // exactly singular (or only NaN pivots): every thread leaves at the same step
            if (tid == 0) s_bad = at == ~0u ? 2 : 1;
            break;
        }
        const int p = (int)(at % GR_NMAX), pp = (int)(at / GR_NMAX);
#pragma unroll
        for (int u = 0; u < GR_NMAX / 32; ++u) {
            if (pos[u] == k) pos[u] = pp;
            if (lane + 32 * u == p) pos[u] = k;
        }
        if (own && r == p % R) {  // the owners of row p write the scaled pivot row and clear their copy
            const zc inv = divz(mkz(1.0, 0.0), colk[p]);
            const int mp = p / R;
#pragma unroll
            for (int m = 0; m < MR; ++m)
                if (m == mp) {
#pragma unroll
                    for (int q = 0; q < MC; ++q) {
                        const int col = c + C * q;
                        rowk[col] = (col == k) ? inv : a[m][q] * inv;
                        a[m][q] = mkz(0.0, 0.0);
                    }
                }
        }
        if (tid == 0) {  // pivots (det and log det are formed from them at the end)
            pivs[k] = colk[p];
            nswap += pp != k;
            step_of_row[p] = k;
            piv_row[k] = p;
        }
        __syncthreads();
        // (C) rank-1 update of the register-resident elements; the cleared pivot row takes the factor -1
        if (own) {
            zc rk[MC];
#pragma unroll
            for (int q = 0; q < MC; ++q) rk[q] = rowk[c + C * q];
#pragma unroll
            for (int m = 0; m < MR; ++m) {
                const zc ci = r + R * m == p ? mkz(-1.0, 0.0) : colk[r + R * m];
#pragma unroll
                for (int q = 0; q < MC; ++q) a[m][q] = submul(a[m][q], ci, rk[q]);
            }
        }
    }
    __syncthreads();
    const int bad = s_bad;
    zc *Ib = Sinv + b * i_bs;
    if (own) {
#pragma unroll
        for (int m = 0; m < MR; ++m)
#pragma unroll
            for (int q = 0; q < MC; ++q) {
                const int row = r + R * m, col = c + C * q;
                if (row < N && col < N) {
                    if (bad)
                        Ib[(long long)row * i_rs + col] = mkz(0.0, 0.0);
                    else
                        Ib[(long long)step_of_row[row] * i_rs + piv_row[col]] = a[m][q];
                }
            }
    }
    if (!bad && tid < N) rowk[tid] = mkz(log(hypot(pivs[tid].x, pivs[tid].y)), atan2(pivs[tid].y, pivs[tid].x));
    __syncthreads();
    if (tid == 0) {
        if (bad) {
            det[b] = mkz(0.0, 0.0);
            logdet[b] = mkz(-INFINITY, 0.0);
            atomicOr(flag, bad);
        } else {
            write_det(N, pivs, rowk, nswap, det + b, logdet + b);
        }
    }
}

// N <= 32: one warp per matrix, lane j holding column j in registers, padded to NB rows (a multiple of four).  The
// same Gauss-Jordan steps with the rows rotated by one register per step: step k's row is always register 0, the
// rows below it follow, the finished rows come last, so every register index is a constant of the unrolled code.
// Lane k passes its column through shared memory; lane i takes candidate i of the pivot search, an arg-max by
// three warp reductions (a non-negative double orders like its bits).  The column interchanges at the end are
// a permutation of the lanes' store addresses.
// Bound: the serial chain of a step (search, division, update).  Measured with the launch and status read: 800
// matrices of N = 32 in 82 us against 134 with the matrix in shared memory, a shuffle search and log and atan2
// by one lane (1650 warp instructions a step); 260 of N = 24 in 47 against 84; 112 of N = 10 in 33 against 46.
constexpr int WI_WARPS = 4;  // matrices per CTA

template <int NB>
__global__ void __launch_bounds__(WI_WARPS * 32) gj_inverse_warp_kernel(
    int N, int batch, const zc *__restrict__ S, long long s_rs, long long s_bs, zc *__restrict__ Sinv, long long i_rs,
    long long i_bs, zc *__restrict__ det, zc *__restrict__ logdet, int *__restrict__ flag) {
    __shared__ zc s_col[WI_WARPS][NB], s_piv[WI_WARPS][NB], s_log[WI_WARPS][NB];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long b = (long long)blockIdx.x * WI_WARPS + warp;
    if (b >= batch) return;  // the whole warp leaves; nothing below synchronises beyond the warp
    zc *colk = s_col[warp], *pivs = s_piv[warp], *plog = s_log[warp];
    const unsigned full = 0xffffffffu;
    const bool own = lane < N;

    const zc *Sb = S + b * s_bs;
    int bad = 0;
    zc a[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        a[i] = mkz(0.0, 0.0);
        if (own && i < N) a[i] = Sb[(long long)i * s_rs + lane];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i)
        if (!isfinite(a[i].x) || !isfinite(a[i].y)) bad = 2;
    bad = __reduce_max_sync(full, bad);

    int nswap = 0, my_perm = 0;  // lane k keeps the row interchanged with row k
    for (int k = 0; k < N && bad == 0; ++k) {
        if (lane == k) {
#pragma unroll
            for (int i = 0; i < NB; ++i) colk[i] = a[i];
#pragma unroll
            for (int i = 0; i < NB; ++i) a[i] = mkz(0.0, 0.0);
        }
        __syncwarp();
        unsigned long long key = 0;
        bool cand = false;  // NaN never becomes a candidate
        if (lane < N - k) {
            const double v = abs1(colk[lane]);
            cand = v == v;
            if (cand) key = (unsigned long long)__double_as_longlong(v);
        }
        const unsigned hi = __reduce_max_sync(full, (unsigned)(key >> 32));
        const unsigned lo = __reduce_max_sync(full, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
        const unsigned who = __ballot_sync(full, cand && key == ((unsigned long long)hi << 32 | lo));
        if ((hi | lo) == 0) {  // exactly singular (or only NaN pivots)
            bad = who ? 1 : 2;
            break;
        }
        const int p = __ffs(who) - 1;
        const zc piv = colk[p];
        if (lane == k) my_perm = k + p;
        if (p != 0) {
            ++nswap;
            const zc c0 = colk[0], r0 = a[0];
            __syncwarp();
            if (lane == 0) colk[p] = c0;
#pragma unroll
            for (int i = 1; i < NB; ++i) {
                const bool h = i == p;
                const zc t = a[i];
                a[i] = mkz(h ? r0.x : t.x, h ? r0.y : t.y);
                a[0] = mkz(h ? t.x : a[0].x, h ? t.y : a[0].y);
            }
            __syncwarp();
        }
        if (lane == 0) pivs[k] = piv;
        const zc inv = divz(mkz(1.0, 0.0), piv);
        const zc rk = lane == k ? inv : a[0] * inv;
#pragma unroll
        for (int i = 1; i < NB; ++i) {
            if (i % 8 == 0) __syncwarp();  // bounds how far ahead the column is loaded (registers)
            a[i - 1] = submul(a[i], colk[i], rk);
        }
        a[NB - 1] = rk;
        __syncwarp();
    }
    // undo the row interchanges as column interchanges, in reverse order: where the lane's column ends up
    int col = lane;
    for (int k = N - 1; k >= 0; --k) {
        const int p = __shfl_sync(full, my_perm, k);
        col = col == k ? p : (col == p ? k : col);
    }
    zc *Ib = Sinv + b * i_bs;
    if (bad) {
        for (int i = 0; i < N; ++i)
            if (own) Ib[(long long)i * i_rs + lane] = mkz(0.0, 0.0);
    } else {
#pragma unroll
        for (int i = 0; i < NB; ++i)  // register i holds row i - (NB - N)
            if (own && i >= NB - N) Ib[(long long)(i - (NB - N)) * i_rs + col] = a[i];
        if (own) plog[lane] = mkz(log(hypot(pivs[lane].x, pivs[lane].y)), atan2(pivs[lane].y, pivs[lane].x));
    }
    __syncwarp();
    if (lane == 0) {
        if (bad) {
            det[b] = mkz(0.0, 0.0);
            logdet[b] = mkz(-INFINITY, 0.0);
            atomicOr(flag, bad);
        } else {
            write_det(N, pivs, plog, nswap, det + b, logdet + b);
        }
    }
}

}  // namespace

size_t overlap_inverse_smem(int N) { return (size_t)N * N * sizeof(zc) + 2 * (size_t)N * sizeof(zc) + N * sizeof(int); }

int overlap_inverse(int N, int batch, const zc *S, long long s_rs, long long s_bs, zc *Sinv, long long i_rs,
                    long long i_bs, zc *det, zc *logdet, int *flag, cudaStream_t st) {
    if (N <= 32) {
        ProfScope prof(st, PROF_INVERSE);
        const unsigned grid = (unsigned)((batch + WI_WARPS - 1) / WI_WARPS);
        const auto launch = [&](auto nb) {
            gj_inverse_warp_kernel<nb.value><<<grid, WI_WARPS * 32, 0, st>>>(N, batch, S, s_rs, s_bs, Sinv, i_rs, i_bs,
                                                                            det, logdet, flag);
        };
        switch ((N + 3) / 4) {
            case 1: launch(std::integral_constant<int, 4>{}); break;
            case 2: launch(std::integral_constant<int, 8>{}); break;
            case 3: launch(std::integral_constant<int, 12>{}); break;
            case 4: launch(std::integral_constant<int, 16>{}); break;
            case 5: launch(std::integral_constant<int, 20>{}); break;
            case 6: launch(std::integral_constant<int, 24>{}); break;
            case 7: launch(std::integral_constant<int, 28>{}); break;
            default: launch(std::integral_constant<int, 32>{}); break;
        }
        ++g_launches;
        PHF_CHECK_LAUNCH();
        return PHF_OK;
    }
    if (N <= 100) {
        // register-resident elimination: MR x MC elements per thread, R x C <= 512 threads, R <= 32
        const bool small = N <= 64;
        const int MR = small ? 4 : 5, MC = 4;
        const int R = (N + MR - 1) / MR, C = (N + MC - 1) / MC;
        const unsigned threads = (unsigned)((R * C + 31) / 32 * 32);
        ProfScope prof(st, PROF_INVERSE);
        if (small)
            gj_inverse_reg_kernel<4, 4, 256, 2><<<batch, threads, 0, st>>>(N, R, C, S, s_rs, s_bs, Sinv, i_rs, i_bs,
                                                                            det, logdet, flag);
        else
            gj_inverse_reg_kernel<5, 4, 512, 1><<<batch, threads, 0, st>>>(N, R, C, S, s_rs, s_bs, Sinv, i_rs, i_bs,
                                                                            det, logdet, flag);
        ++g_launches;
        PHF_CHECK_LAUNCH();
        return PHF_OK;
    }
    size_t smem = overlap_inverse_smem(N);
    PHF_CUDA(cudaFuncSetAttribute(gj_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    ProfScope prof(st, PROF_INVERSE);
    gj_inverse_kernel<<<batch, dim3(GJ_T, GJ_T), smem, st>>>(N, S, s_rs, s_bs, Sinv, i_rs, i_bs, det, logdet, flag);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

}  // namespace phf

extern "C" int phf_overlap_inverse(int n, int batch, const double *dS, double *dSinv, double *ddet, double *dlogdet,
                                   int *dflag, void *stream) {
    using namespace phf;
    set_error(PHF_OK, "");
    if (n <= 0 || batch <= 0 || !dS || !dSinv || !ddet || !dlogdet || !dflag) {
        set_error(PHF_ERR_ARG, "phf_overlap_inverse: bad sizes or null pointer");
        return PHF_ERR_ARG;
    }
    if (n > 112) {  // the shared-memory form holds n^2 complex per CTA
        set_error(PHF_ERR_UNSUPPORTED, "phf_overlap_inverse: n above the inverse's limit of 112");
        return PHF_ERR_UNSUPPORTED;
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const long long nn = (long long)n * n;
    PHF_CUDA(cudaMemsetAsync(dflag, 0, sizeof(int), st));
    PHF_TRY(overlap_inverse(n, batch, reinterpret_cast<const zc *>(dS), n, nn, reinterpret_cast<zc *>(dSinv), n, nn,
                            reinterpret_cast<zc *>(ddet), reinterpret_cast<zc *>(dlogdet), dflag, st));
    int flag = 0;
    PHF_CUDA(cudaMemcpyAsync(&flag, dflag, sizeof(int), cudaMemcpyDeviceToHost, st));
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        set_error(PHF_ERR_CUDA, "stream synchronize failed");
        return PHF_ERR_CUDA;
    }
    if (flag & 1) {
        set_error(PHF_ERR_SINGULAR, "phf_overlap_inverse: an exactly singular matrix");
        return PHF_ERR_SINGULAR;
    }
    if (flag & 2) {
        set_error(PHF_ERR_NONFINITE, "phf_overlap_inverse: a non-finite entry");
        return PHF_ERR_NONFINITE;
    }
    return PHF_OK;
}
