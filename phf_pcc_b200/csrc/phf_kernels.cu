// Memory-bound kernels of the projected-HF pipeline: traces of the Cholesky-projected
// overlaps, the energy/gradient epilogue, the weighted (Wigner x point-group) accumulation
// over grid points, and layout transforms.  All reductions run in a fixed order, so two
// runs give bit-identical results.
#include "phf_common.cuh"

namespace phf {

namespace {

constexpr int NT = 256;

// block-wide complex sum with a fixed tree (deterministic for a fixed block size)
__device__ zc block_sum(zc v, zc *sh) {
    const int tid = threadIdx.x;
    sh[tid] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (tid < s) sh[tid] = sh[tid] + sh[tid + s];
        __syncthreads();
    }
    zc r = sh[0];
    __syncthreads();
    return r;
}

// For each Cholesky vector L and grid point w, with T_Lw = bra^H B_L X_w (N x N):
//   d = tr T, e2part[w*L_tot + L] = d^2 - tr(T T), and T <- d I - T  (in place).
// T_Lw is the block at rows L*N, columns w*N of a (L_tot*N) x ldT matrix.
__global__ void __launch_bounds__(NT) tprime_kernel(int Ltot, int N, zc *T, long long ldT, zc *e2part) {
    __shared__ zc sh[NT];
    const long long L = blockIdx.x, w = blockIdx.y;
    zc *base = T + L * N * ldT + w * N;
    zc dd = mkz(0, 0), t2 = mkz(0, 0);
    for (int j = threadIdx.x; j < N; j += NT) dd = dd + base[(long long)j * ldT + j];
    for (int e = threadIdx.x; e < N * N; e += NT) {
        int j = e / N, jp = e - j * N;
        t2 = t2 + base[(long long)j * ldT + jp] * base[(long long)jp * ldT + j];
    }
    dd = block_sum(dd, sh);
    t2 = block_sum(t2, sh);
    if (threadIdx.x == 0) e2part[w * Ltot + L] = dd * dd - t2;
    for (int e = threadIdx.x; e < N * N; e += NT) {
        int j = e / N, jp = e - j * N;
        long long o = (long long)j * ldT + jp;
        zc t = base[o];
        base[o] = (j == jp) ? (dd - t) : mkz(-t.x, -t.y);
    }
}

// out[r] = scale * sum_c in[r * ncols + c]
__global__ void __launch_bounds__(NT) rowsum_kernel(int ncols, const zc *in, zc *out, double scale) {
    __shared__ zc sh[NT];
    const long long r = blockIdx.x;
    zc s = mkz(0, 0);
    for (int c = threadIdx.x; c < ncols; c += NT) s = s + in[r * ncols + c];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) out[r] = scale * s;
}

// out[w] = scale * sum_{r,j} conj(C[r*N + j]) * X[r*ldX + w*N + j]   (tr(C^H X_w)), minus
// sub_scale * sub[w] when `sub` is given
__global__ void __launch_bounds__(NT) trace_conj_kernel(int M, int N, const zc *C, zc *X, long long ldX, zc *out,
                                                        double scale, const zc *add, const zc *sub, double sub_scale) {
    __shared__ zc sh[NT];
    const long long w = blockIdx.x;
    zc s = mkz(0, 0);
    for (int e0 = threadIdx.x; e0 < M * N; e0 += 4 * NT) {  // four loads in flight, summed in order
        zc x[4], c[4];
        long long o[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = e0 + u * NT;
            if (e < M * N) {
                const int r = e / N, j = e - r * N;
                o[u] = (long long)r * ldX + w * N + j;
                x[u] = X[o[u]];
                c[u] = C[e];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (e0 + u * NT < M * N) {
                s = s + conjz(c[u]) * x[u];
                if (add) X[o[u]] = x[u] + add[o[u]];  // X <- X + add once the trace has read X
            }
    }
    s = block_sum(s, sh);
    if (threadIdx.x == 0) out[w] = sub ? scale * s - sub_scale * sub[w] : scale * s;
}

// Neumaier compensated add of a complex term into (s, c)
__device__ __forceinline__ void neumaier(double &s, double &c, double x) {
    double t = s + x;
    if (fabs(s) >= fabs(x)) c += (s - t) + x;
    else c += (x - t) + s;
    s = t;
}

// Weighted accumulation over a chunk of grid points (PHFTools.f90:137-166) with the energy/gradient epilogue
// (Gradient, PHFTools.f90:291-308, in the rank-N form) applied on the way.  With h_w = e1_w + e2_w, N_w = det S_w
// and c_w = Wt[s, w0 + w] N_w (both conjugated for the ket side, which has no h: e1 null):
//   accG[a] += sum_w c_w (G_w + h_w R_w),  accR[a] += sum_w c_w R_w,  accHS[a] += sum_w c_w (h_w, 1)
// with a = slotmap[s]; G holds HX + GammaX - X W_w, R holds X_w.
// Two stages with a fixed partition, so the result does not depend on scheduling:
//   stage 1: thread (element, group q) sums the points [q*ACC_GROUP, (q+1)*ACC_GROUP) in order
//            with Neumaier compensation into part[q] (sum, compensation); the two scalars are element MN;
//   stage 2: ACC_LANES lanes an element add every ACC_LANES-th group, then each other's sums in a fixed tree, and one
//            adds the result into the running (acc, comp); a thread for all groups was a chain of 100 loads and
//            compensated additions for 3200 points (68 against 18 us).
// Bound: G and R read once; at small sizes the serial chain of the 32 points, so their loads go four ahead (eight
// take 10 against 11.5 us at M = 40, but 85 against 75 for 3200 points at M = 128) and the group's factors come
// from shared memory (M = 40 to 96: 12 us against 34 as one load after another, after 4 to 9 us of a separate
// epilogue that wrote G and R again).
constexpr int ACC_GROUP = 32, ACC_NT = 128, ACC_LANES = 8;

struct AccPart {
    double gs_r, gs_i, gc_r, gc_i, rs_r, rs_i, rc_r, rc_i;
};

__global__ void __launch_bounds__(ACC_NT) accumulate_partial_kernel(int nslot, int M, int N, int b, const zc *Wt,
                                                                    long long nomega, long long w0,
                                                                    const zc *__restrict__ G, const zc *__restrict__ R,
                                                                    long long ldX, const zc *det, const zc *e1,
                                                                    const zc *e2, AccPart *part, int conj_w) {
    __shared__ zc s_c[ACC_GROUP], s_h[ACC_GROUP];
    const long long MN = (long long)M * N;
    const long long e = blockIdx.x * (long long)ACC_NT + threadIdx.x;
    const int q = blockIdx.y, wa = q * ACC_GROUP, nw = min(b - wa, ACC_GROUP);
    const long long r = e / N, j = e - r * N;
    const zc *g = G + r * ldX + (long long)wa * N + j, *x = R + r * ldX + (long long)wa * N + j;
    for (int s = blockIdx.z; s < nslot; s += gridDim.z) {
        __syncthreads();
        if (threadIdx.x < nw) {
            const int w = wa + threadIdx.x;
            const zc c = Wt[(long long)s * nomega + w0 + w] * det[w];
            s_c[threadIdx.x] = conj_w ? conjz(c) : c;
            s_h[threadIdx.x] = e1 ? e1[w] + e2[w] : mkz(0.0, 0.0);
        }
        __syncthreads();
        if (e > MN) continue;
        AccPart P = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int w4 = 0; w4 < nw; w4 += 4) {
            zc gv[4], xv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                gv[u] = mkz(0.0, 0.0);
                xv[u] = mkz(1.0, 0.0);  // element MN: c h and c
                if (e < MN && w4 + u < nw) {
                    gv[u] = g[(long long)(w4 + u) * N];
                    xv[u] = x[(long long)(w4 + u) * N];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (w4 + u < nw) {
                    const zc c = s_c[w4 + u];
                    const zc tg = c * (e1 ? gv[u] + s_h[w4 + u] * xv[u] : gv[u]), tr = c * xv[u];
                    neumaier(P.gs_r, P.gc_r, tg.x);
                    neumaier(P.gs_i, P.gc_i, tg.y);
                    neumaier(P.rs_r, P.rc_r, tr.x);
                    neumaier(P.rs_i, P.rc_i, tr.y);
                }
        }
        part[((long long)q * nslot + s) * (MN + 1) + e] = P;
    }
}

__device__ __forceinline__ void add_part(double &s, double &c, double ps, double pc) {
    neumaier(s, c, ps);
    c += pc;
}

__global__ void __launch_bounds__(ACC_NT) accumulate_final_kernel(int nslot, int M, int N, const int *slotmap,
                                                                  int ngroups, const AccPart *__restrict__ part,
                                                                  zc *accG, zc *compG, zc *accR, zc *compR, zc *accHS,
                                                                  zc *compHS) {
    const long long MN = (long long)M * N, nel = (long long)nslot * (MN + 1);
    const int lane = threadIdx.x % ACC_LANES;
    for (long long e0 = blockIdx.x * (long long)(ACC_NT / ACC_LANES); e0 < nel;
         e0 += (long long)gridDim.x * (ACC_NT / ACC_LANES)) {
        const long long e = e0 + threadIdx.x / ACC_LANES;
        AccPart A = {0, 0, 0, 0, 0, 0, 0, 0};
        const auto add = [&](const AccPart &P) {
            add_part(A.gs_r, A.gc_r, P.gs_r, P.gc_r);
            add_part(A.gs_i, A.gc_i, P.gs_i, P.gc_i);
            add_part(A.rs_r, A.rc_r, P.rs_r, P.rc_r);
            add_part(A.rs_i, A.rc_i, P.rs_i, P.rc_i);
        };
        if (e < nel) {
#pragma unroll 2
            for (int q = lane; q < ngroups; q += ACC_LANES) add(part[(long long)q * nel + e]);
        }
#pragma unroll
        for (int off = ACC_LANES / 2; off > 0; off >>= 1) {
            AccPart P;
            P.gs_r = __shfl_down_sync(0xffffffffu, A.gs_r, off, ACC_LANES);
            P.gs_i = __shfl_down_sync(0xffffffffu, A.gs_i, off, ACC_LANES);
            P.gc_r = __shfl_down_sync(0xffffffffu, A.gc_r, off, ACC_LANES);
            P.gc_i = __shfl_down_sync(0xffffffffu, A.gc_i, off, ACC_LANES);
            P.rs_r = __shfl_down_sync(0xffffffffu, A.rs_r, off, ACC_LANES);
            P.rs_i = __shfl_down_sync(0xffffffffu, A.rs_i, off, ACC_LANES);
            P.rc_r = __shfl_down_sync(0xffffffffu, A.rc_r, off, ACC_LANES);
            P.rc_i = __shfl_down_sync(0xffffffffu, A.rc_i, off, ACC_LANES);
            add(P);
        }
        if (lane != 0 || e >= nel) continue;
        const int s = (int)(e / (MN + 1));
        const long long rj = e - (long long)s * (MN + 1);
        const bool scalars = rj == MN;
        if (scalars && !accHS) continue;
        const long long a = scalars ? 2LL * slotmap[s] : (long long)slotmap[s] * MN + rj;
        zc *pg = scalars ? accHS : accG, *pgc = scalars ? compHS : compG;
        zc *pr = scalars ? accHS + 1 : accR, *prc = scalars ? compHS + 1 : compR;
        double gs_r = pg[a].x, gs_i = pg[a].y, gc_r = pgc[a].x, gc_i = pgc[a].y;
        double rs_r = pr[a].x, rs_i = pr[a].y, rc_r = prc[a].x, rc_i = prc[a].y;
        add_part(gs_r, gc_r, A.gs_r, A.gc_r);
        add_part(gs_i, gc_i, A.gs_i, A.gc_i);
        add_part(rs_r, rc_r, A.rs_r, A.rc_r);
        add_part(rs_i, rc_i, A.rs_i, A.rc_i);
        pg[a] = mkz(gs_r, gs_i);
        pgc[a] = mkz(gc_r, gc_i);
        pr[a] = mkz(rs_r, rs_i);
        prc[a] = mkz(rc_r, rc_i);
    }
}

// out[i] = v through two 8-byte stores: the caller's buffers are aligned to a double only
__device__ __forceinline__ void store8(zc *out, long long i, zc v) {
    double *d = reinterpret_cast<double *>(out) + 2 * i;
    d[0] = v.x;
    d[1] = v.y;
}

// The accumulated sums with their compensations: out[slot][r] = acc[slot][src(r)] + comp[slot][src(r)], averaged with
// the ket side's sums where given; src(r) = rowmap[r] (null: r).  Block rows 0 .. 2 nslot - 1 are the gradient and
// density matrices, one more holds the scalars.
__global__ void fold_out_kernel(int nslot, int M, int N, const int *rowmap, FoldSums S, zc *outG, zc *outR,
                                zc *outHS) {
    const long long MN = (long long)M * N;
    for (long long y = blockIdx.y; y < 2LL * nslot + 1; y += gridDim.y) {
        if (y == 2LL * nslot) {
            for (long long i = blockIdx.x * (long long)NT + threadIdx.x; i < 2LL * nslot; i += (long long)gridDim.x * NT)
                store8(outHS, i, S.HS[i] + S.cHS[i]);
            continue;
        }
        const long long slot = y >> 1;
        const bool dens = y & 1;
        const zc *acc = dens ? S.R : S.G, *comp = dens ? S.cR : S.cG;
        const zc *ka = dens ? S.KR : S.KG, *kc = dens ? S.cKR : S.cKG;
        zc *out = (dens ? outR : outG) + slot * MN;
        for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < MN; e += (long long)gridDim.x * NT) {
            const long long r = e / N, j = e - r * N;
            const long long o = slot * MN + (rowmap ? (long long)rowmap[r] * N + j : e);
            zc v = acc[o] + comp[o];
            if (ka) v = 0.5 * (v + (ka[o] + kc[o]));
            store8(out, e, v);
        }
    }
}

// H2r[(i M + k) M^2 + (l M + j)] = H2(i, j, k, l) with H2 in Fortran order (MakeGamma operand
// reshaped to an M^2 x M^2 matrix acting on vec(rho) with rho(l, j) at l M + j)
__global__ void permute_h2_kernel(int M, const zc *H2, zc *H2r) {
    const long long M2 = (long long)M * M, tot = M2 * M2;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < tot; e += (long long)gridDim.x * NT) {
        long long row = e / M2, col = e - row * M2;
        long long i = row / M, k = row - i * M, l = col / M, j = col - l * M;
        H2r[e] = H2[i + M * (j + M * (k + M * l))];
    }
}

// out[r] = in[rowmap[r]] (M x N), into two buffers
__global__ void permute_rows_kernel(int M, int N, const int *rowmap, const zc *in, zc *out, zc *out2) {
    const long long tot = (long long)M * N;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < tot; e += (long long)gridDim.x * NT) {
        const long long r = e / N, j = e - r * N;
        out[e] = out2[e] = in[(long long)rowmap[r] * N + j];
    }
}

// P[(p n + q) ldp + w] = rho_w[2p][2q] + rho_w[2p+1][2q+1]  (spin-summed density for J)
__global__ void gather_p_kernel(int n, int b, const zc *rho, zc *P, long long ldp) {
    const int M = 2 * n;
    const long long tot = (long long)n * n * b;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < tot; e += (long long)gridDim.x * NT) {
        long long pq = e / b, w = e - pq * b;
        int p = (int)(pq / n), q = (int)(pq - (long long)p * n);
        const zc *R = rho + w * (long long)M * M;
        P[pq * ldp + w] = R[(long long)(2 * p) * M + 2 * q] + R[(long long)(2 * p + 1) * M + 2 * q + 1];
    }
}

// Kin[(l n + j) ldk + 4 w + 2 sigma + tau] = rho_w[2l + sigma][2j + tau]  (exchange operand)
__global__ void gather_kin_kernel(int n, int b, const zc *rho, zc *Kin, long long ldk) {
    const int M = 2 * n;
    const long long tot = (long long)n * n * b * 4;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < tot; e += (long long)gridDim.x * NT) {
        long long lj = e / (4LL * b), c = e - lj * 4LL * b;
        long long w = c >> 2;
        int sg = (int)((c >> 1) & 1), tu = (int)(c & 1);
        int l = (int)(lj / n), j = (int)(lj - (long long)l * n);
        Kin[lj * ldk + c] = rho[w * (long long)M * M + (long long)(2 * l + sg) * M + 2 * j + tu];
    }
}

// Gamma_w[2i + sigma][2k + tau] = delta_{sigma tau} J[(i, k), w] - K_{sigma tau}[(i, k), w]
// J: complex J[(i n + k) ldj + w], or real/imaginary pairs with element (ik, c) of Jr at
//    Jr[ik jrs + c jcs], c = 2 w + part;
// K: complex Kc[(i n + k) ldk + 4 w + st], or pairs with element (ik, c) of Kr at Kr[ik krs + c kcs],
//    c = 2 (4 w + st) + part.  ksym (complex Kc only): K from its symmetric-form parts, KS of the pair
//    (min(i, k), max(i, k)) at row pair_le and KA at row n(n + 1)/2 + pair_lt (row order of the pairs),
//    K[i][k] = KS + KA for i < k, KS - KA for i > k, KS for i = k.  ksym 2: J too at pair rows, as
//    sum_L B_L[i][k] (2 - delta_ik) d_L (so J = J[pair] / 2 off the diagonal).
__global__ void assemble_gamma_kernel(int n, int b, const zc *J, long long ldj, const double *Jr, long long jrs,
                                      long long jcs, const zc *Kc, long long ldk, const double *Kr, long long krs,
                                      long long kcs, zc *Gam, int ksym, const double *h) {
    const int M = 2 * n;
    const long long tot = (long long)M * M * b;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < tot; e += (long long)gridDim.x * NT) {
        long long w = e / ((long long)M * M), rc = e - w * (long long)M * M;
        int r = (int)(rc / M), c = (int)(rc - (long long)r * M);
        int i = r >> 1, sg = r & 1, k = c >> 1, tu = c & 1;
        long long ik = (long long)i * n + k;
        int st = sg * 2 + tu;
        zc kv;
        if (Kc && ksym) {
            const long long lo = i < k ? i : k, hi = i < k ? k : i, nn = n;
            const long long ts = lo * nn - lo * (lo - 1) / 2 + (hi - lo);
            kv = Kc[ts * ldk + 4 * w + st];
            ik = ksym == 2 ? ts : ik;
            if (lo != hi) {
                const long long ta = nn * (nn + 1) / 2 + lo * (nn - 1) - lo * (lo - 1) / 2 + (hi - lo - 1);
                const zc ka = Kc[ta * ldk + 4 * w + st];
                kv = i < k ? kv + ka : kv - ka;
            }
        } else if (Kc) {
            kv = Kc[ik * ldk + 4 * w + st];
        } else {
            const long long cc = 2 * (4 * w + st);
            kv = mkz(Kr[ik * krs + cc * kcs], Kr[ik * krs + (cc + 1) * kcs]);
        }
        zc g = mkz(-kv.x, -kv.y);
        if (sg == tu) {
            if (J) g = g + (ksym == 2 && i != k ? 0.5 : 1.0) * J[ik * ldj + w];
            else g = g + mkz(Jr[ik * jrs + 2 * w * jcs], Jr[ik * jrs + (2 * w + 1) * jcs]);
            if (h) g.x += h[(long long)i * n + k];
        }
        Gam[e] = g;
    }
}

// ket-side gradient: V_w += H1 C + conj(h_w) C   (V already holds Gamma_w^H C - C W_w^H; Hb = H1 C is
// null when Gamma holds H1 + J - K, whose adjoint already brought H1 C in)
__global__ void ket_prep_kernel(int M, int N, int b, const zc *Hb, const zc *bra, const zc *e1, const zc *e2, zc *V,
                                long long ld) {
    const long long total = (long long)M * b * N;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < total; e += (long long)gridDim.x * NT) {
        long long r = e / ((long long)b * N), c = e - r * ((long long)b * N);
        int w = (int)(c / N), j = (int)(c - (long long)w * N);
        zc h = conjz(e1[w] + e2[w]);
        const zc hb = Hb ? Hb[r * N + j] : mkz(0.0, 0.0);
        V[r * ld + c] = V[r * ld + c] + hb + h * bra[r * N + j];
    }
}

// Y_w = R1[il] T2[:, rem] for a spin rotation R1 that is block diagonal with one 2 x 2 block per
// spatial orbital in the interleaved order r = 2p + sigma (R1b[(il n + p) 4 + 2 sigma + tau] =
// R1[il][2p + sigma][2p + tau]): row r of Y takes two rows of T2.  Point w = w0 + wl of the chunk
// belongs to Lebedev point il = w / blk and takes column block rem = w % blk of T2; Y is row-major
// M x (bc N) with leading dimension ld, as the GEMM form writes it.
__global__ void spin_block_y_kernel(int n, int N, int bc, int w0, int blk, const zc *__restrict__ R1b,
                                    const zc *__restrict__ T2, long long ld2, zc *__restrict__ Ys, long long ld) {
    const long long cols = (long long)bc * N, total = 2LL * n * cols;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < total; e += (long long)gridDim.x * NT) {
        const int r = (int)(e / cols);
        const long long c = e - (long long)r * cols;
        const int wl = (int)(c / N), j = (int)(c - (long long)wl * N);
        const int w = w0 + wl, il = w / blk, rem = w - il * blk;
        const int pp = r >> 1, sg = r & 1;
        const zc *B = R1b + ((long long)il * n + pp) * 4 + 2 * sg;
        const long long tc = (long long)rem * N + j;
        Ys[(long long)r * ld + c] = B[0] * T2[(long long)(2 * pp) * ld2 + tc] + B[1] * T2[(long long)(2 * pp + 1) * ld2 + tc];
    }
}

// Coulomb term of the tensor-core path: Gamma_w[2i + s][2k + s] += J_w(i, k) (+ h[i][k] with `h`: the
// one-electron matrix folded in, Gamma becoming the Fock matrix H1 + J - K) for both spins s, with
// J_w's real and imaginary parts at Jr[ik jrs + (2w) jcs] and Jr[ik jrs + (2w + 1) jcs] (Gamma already
// holds -K from the exchange GEMM).
__global__ void add_coulomb_diag_kernel(int n, int b, const double *Jr, long long jrs, long long jcs, zc *Gam,
                                        const double *h) {
    const int M = 2 * n;
    const long long nn = (long long)n * n, tot = 2LL * nn * b;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < tot; e += (long long)gridDim.x * NT) {
        const long long w = e / (2 * nn), rem = e - w * 2 * nn;
        const int sg = (int)(rem / nn);
        const long long ik = rem - (long long)sg * nn;
        const int i = (int)(ik / n), k = (int)(ik - (long long)i * n);
        zc *g = Gam + (w * M + 2 * i + sg) * M + 2 * k + sg;
        zc jv = mkz(Jr[ik * jrs + 2 * w * jcs], Jr[ik * jrs + (2 * w + 1) * jcs]);
        if (h) jv.x += h[ik];
        *g = *g + jv;
    }
}

// Symmetric and antisymmetric FP64 exchange rows of one panel from its Gram block (the symmetric
// exchange form; the tensor-core slicer slice_ek_sym_panel_kernel does the same with slices):
// pair (i, k) = pairs[t0 + r] of symmetric row r, B[l][j] = G[(i - i0) n + l][(k - k0) n + j];
// EKs[r][pair_le(l, j)] = B[l][j] + B[j][l] (l < j), B[l][l] (l = j); for i < k
// EKa[r - (i - i0) - 1][pair_lt(l, j)] = B[l][j] - B[j][l] (l < j).  Row lengths n(n+1)/2, n(n-1)/2.
// 32 x 32 tile pairs through shared memory, so that both B[l][j] and B[j][l] are read in rows.
__global__ void __launch_bounds__(256) ek_sym_panel_kernel(int n, int i0, int k0, const int *__restrict__ pairs,
                                                           long long t0, const double *__restrict__ G, long long ldg,
                                                           double *__restrict__ EKs, double *__restrict__ EKa) {
    __shared__ double T1[32 * 33], T2[32 * 33];
    const long long r = blockIdx.x, nn = n;
    const int pr = __ldg(pairs + t0 + r), i = pr >> 16, k = pr & 0xffff;
    const bool anti = i < k;
    const long long ra = r - (i - i0) - 1;
    const double *g = G + (long long)(i - i0) * n * ldg + (long long)(k - k0) * n;
    double *es = EKs + r * (nn * (nn + 1) / 2), *ea = anti ? EKa + ra * (nn * (nn - 1) / 2) : nullptr;
    const int nt = (n + 31) / 32, lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int lt = 0; lt < nt; ++lt) {
        for (int jt = lt; jt < nt; ++jt) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int a = ty + 8 * q;
                const int l1 = lt * 32 + a, j1 = jt * 32 + lane;
                T1[a * 33 + lane] = (l1 < n && j1 < n) ? g[(long long)l1 * ldg + j1] : 0.0;
                if (jt != lt) {
                    const int l2 = jt * 32 + a, j2 = lt * 32 + lane;
                    T2[a * 33 + lane] = (l2 < n && j2 < n) ? g[(long long)l2 * ldg + j2] : 0.0;
                }
            }
            __syncthreads();
            const double *U = (jt == lt) ? T1 : T2;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int a = ty + 8 * q, l = lt * 32 + a, j = jt * 32 + lane;
                if (l <= j && j < n) {
                    const double x = T1[a * 33 + lane], y = U[lane * 33 + a];
                    es[(long long)l * nn - (long long)l * (l - 1) / 2 + (j - l)] = (l == j) ? x : x + y;
                    if (anti && l < j) ea[(long long)l * (nn - 1) - (long long)l * (l - 1) / 2 + (j - l - 1)] = x - y;
                }
            }
            __syncthreads();
        }
    }
}

// Kin in the symmetric exchange form: rows t = pair_le(l, j) (pairs[t] = l << 16 | j) hold
// rho_s^{st}[l][j] = (rho_w[2l + s][2j + t] + rho_w[2j + s][2l + t]) / 2 at column 4w + st (row stride ldk);
// rows n(n+1)/2 + pair_lt(l, j), l < j, the antisymmetric halves (difference / 2).  rho_w dense M x M.
// With P: also P[t ldp + w] = the symmetric half of rho^{aa} + rho^{bb} (the thread of st = 0 adds st = 3's).
__global__ void gather_kin_sym_kernel(int n, int b, const int *__restrict__ pairs, const zc *rho, zc *Kin,
                                      long long ldk, zc *P, long long ldp) {
    const int M = 2 * n;
    const long long nn = n, kks = nn * (nn + 1) / 2, tot = kks * b * 4;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < tot; e += (long long)gridDim.x * NT) {
        const long long t = e / (4LL * b), c = e - t * 4LL * b, w = c >> 2;
        const int sg = (int)((c >> 1) & 1), tu = (int)(c & 1);
        const int pr = pairs[t], l = pr >> 16, j = pr & 0xffff;
        const zc *R = rho + w * (long long)M * M;
        const zc v = R[(long long)(2 * l + sg) * M + 2 * j + tu];
        if (l == j) {
            Kin[t * ldk + c] = v;
        } else {
            const zc u = R[(long long)(2 * j + sg) * M + 2 * l + tu];
            Kin[t * ldk + c] = mkz(0.5 * (v.x + u.x), 0.5 * (v.y + u.y));
            const long long ta = kks + (long long)l * (nn - 1) - (long long)l * (l - 1) / 2 + (j - l - 1);
            Kin[ta * ldk + c] = mkz(0.5 * (v.x - u.x), 0.5 * (v.y - u.y));
        }
        if (P && (c & 3) == 0) {
            const zc p = v + R[(long long)(2 * l + 1) * M + 2 * j + 1];
            const zc q = R[(long long)(2 * j) * M + 2 * l] + R[(long long)(2 * j + 1) * M + 2 * l + 1];
            P[t * ldp + w] = mkz(0.5 * (p.x + q.x), 0.5 * (p.y + q.y));
        }
    }
}

// One panel of the FP64 exchange matrix from its Gram block (streamed form): for r = (i - i0) n + k,
// EKp[r][l n + j] = G[(i - i0) n + l][k n + j] (ldg, lde: row strides), i.e. (il|kj) for the panel's i.
// One CTA per output row; for fixed l the n values j are contiguous on both sides.
__global__ void ek_panel_kernel(int n, const double *__restrict__ G, long long ldg, double *__restrict__ EKp,
                                long long lde) {
    const long long r = blockIdx.x;
    const int il = (int)(r / n), k = (int)(r - (long long)il * n);
    const double *g = G + (long long)il * n * ldg + (long long)k * n;
    double *e = EKp + r * lde;
    const int kk = n * n;
    for (int t = threadIdx.x; t < kk; t += NT) {
        const int l = t / n, j = t - l * n;
        e[t] = g[(long long)l * ldg + j];
    }
}

inline int grid_for(long long n) {
    long long g = (n + NT - 1) / NT;
    if (g > 148LL * 16) g = 148LL * 16;
    if (g < 1) g = 1;
    return (int)g;
}

}  // namespace

int launch_tprime(int Ltot, int N, int b, zc *T, long long ldT, zc *e2part, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    tprime_kernel<<<dim3(Ltot, b), NT, 0, st>>>(Ltot, N, T, ldT, e2part);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_rowsum(int nrows, int ncols, const zc *in, zc *out, double scale, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    rowsum_kernel<<<nrows, NT, 0, st>>>(ncols, in, out, scale);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_trace_conj(int M, int N, int b, const zc *C, zc *X, long long ldX, zc *out, double scale, cudaStream_t st,
                      const zc *add, const zc *sub, double sub_scale) {
    ProfScope prof(st, PROF_MEMORY);
    trace_conj_kernel<<<b, NT, 0, st>>>(M, N, C, X, ldX, out, scale, add, sub, sub_scale);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

// G <- G + A over a chunk (M rows x b N columns, row stride ldX)
__global__ void __launch_bounds__(NT) add_inplace_kernel(long long rows, long long cols, const zc *A, zc *G,
                                                         long long ldX) {
    const long long total = rows * cols;
    for (long long e = blockIdx.x * (long long)NT + threadIdx.x; e < total; e += (long long)gridDim.x * NT) {
        const long long r = e / cols, c = e - r * cols, o = r * ldX + c;
        G[o] = G[o] + A[o];
    }
}

int launch_add_inplace(int M, int N, int b, const zc *A, zc *G, long long ldX, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    add_inplace_kernel<<<grid_for((long long)M * b * N), NT, 0, st>>>(M, (long long)b * N, A, G, ldX);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

size_t accumulate_scratch_bytes(int nslot, int M, int N, int b) {
    const long long ngroups = (b + ACC_GROUP - 1) / ACC_GROUP;
    return (size_t)ngroups * ((size_t)nslot * M * N + nslot) * sizeof(AccPart);
}

int launch_accumulate(int nslot, int M, int N, int b, const zc *Wt, long long nomega, long long w0, const int *slotmap,
                      const zc *G, const zc *R, long long ldX, const zc *det, const zc *e1, const zc *e2, zc *accG,
                      zc *compG, zc *accR, zc *compR, zc *accHS, zc *compHS, void *scratch, cudaStream_t st,
                      int conj_weights) {
    const int ngroups = (b + ACC_GROUP - 1) / ACC_GROUP;
    AccPart *part = reinterpret_cast<AccPart *>(scratch);
    const long long nel = (long long)M * N + 1;
    {
        ProfScope prof(st, PROF_MEMORY);
        const dim3 grid((unsigned)((nel + ACC_NT - 1) / ACC_NT), (unsigned)ngroups, (unsigned)std::min(nslot, 65535));
        accumulate_partial_kernel<<<grid, ACC_NT, 0, st>>>(nslot, M, N, b, Wt, nomega, w0, G, R, ldX, det, e1, e2, part,
                                                           conj_weights);
    }
    ++g_launches;
    PHF_CHECK_LAUNCH();
    {
        ProfScope prof(st, PROF_MEMORY);
        const long long ctas = std::min<long long>((nslot * nel + ACC_NT / ACC_LANES - 1) / (ACC_NT / ACC_LANES), 1 << 20);
        accumulate_final_kernel<<<(unsigned)ctas, ACC_NT, 0, st>>>(nslot, M, N, slotmap, ngroups, part, accG, compG, accR,
                                                                   compR, accHS, compHS);
    }
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_ket_prep(int M, int N, int b, const zc *Hb, const zc *bra, const zc *e1, const zc *e2, zc *V, long long ld,
                    cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    ket_prep_kernel<<<grid_for((long long)M * b * N), NT, 0, st>>>(M, N, b, Hb, bra, e1, e2, V, ld);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_fold_out(int nslot, int M, int N, const int *rowmap, const FoldSums &S, zc *outG, zc *outR, zc *outHS,
                    cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    fold_out_kernel<<<dim3(grid_for((long long)M * N), (unsigned)std::min(2 * nslot + 1, 65535)), NT, 0, st>>>(
        nslot, M, N, rowmap, S, outG, outR, outHS);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_permute_h2(int M, const zc *H2, zc *H2r, cudaStream_t st) {
    long long tot = (long long)M * M * M * M;
    ProfScope prof(st, PROF_MEMORY);
    permute_h2_kernel<<<grid_for(tot), NT, 0, st>>>(M, H2, H2r);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_permute_rows(int M, int N, const int *rowmap, const zc *in, zc *out, zc *out2, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    permute_rows_kernel<<<grid_for((long long)M * N), NT, 0, st>>>(M, N, rowmap, in, out, out2);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_gather_p(int n, int b, const zc *rho, zc *P, long long ldp, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    gather_p_kernel<<<grid_for((long long)n * n * b), NT, 0, st>>>(n, b, rho, P, ldp);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_gather_kin(int n, int b, const zc *rho, zc *Kin, long long ldk, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    gather_kin_kernel<<<grid_for((long long)n * n * b * 4), NT, 0, st>>>(n, b, rho, Kin, ldk);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_spin_block_y(int n, int N, int bc, int w0, int blk, const zc *R1b, const zc *T2, long long ld2, zc *Ys,
                        long long ld, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    spin_block_y_kernel<<<grid_for(2LL * n * bc * N), NT, 0, st>>>(n, N, bc, w0, blk, R1b, T2, ld2, Ys, ld);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_add_coulomb_diag(int n, int b, const double *Jr, long long jrs, long long jcs, zc *Gam, cudaStream_t st,
                            const double *h) {
    ProfScope prof(st, PROF_MEMORY);
    add_coulomb_diag_kernel<<<grid_for(2LL * n * n * b), NT, 0, st>>>(n, b, Jr, jrs, jcs, Gam, h);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

// out (2M x 2N): rows 2j and 2j + 1 of the real operand of rho = X bra^H (see launch_bra_rho_operand)
__global__ void bra_rho_operand_kernel(int M, int N, const zc *bra, double *out) {
    const long long total = (long long)M * N;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(e / N), k = (int)(e - (long long)j * N);
        const zc b = bra[e];
        double *r0 = out + (long long)(2 * j) * (2 * N) + 2 * k, *r1 = r0 + 2 * N;
        r0[0] = b.x;
        r0[1] = b.y;
        r1[0] = -b.y;
        r1[1] = b.x;
    }
}

int launch_bra_rho_operand(int M, int N, const zc *bra, double *out, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    bra_rho_operand_kernel<<<grid_for((long long)M * N), NT, 0, st>>>(M, N, bra, out);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_ek_sym_panel(int n, int i0, int ipanel, int k0, const int *pairs, const double *G, long long ldg,
                        double *EKs, double *EKa, cudaStream_t st) {
    const long long rows_s = (long long)ipanel * (n - i0) - (long long)ipanel * (ipanel - 1) / 2;
    if (n < 1 || n > 65535 || i0 < 0 || ipanel < 1 || i0 + ipanel > n || k0 < 0 || k0 > i0 ||
        ldg < ((long long)n - k0) * n) {
        set_error(PHF_ERR_ARG, "launch_ek_sym_panel: panel outside the index range or a short Gram block");
        return PHF_ERR_ARG;
    }
    const long long nn = n, t0 = (long long)i0 * nn - (long long)i0 * (i0 - 1) / 2;
    ProfScope prof(st, PROF_MEMORY);
    ek_sym_panel_kernel<<<(unsigned)rows_s, 256, 0, st>>>(n, i0, k0, pairs, t0, G, ldg, EKs, EKa);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_gather_kin_sym(int n, int b, const int *pairs, const zc *rho, zc *Kin, long long ldk, cudaStream_t st,
                          zc *P, long long ldp) {
    ProfScope prof(st, PROF_MEMORY);
    gather_kin_sym_kernel<<<grid_for((long long)n * (n + 1) / 2 * b * 4), NT, 0, st>>>(n, b, pairs, rho, Kin, ldk, P,
                                                                                       ldp);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_ek_panel(int n, int ipanel, const double *G, long long ldg, double *EKp, long long lde, cudaStream_t st) {
    ProfScope prof(st, PROF_MEMORY);
    ek_panel_kernel<<<(unsigned)((long long)ipanel * n), NT, 0, st>>>(n, G, ldg, EKp, lde);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

int launch_assemble_gamma(int n, int b, const zc *J, long long ldj, const double *Jr, long long jrs, long long jcs,
                          const zc *Kc, long long ldk, const double *Kr, long long krs, long long kcs, zc *Gam,
                          cudaStream_t st, int ksym, const double *h) {
    ProfScope prof(st, PROF_MEMORY);
    assemble_gamma_kernel<<<grid_for(4LL * n * n * b), NT, 0, st>>>(n, b, J, ldj, Jr, jrs, jcs, Kc, ldk, Kr, krs, kcs,
                                                                    Gam, ksym, h);
    ++g_launches;
    PHF_CHECK_LAUNCH();
    return PHF_OK;
}

}  // namespace phf
