// Complex FP64 LU factorisation and solves of the FP64 path, batched.
//
// GB300's FP64 pipe does two FMA per clock and SM, so an LU on it is bound by
// that pipe wherever it runs: 32-column panels on one SM per matrix took
// 340 us each, the trailing updates ran at the pipe's 1.05 TFLOP/s.  Here
//   - the panel (ZLU_NB columns) is spread over a cluster of CTAs, rows split,
//     each CTA's share in its shared memory (zlu_panel_kernel): the FP64 pipes
//     of up to 8 SMs work on one matrix, one cluster barrier per column
//     (n = 642: 270 us per 64 columns of one matrix, was 680);
//   - everything of rank ZLU_NB -- the trailing updates of the factorisation and
//     of both triangular solves -- runs on the tensor cores on 10 BF16 slices
//     per operand (tc_gemm.cu): 2^-59 of a row's and a column's largest entry, and
//     meshes and source sets grade rows or columns, not the panel's inside (edge
//     lengths over 1:1400, distances over 1:1e4: as near as FP64 updates or nearer);
//   - the triangular solves with the ZLU_NB x ZLU_NB diagonal blocks stay in
//     FP64 substitution (zlu_trsm_kernel).
// LAPACK getrf semantics: pivot of largest |re| + |im|, first row on ties,
// interchanges of whole rows, ipiv 0-based; a zero pivot sets
// IA_INFO_SINGULAR, a column without a comparable value IA_INFO_NONFINITE.
// Transfer matrices of 642 nodes and 120 points: 1 bin 16.4 -> 6.3 ms, 23 bins
// 58.9 -> 26.5 ms (the assembly is 1.2 and 13 ms of these).
// Replaces cusolverDnZZgels / zgels_ (CUDA/ibem.cuh:391, :755).
#include <cooperative_groups.h>
#include "ia_common.cuh"
#include "ia_internal.h"

namespace ia {

namespace cg = cooperative_groups;

// Width of a panel and rank of an update.  64: half the FP64 work of 128 in
// panels and diagonal blocks at the same tensor-core time (a rank-64 update's
// tile costs ~10 us of MMAs and ~6 us of set-up and epilogue).
constexpr int ZLU_NB = 64;
// Small matrices of more than one panel: panels of 32 columns and rank-32 FP64
// GEMMs (staged panels, dense.cu).  For a few bins the panels' latency sets the
// time and the two forms are level (transfer of 8 bins: n = 92 1.07 ms against
// 1.08 with rank-64 slice products; n = 162, 1 bin 1.42 and 1.41 ms); at 64 bins
// the slices would gain 6 % (n = 162), but the choice must not depend on the
// batch: a bin's results are bitwise those it has alone or in another split.
constexpr int ZLU_SMALL_N = 192;
constexpr int ZP_THREADS = 256;
constexpr int ZP_MAX_CS = 8;
constexpr size_t ZP_SMEM_MAX = 200 * 1024;

// |re| + |im| as an integer key (1 + its bits; 0 for a NaN and for no candidate):
// comparisons then stay off the FP64 pipe, where one warp instruction takes 16
// cycles and a column's reductions would cost as much as its update
typedef unsigned long long zp_key;
__device__ __forceinline__ zp_key zp_abs(double2 a)
{
    const zp_key k = (zp_key)__double_as_longlong(fabs(a.x) + fabs(a.y));
    return k <= 0x7FF0000000000000ull ? k + 1 : 0;
}
__device__ __forceinline__ bool zp_better(zp_key v, int i, zp_key bv, int bi) { return v > bv || (v == bv && i < bi); }

// Panel rows k0..n-1, columns k0..k0+nb-1 of one matrix over the cluster: CTA q
// holds rows [q rpc, (q+1) rpc) of the panel, column-major in shared memory.
// Per column every CTA publishes its pivot candidate with the candidate's
// panel row, and the owner of the current row that row (double-buffered by
// column parity, so one cluster barrier per column is enough: a buffer is
// rewritten two columns later, past a barrier that every reader has reached);
// after the barrier each CTA picks the same pivot, copies the pivot row, does
// its side of the interchange and updates its own rows.  The search of the
// next column rides in the update.
__global__ void __launch_bounds__(ZP_THREADS) zlu_panel_kernel(int n, double2 *A, int lda, long long sA, int *ipiv,
                                                              int k0, int nb, int rpc, int *info)
{
    cg::cluster_group cluster = cg::this_cluster();
    const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int f = blockIdx.x / cs;
    extern __shared__ __align__(16) unsigned char zp_smem[];
    double2 *P = reinterpret_cast<double2 *>(zp_smem);     // nb columns of rpc rows
    double2 *prow = P + (size_t)nb * rpc;                  // nb: the pivot row
    double2 *pub = prow + nb;                              // 2 x (candidate row, current row) x nb
    __shared__ zp_key s_val[2], s_wv[ZP_THREADS / 32];
    __shared__ int s_idx[2], s_wi[ZP_THREADS / 32];
    __shared__ double2 s_inv;
    A += f * sA;
    ipiv += (size_t)f * n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int pr = n - k0, r0 = rank * rpc, nr = max(0, min(rpc, pr - r0));   // panel rows r0 .. r0 + nr - 1
    for (int e = tid; e < nr * nb; e += ZP_THREADS) {
        const int c = e / nr, i = e - c * nr;
        P[(size_t)c * rpc + i] = A[k0 + r0 + i + (size_t)(k0 + c) * lda];
    }
    __syncthreads();
    // thread (row i of a slab of RT rows, column group g of NG)
    const int RT = min(ZP_THREADS, (rpc + 31) & ~31), NG = ZP_THREADS / RT;
    const int ti = tid % RT, tg = tid / RT;
    zp_key best = 0;
    int bi = n;
    if (tg == 0)
        for (int i = ti; i < nr; i += RT) {
            const zp_key v = zp_abs(P[i]);
            if (v > best) {
                best = v;
                bi = r0 + i;
            }
        }
    for (int j = 0; j < nb; ++j) {
        // this CTA's candidate, published with its row
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const zp_key ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (zp_better(ov, oi, best, bi)) {
                best = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            s_wv[wid] = best;
            s_wi[wid] = bi;
        }
        __syncthreads();
        best = s_wv[0];
        bi = s_wi[0];
        for (int w = 1; w < ZP_THREADS / 32; ++w)
            if (zp_better(s_wv[w], s_wi[w], best, bi)) {
                best = s_wv[w];
                bi = s_wi[w];
            }
        const int par = j & 1;
        double2 *crow = pub + (size_t)(2 * par) * nb, *jrow = crow + nb;
        if (tid == 0) {
            s_val[par] = best;
            s_idx[par] = bi;
        }
        const int own_j = j / rpc;
        if (tid < nb) {
            if (bi < n) crow[tid] = P[(size_t)tid * rpc + (bi - r0)];
            if (rank == own_j) jrow[tid] = P[(size_t)tid * rpc + (j - r0)];
        }
        cluster.sync();
        zp_key bv = 0;
        int piv = n;
        if (lane < cs) {
            bv = *cluster.map_shared_rank(&s_val[par], lane);
            piv = *cluster.map_shared_rank(&s_idx[par], lane);
        }
#pragma unroll
        for (int o = ZP_MAX_CS / 2; o > 0; o >>= 1) {
            const zp_key ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, piv, o);
            if (zp_better(ov, oi, bv, piv)) {
                bv = ov;
                piv = oi;
            }
        }
        bv = __shfl_sync(0xffffffffu, bv, 0);
        piv = __shfl_sync(0xffffffffu, piv, 0);
        if (bv <= 1) piv = j;   // no comparable entry (0), or the largest is zero (1)
        if (rank == 0 && tid == 0) {
            if (bv <= 1) atomicOr(&info[f], bv ? IA_INFO_SINGULAR : IA_INFO_NONFINITE);
            ipiv[k0 + j] = k0 + piv;
        }
        if (tid < nb) {
            const int own_p = piv / rpc;
            double2 *rj = cluster.map_shared_rank(jrow, own_j);
            double2 pv;
            if (piv == j) {
                pv = rj[tid];
            } else {
                pv = cluster.map_shared_rank(crow, own_p)[tid];
                if (rank == own_p) P[(size_t)tid * rpc + (piv - r0)] = rj[tid];
                if (rank == own_j) P[(size_t)tid * rpc + (j - r0)] = pv;
            }
            prow[tid] = pv;
            if (tid == j && (pv.x != 0.0 || pv.y != 0.0)) s_inv = zrcp_x(pv);   // one division
        }
        __syncthreads();
        // multipliers of the rows below j
        const int i0 = max(0, j + 1 - r0);
        double2 *cj = P + (size_t)j * rpc;
        const double2 d = prow[j];
        if (d.x != 0.0 || d.y != 0.0) {
            const double2 inv = s_inv;
            for (int i = i0 + tid; i < nr; i += ZP_THREADS) cj[i] = zmul(cj[i], inv);
        }
        __syncthreads();
        best = 0;
        bi = n;
        if (j + 1 < nb && tg < NG) {
            for (int i = i0 + ti; i < nr; i += RT) {
                const double2 l = cj[i];
                for (int c = j + 1 + tg; c < nb; c += NG) {
                    double2 *p = P + (size_t)c * rpc + i;
                    double2 v = *p;
                    zfms(v, l, prow[c]);
                    *p = v;
                    if (c == j + 1) {
                        const zp_key av = zp_abs(v);
                        if (av > best) {
                            best = av;
                            bi = r0 + i;
                        }
                    }
                }
            }
        }
        // (the next column's candidate reduction starts with warp shuffles and
        // a CTA barrier, after which every update above is visible)
    }
    cluster.sync();   // no CTA leaves while another may read its published rows
    for (int e = tid; e < nr * nb; e += ZP_THREADS) {
        const int c = e / nr, i = e - c * nr;
        A[k0 + r0 + i + (size_t)(k0 + c) * lda] = P[(size_t)c * rpc + i];
    }
}

// The net row permutation of the interchanges j <-> ipiv[j], j = k0 .. kend-1,
// simulated once per CTA in shared memory: cur[i] = the row that ends in
// position i (rows k0 .. n-1, stored at cur[i - k0]).
__device__ __forceinline__ void zlu_permutation(int n, const int *ipiv, int k0, int kend, int *cur)
{
    for (int i = k0 + (int)threadIdx.x; i < n; i += blockDim.x) cur[i - k0] = i;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int j = k0; j < kend; ++j) {
            const int p = ipiv[j];
            if (p != j) {
                const int t = cur[j - k0];
                cur[j - k0] = cur[p - k0];
                cur[p - k0] = t;
            }
        }
    __syncthreads();
}

// Interchanges of a panel applied to the columns outside [k0, kend), a warp per
// column: the at most 2 ZLU_NB moved rows are listed once per CTA, then each
// column loads all its old values and stores them (independent accesses, where
// interchanging one by one was a chain of 34 us).
constexpr int ZS_WARPS = 8;

__global__ void __launch_bounds__(32 * ZS_WARPS) zlu_laswp_kernel(int n, double2 *A, int lda, long long sA,
                                                                  const int *ipiv, int k0, int kend)
{
    extern __shared__ int zs_cur[];   // n - k0
    __shared__ int dst[2 * ZLU_NB], src[2 * ZLU_NB], s_cnt, s_piv[ZLU_NB];
    const int f = blockIdx.y, nb = kend - k0, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    A += f * sA;
    ipiv += (size_t)f * n;
    if (threadIdx.x == 0) s_cnt = 0;
    if (threadIdx.x < nb) s_piv[threadIdx.x] = ipiv[k0 + threadIdx.x];
    __syncthreads();
    zlu_permutation(n, s_piv - k0, k0, kend, zs_cur);
    for (int i = k0 + (int)threadIdx.x; i < n; i += blockDim.x)
        if (zs_cur[i - k0] != i) {
            const int s = atomicAdd(&s_cnt, 1);   // at most 2 nb rows move; their order does not matter
            dst[s] = i;
            src[s] = zs_cur[i - k0];
        }
    __syncthreads();
    const int cnt = s_cnt;
    int c = blockIdx.x * ZS_WARPS + wid;
    if (c >= n - nb) return;
    if (c >= k0) c += nb;
    double2 *a = A + (size_t)c * lda;
    double2 v[2 * ZLU_NB / 32];
#pragma unroll
    for (int q = 0; q < 2 * ZLU_NB / 32; ++q)
        if (lane + 32 * q < cnt) v[q] = a[src[lane + 32 * q]];
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2 * ZLU_NB / 32; ++q)
        if (lane + 32 * q < cnt) a[dst[lane + 32 * q]] = v[q];
}

// All interchanges applied to one right-hand-side column per CTA
__global__ void __launch_bounds__(256) zlu_apply_pivots_kernel(int n, const int *ipiv, double2 *B, int ldb,
                                                              long long sB)
{
    extern __shared__ __align__(16) unsigned char zap_smem[];
    double2 *col = reinterpret_cast<double2 *>(zap_smem);     // n
    int *cur = reinterpret_cast<int *>(col + n), *pv = cur + n;
    const int f = blockIdx.y;
    ipiv += (size_t)f * n;
    double2 *b = B + f * sB + (size_t)blockIdx.x * ldb;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        pv[i] = ipiv[i];
        col[i] = b[i];
    }
    __syncthreads();
    zlu_permutation(n, pv, 0, n, cur);
    for (int i = threadIdx.x; i < n; i += blockDim.x) b[i] = col[cur[i]];
}

// X <- T^-1 X for one diagonal block T (nb <= 64; unit lower, or upper) and
// ZT_RB columns of X per CTA, a warp per column: two 32-row halves, lane per
// row, each solved entry broadcast by shuffle; the off-diagonal quarter from
// shared memory between them.  Four columns per CTA: a column costs ~6000
// cycles of its SM's FP64 pipe, so a few columns per CTA spread one matrix over
// the SMs, and three CTAs share an SM.
constexpr int ZT_RB = 4;
constexpr int ZT_LD = ZLU_NB + 1;

__device__ __forceinline__ double2 shfl_z(double2 v, int src)
{
    return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

template <bool UPPER>
__global__ void __launch_bounds__(32 * ZT_RB) zlu_trsm_kernel(int nb, const double2 *Tm, int ldt, long long sT,
                                                             double2 *X, int ldx, long long sX, int ncols)
{
    extern __shared__ __align__(16) unsigned char zt_smem[];
    double2 *D = reinterpret_cast<double2 *>(zt_smem);            // D[c * ZT_LD + r], zero outside the triangle
    double2 *q = D + ZLU_NB * ZT_LD;                              // 1 / d_r (UPPER)
    const int f = blockIdx.y, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    Tm += f * sT;
    const double2 zero = make_double2(0.0, 0.0);
    const int nd = nb <= 32 ? 32 : ZLU_NB;   // rows and columns of the block that are used
    for (int e = threadIdx.x; e < nd * nd; e += 32 * ZT_RB) {
        const int r = e % nd, c = e / nd;
        const bool in = r < nb && c < nb && (UPPER ? r <= c : r > c);
        D[c * ZT_LD + r] = in ? Tm[r + (size_t)c * ldt] : zero;
    }
    __syncthreads();
    if (UPPER) {
        // rows times the reciprocal of their diagonal entry: the substitution
        // then has no division in its chain
        for (int r = threadIdx.x; r < ZLU_NB; r += 32 * ZT_RB)
            q[r] = r < nb ? zdiv(make_double2(1.0, 0.0), D[r * ZT_LD + r]) : zero;
        __syncthreads();
        for (int e = threadIdx.x; e < nd * nd; e += 32 * ZT_RB) {
            const int r = e % nd, c = e / nd;
            if (r < c) D[c * ZT_LD + r] = zmul(D[c * ZT_LD + r], q[r]);
        }
        __syncthreads();
    }
    const int col = blockIdx.x * ZT_RB + wid;
    if (col >= ncols) return;
    double2 *x = X + f * sX + (size_t)col * ldx;
    double2 v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        v[h] = lane + 32 * h < nb ? x[lane + 32 * h] : zero;
        if (UPPER) v[h] = zmul(v[h], q[lane + 32 * h]);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int h = UPPER ? 1 - s : s, b0 = 32 * h;
        if (h == 1 && nb <= 32) continue;   // a block of one half
        // the half's own triangle
        double2 w = v[h];
#pragma unroll 8
        for (int t = 0; t < 31; ++t) {
            const int r = UPPER ? 31 - t : t;
            const double2 xr = shfl_z(w, r);
            if (UPPER ? lane < r : lane > r) zfms(w, D[(b0 + r) * ZT_LD + b0 + lane], xr);
        }
        v[h] = w;
        // the other half's rows (after the first half only)
        if (s == 0 && nb > 32) {
            double2 o = v[1 - h];
            const int o0 = 32 * (1 - h);
#pragma unroll 8
            for (int r = 0; r < 32; ++r) zfms(o, D[(b0 + r) * ZT_LD + o0 + lane], shfl_z(w, r));
            v[1 - h] = o;
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (lane + 32 * h < nb) x[lane + 32 * h] = v[h];
}

static constexpr size_t zt_smem_bytes() { return sizeof(double2) * (size_t)ZLU_NB * (ZT_LD + 1); }

template <bool UPPER>
static int ztrsm(ia_context *ctx, int nb, const double2 *T, int ldt, long long sT, double2 *X, int ldx, long long sX,
                 int ncols, int batch)
{
    IA_CUDA_TRY(allow_shared<(int)zt_smem_bytes()>(zlu_trsm_kernel<UPPER>));
    zlu_trsm_kernel<UPPER><<<dim3((ncols + ZT_RB - 1) / ZT_RB, batch), 32 * ZT_RB, zt_smem_bytes(), ctx->stream>>>(
        nb, T, ldt, sT, X, ldx, sX, ncols);
    IA_LAUNCH_CHECK(ctx);
    return IA_OK;
}

// ---- FP64 products on the tensor cores -------------------------------------
// K per product (exact level sums) and bytes of slice planes held at once;
// longer products accumulate over K, larger batches go in groups of bins.
constexpr int ZTC_K = 768;
constexpr size_t ZTC_PLANE_BYTES = size_t(2) << 30;

static size_t ztc_bytes(int M, int N, int K, int batch)
{
    const int k = K < ZTC_K ? K : ZTC_K;
    return tc_planes_bytes(M, k, TC_SLICES_FP64, false, batch) + tc_planes_bytes(N, k, TC_SLICES_FP64, true, batch) + 512;
}

size_t zgemm_tc_ws_bytes(int M, int N, int K, int batch)
{
    const size_t one = ztc_bytes(M, N, K, 1), all = one * batch, cap = one > ZTC_PLANE_BYTES ? one : ZTC_PLANE_BYTES;
    return all < cap ? all : cap;
}

int zgemm_tc(ia_context *ctx, Op opa, Op opb, int M, int N, int K, double alpha, const double2 *A, int lda,
             long long sA, const double2 *B, int ldb, long long sB, double beta, double2 *C, int ldc, long long sC,
             int batch, int *info, WsCursor scratch)
{
    if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return IA_ERR_ARG;
    const size_t fit = scratch.cap > scratch.off ? (scratch.cap - scratch.off) / ztc_bytes(M, N, K, 1) : 0;
    if (fit < 1) return IA_ERR_ALLOC;
    const int groups = (int)((batch + fit - 1) / fit), g = (batch + groups - 1) / groups;
    for (int f0 = 0; f0 < batch; f0 += g) {
        const int nf = batch - f0 < g ? batch - f0 : g;
        for (int k0 = 0; k0 < K; k0 += ZTC_K) {
            const int kk = K - k0 < ZTC_K ? K - k0 : ZTC_K;
            WsCursor cur = scratch;
            TcPlanes pa{}, pb{};
            const double2 *a = A + f0 * sA + (opa == OP_N ? (size_t)k0 * lda : (size_t)k0);
            const double2 *b = B + f0 * sB + (opb == OP_N ? (size_t)k0 : (size_t)k0 * ldb);
            int st = tc_slice_pair(ctx, opa, a, lda, sA, M, opb, b, ldb, sB, N, kk, TC_SLICES_FP64, nf, pa, pb, cur);
            if (!st)
                st = tc_gemm(ctx, pa, pb, M, N, alpha, k0 ? 1.0 : beta, C + f0 * sC, ldc, sC, nf,
                             info ? info + f0 : nullptr);
            if (st) return st;
        }
    }
    return IA_OK;
}

// ---- factorisation and solves ------------------------------------------------
// cluster size for a panel of pr rows: the smallest whose shares fit, doubled
// while the batch leaves SMs idle and a CTA keeps 32 rows
static bool zlu_panel_shape(const ia_context *ctx, int pr, int nb, int batch, int &cs, int &rpc, size_t &smem)
{
    auto bytes = [&](int r) { return sizeof(double2) * ((size_t)nb * r + 5 * (size_t)nb); };
    int best = 0;
    for (int c : {1, 2, 4, 8}) {
        const int r = (pr + c - 1) / c;
        if (bytes(r) > ZP_SMEM_MAX) continue;
        if (!best || (c * batch <= ctx->sm_count && r >= 32)) best = c;
    }
    if (!best) return false;
    cs = best;
    rpc = (pr + cs - 1) / cs;
    smem = bytes(rpc);
    return true;
}

// the tensor-core solver takes every n whose widest panel fits a cluster
// (n <= 1560); above, the FP64 pipe's blocked solver (dense.cu)
static bool zlu_ok(const ia_context *ctx, int n)
{
    int cs, rpc;
    size_t smem;
    return zlu_panel_shape(ctx, n, ZLU_NB, 1, cs, rpc, smem);
}

size_t zlu_ws_bytes(int n, int nrhs, int batch)
{
    const int w = nrhs > n ? nrhs : n;
    return zgemm_tc_ws_bytes(n, w, ZLU_NB, batch);
}

int zgetrf_ws(ia_context *ctx, int n, double2 *A, int lda, long long sA, int *ipiv, int *info, int batch,
              WsCursor scratch, bool plain)
{
    if (!zlu_ok(ctx, n)) return zgetrf_batched(ctx, n, A, lda, sA, ipiv, info, batch);
    IA_CUDA_TRY(allow_shared<(int)ZP_SMEM_MAX>(zlu_panel_kernel));
    int st;
    const bool small = plain || (n > ZLU_NB && n <= ZLU_SMALL_N);
    const int NB = small ? ZLU_NB / 2 : ZLU_NB;
    for (int k0 = 0; k0 < n; k0 += NB) {
        const int nb = n - k0 < NB ? n - k0 : NB, kend = k0 + nb, rest = n - kend;
        int cs, rpc;
        size_t smem;
        if (!zlu_panel_shape(ctx, n - k0, nb, batch, cs, rpc, smem)) return IA_ERR_TOO_LARGE;
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3((unsigned)(cs * batch));
        lc.blockDim = dim3(ZP_THREADS);
        lc.dynamicSmemBytes = smem;
        lc.stream = ctx->stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        lc.attrs = at;
        lc.numAttrs = 1;
        IA_CUDA_TRY(cudaLaunchKernelEx(&lc, zlu_panel_kernel, n, A, lda, sA, ipiv, k0, nb, rpc, info));
        IA_LAUNCH_CHECK(ctx);
        if (n > nb) {
            zlu_laswp_kernel<<<dim3((n - nb + ZS_WARPS - 1) / ZS_WARPS, batch), 32 * ZS_WARPS,
                               sizeof(int) * (size_t)(n - k0), ctx->stream>>>(n, A, lda, sA, ipiv, k0, kend);
            IA_LAUNCH_CHECK(ctx);
        }
        if (rest <= 0) break;
        double2 *u12 = A + k0 + (size_t)kend * lda;
        if ((st = ztrsm<false>(ctx, nb, A + k0 + (size_t)k0 * lda, lda, sA, u12, lda, sA, rest, batch))) return st;
        const double2 *l21 = A + kend + (size_t)k0 * lda;
        double2 *a22 = A + kend + (size_t)kend * lda;
        if (small)
            st = zgemm_batched(ctx, OP_N, OP_N, rest, rest, nb, make_double2(-1.0, 0.0), l21, lda, sA, u12, lda, sA,
                               make_double2(1.0, 0.0), a22, lda, sA, batch);
        else
            st = zgemm_tc(ctx, OP_N, OP_N, rest, rest, nb, -1.0, l21, lda, sA, u12, lda, sA, 1.0, a22, lda, sA, batch,
                          info, scratch);
        if (st) return st;
    }
    return IA_OK;
}

int zgetrs_ws(ia_context *ctx, int n, int nrhs, const double2 *LU, int lda, long long sA, const int *ipiv, double2 *B,
              int ldb, long long sB, int batch, int *info, WsCursor scratch)
{
    if (n <= 0 || nrhs <= 0 || batch <= 0) return IA_OK;
    if (!zlu_ok(ctx, n)) return zgetrs_batched(ctx, n, nrhs, LU, lda, sA, ipiv, B, ldb, sB, batch);
    int st;
    const size_t psm = (size_t)n * (sizeof(double2) + 2 * sizeof(int));
    zlu_apply_pivots_kernel<<<dim3(nrhs, batch), 256, psm, ctx->stream>>>(n, ipiv, B, ldb, sB);
    IA_LAUNCH_CHECK(ctx);
    for (int k0 = 0; k0 < n; k0 += ZLU_NB) {
        const int nb = n - k0 < ZLU_NB ? n - k0 : ZLU_NB, kend = k0 + nb;
        if ((st = ztrsm<false>(ctx, nb, LU + k0 + (size_t)k0 * lda, lda, sA, B + k0, ldb, sB, nrhs, batch))) return st;
        if (kend < n && (st = zgemm_tc(ctx, OP_N, OP_N, n - kend, nrhs, nb, -1.0, LU + kend + (size_t)k0 * lda, lda,
                                       sA, B + k0, ldb, sB, 1.0, B + kend, ldb, sB, batch, info, scratch)))
            return st;
    }
    for (int k0 = ((n - 1) / ZLU_NB) * ZLU_NB; k0 >= 0; k0 -= ZLU_NB) {
        const int nb = n - k0 < ZLU_NB ? n - k0 : ZLU_NB;
        if ((st = ztrsm<true>(ctx, nb, LU + k0 + (size_t)k0 * lda, lda, sA, B + k0, ldb, sB, nrhs, batch))) return st;
        if (k0 > 0 && (st = zgemm_tc(ctx, OP_N, OP_N, k0, nrhs, nb, -1.0, LU + (size_t)k0 * lda, lda, sA, B + k0, ldb,
                                     sB, 1.0, B, ldb, sB, batch, info, scratch)))
            return st;
    }
    return IA_OK;
}

}  // namespace ia
