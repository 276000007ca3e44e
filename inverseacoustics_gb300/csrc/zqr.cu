// Complex FP64 Householder QR over a cluster of CTAs per matrix, with or
// without column pivoting (Businger-Golub).
//
// Bound by the FP64 pipe (two FMA per clock and SM): 8 FMA per element and step
// for the update, 2 more for the exact remaining norms of the pivoted form.
// One CTA per matrix left most SMs idle, and FP64 instructions that are
// predicated off still take the pipe's time.  Per call: 48 bins of 1280 x 192
// 73 -> 40 ms, 64 of 256 x 256 46 -> 14, 23 of 642 x 120 16 -> 4.6.  Here the columns of one matrix are dealt cyclically to the
// CTAs of a cluster, a warp per column; per step
//   - every CTA publishes its pivot candidate; one cluster barrier;
//   - every CTA reads the pivot column's rows (from L2; its owner wrote them
//     before the barrier) and forms the reflector itself, so the reflector is
//     not broadcast and a step needs one cluster barrier;
//   - a column's rows sit in the warp's registers between the two passes, the
//     32-row groups past the column's end skipped by branches.
// Nothing moves when columns are pivoted: perm says which column is which, and
// R's column k stands in column perm[k] (rows 0..k).  The arithmetic and its
// order are qr_kernel's (wide_solve.cu), pivots and ties included, whatever the
// cluster size: bitwise the same factors.
#include <cooperative_groups.h>
#include "ia_common.cuh"
#include "ia_internal.h"

namespace ia {

namespace cg = cooperative_groups;

constexpr int ZQ_THREADS = 256, ZQ_WARPS = ZQ_THREADS / 32, ZQ_MAX_CS = 8;
constexpr int ZQ_VWARPS = 16;   // partial sums of a reflector's norm (qr_kernel's 512 threads)

// order-preserving key of a remaining squared norm (0: a NaN, never preferred),
// so that the pivot search stays off the FP64 pipe
typedef unsigned long long zq_key;
__device__ __forceinline__ zq_key zq_norm_key(double v)
{
    const zq_key k = (zq_key)__double_as_longlong(fabs(v));
    return k <= 0x7FF0000000000000ull ? k + 1 : 0;
}

// KPL: 32-row slots of a column in registers (0: streamed twice); ZQ_GROUP of
// them are skipped or run together (one branch)
template <int KPL, int ZQ_GROUP, bool PIV>
__global__ void __launch_bounds__(ZQ_THREADS, 1) zqr_cluster_kernel(int rows, int cols, double2 *A, int lda,
                                                                   long long sA, double2 *tau, int *perm)
{
    cg::cluster_group cluster = cg::this_cluster();
    const int cs = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int f = blockIdx.x / cs;
    extern __shared__ __align__(16) unsigned char zq_smem[];
    double2 *xs = reinterpret_cast<double2 *>(zq_smem);          // rows: the scaled reflector (rows > j)
    double *cn = reinterpret_cast<double *>(xs + rows);          // own columns' remaining norms^2 (PIV)
    int *ord = reinterpret_cast<int *>(cn + cols);               // column in each position (PIV)
    int *pos = ord + cols;                                       // position of each column (PIV)
    __shared__ zq_key s_key[2];
    __shared__ int s_pos[2];
    __shared__ double s_red[ZQ_VWARPS];
    __shared__ double2 s_tau, s_sc, s_beta;
    __shared__ int s_none;
    A += f * sA;
    if (tau) tau += (size_t)f * cols;
    if (PIV) perm += (size_t)f * cols;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nown = cols > rank ? (cols - rank + cs - 1) / cs : 0;   // columns rank, rank + cs, ...
    const double2 zero = make_double2(0.0, 0.0);
    if (PIV) {
        for (int c = tid; c < cols; c += ZQ_THREADS) ord[c] = pos[c] = c;
        for (int q = wid; q < nown; q += ZQ_WARPS) {
            const double2 *c = A + (size_t)(rank + q * cs) * lda;
            double a = 0;
            for (int i = lane; i < rows; i += 32) a += zabs2(c[i]);
            a = warp_sum(a);
            if (lane == 0) cn[q] = a;
        }
    }
    const int steps = cols < rows ? cols : rows;
    int p = -1;              // the previous step's column
    for (int j = 0; j < steps; ++j) {
        const int par = j & 1;
        __syncthreads();     // this CTA's updates (and norms) are done
        if (PIV && wid == 0) {
            zq_key best = 0;
            int bi = cols;
            for (int q = lane; q < nown; q += 32) {
                const int ps = pos[rank + q * cs];
                if (ps < j) continue;
                const zq_key k = zq_norm_key(cn[q]);
                if (k > best || (k == best && ps < bi)) {
                    best = k;
                    bi = ps;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const zq_key ov = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) {
                    best = ov;
                    bi = oi;
                }
            }
            if (lane == 0) {
                s_key[par] = best;
                s_pos[par] = bi;
            }
        }
        cluster.sync();
        // every reader of the previous pivot column is past its loads: its
        // owner stores the diagonal (and, unpivoted, the reflector)
        if (p >= 0 && p % cs == rank && !s_none) {
            double2 *c = A + (size_t)p * lda;
            if (tid == 0) c[j - 1] = s_beta;
            if (!PIV)
                for (int i = j + tid; i < rows; i += ZQ_THREADS) c[i] = xs[i];
        }
        p = j;
        if (PIV) {
            zq_key bv = 0;
            int bi = cols;
            if (lane < cs) {
                bv = *cluster.map_shared_rank(&s_key[par], lane);
                bi = *cluster.map_shared_rank(&s_pos[par], lane);
            }
#pragma unroll
            for (int o = ZQ_MAX_CS / 2; o > 0; o >>= 1) {
                const zq_key ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > bv || (ov == bv && oi < bi)) {
                    bv = ov;
                    bi = oi;
                }
            }
            bi = __shfl_sync(0xffffffffu, bi, 0);
            p = ord[bi];
            __syncthreads();   // everyone has read ord
            if (tid == 0) {
                const int cj = ord[j];
                ord[j] = p;
                ord[bi] = cj;
                pos[p] = j;
                pos[cj] = cj == p ? j : bi;
                if (rank == 0) perm[j] = p;
            }
        }
        __syncthreads();     // xs is free (the store above read it)
        const double2 *x = A + (size_t)p * lda;
        const int len = rows - j;
        // sum of |x_i|^2, i >= 1, over 512 strided partial sums (two per thread)
#pragma unroll
        for (int h = 0; h < ZQ_VWARPS / ZQ_WARPS; ++h) {
            double sg = 0;
            for (int i = 1 + tid + h * ZQ_THREADS; i < len; i += 32 * ZQ_VWARPS) {
                const double2 v = __ldcg(x + j + i);
                xs[j + i] = v;
                sg += zabs2(v);
            }
            sg = warp_sum(sg);
            if (lane == 0) s_red[wid + h * ZQ_WARPS] = sg;
        }
        __syncthreads();
        if (tid == 0) {
            double sigma = 0;
            for (int w = 0; w < ZQ_VWARPS; ++w) sigma += s_red[w];
            const double2 alpha = __ldcg(x + j);
            s_none = sigma == 0 && alpha.y == 0;
            if (s_none) {
                s_tau = zero;
            } else {
                const double nrm = sqrt(zabs2_y(alpha) + sigma);
                const double beta = alpha.x >= 0 ? -nrm : nrm;
                s_tau = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
                s_sc = zrcp_y(make_double2(alpha.x - beta, alpha.y));
                s_beta = make_double2(beta, 0);
            }
            if (tau && p % cs == rank) tau[j] = s_tau;
        }
        __syncthreads();
        const bool none = s_none != 0;
        if (!none) {
            const double2 sc = s_sc;
            for (int i = 1 + tid; i < len; i += ZQ_THREADS) xs[j + i] = zmul(xs[j + i], sc);
        }
        __syncthreads();
        const double2 ctau = zconj(s_tau);
        const double2 *xj = xs + j;
        // own remaining columns (unpivoted: those after j)
        for (int q = wid; q < nown; q += ZQ_WARPS) {
            const int cidx = rank + q * cs;
            if (PIV ? pos[cidx] <= j : cidx <= j) continue;
            double2 *col = A + (size_t)cidx * lda + j;
            if (none) {
                // no reflector: the norm loses its row j
                if (PIV && lane == 0) {
                    const double v = cn[q] - zabs2(col[0]);
                    cn[q] = v > 0 ? v : 0;
                }
                continue;
            }
            double2 w = lane == 0 ? col[0] : zero;
            const double2 c0 = w;
            double nr = 0;
            if (KPL > 0) {
                constexpr int K = KPL > 0 ? KPL : 1;
                double2 v[K];
#pragma unroll
                for (int b = 0; b < K / ZQ_GROUP; ++b)
                    if (32 * ZQ_GROUP * b + 1 < len) {
#pragma unroll
                        for (int u = 0; u < ZQ_GROUP; ++u) {
                            const int i = 1 + lane + 32 * (b * ZQ_GROUP + u);
                            v[b * ZQ_GROUP + u] = i < len ? col[i] : zero;
                        }
                    }
#pragma unroll
                for (int b = 0; b < K / ZQ_GROUP; ++b)
                    if (32 * ZQ_GROUP * b + 1 < len) {
#pragma unroll
                        for (int u = 0; u < ZQ_GROUP; ++u) {
                            const int i = 1 + lane + 32 * (b * ZQ_GROUP + u);
                            if (i < len) zcfma(w, xj[i], v[b * ZQ_GROUP + u]);
                        }
                    }
                w = warp_sum2(w);
                w = zmul(ctau, w);
                if (lane == 0) col[0] = zsub(c0, w);
#pragma unroll
                for (int b = 0; b < K / ZQ_GROUP; ++b)
                    if (32 * ZQ_GROUP * b + 1 < len) {
#pragma unroll
                        for (int u = 0; u < ZQ_GROUP; ++u) {
                            const int i = 1 + lane + 32 * (b * ZQ_GROUP + u);
                            if (i < len) {
                                zfms(v[b * ZQ_GROUP + u], xj[i], w);
                                col[i] = v[b * ZQ_GROUP + u];
                                if (PIV) nr += zabs2(v[b * ZQ_GROUP + u]);
                            }
                        }
                    }
            } else {
                for (int i = 1 + lane; i < len; i += 32) zcfma(w, xj[i], col[i]);
                w = warp_sum2(w);
                w = zmul(ctau, w);
                if (lane == 0) col[0] = zsub(c0, w);
                for (int i = 1 + lane; i < len; i += 32) {
                    double2 e = col[i];
                    zfms(e, xj[i], w);
                    col[i] = e;
                    if (PIV) nr += zabs2(e);
                }
            }
            if (PIV) {
                nr = warp_sum(nr);
                if (lane == 0) cn[q] = nr;
            }
        }
    }
    cluster.sync();   // the last column's readers are done; no CTA leaves before its published words are read
    if (p >= 0 && p % cs == rank && !s_none) {
        double2 *c = A + (size_t)p * lda;
        if (tid == 0) c[steps - 1] = s_beta;
        if (!PIV)
            for (int i = steps + tid; i < rows; i += ZQ_THREADS) c[i] = xs[i];
    }
}

static size_t zq_smem_bytes(int rows, int cols)
{
    return sizeof(double2) * (size_t)rows + (sizeof(double) + 2 * sizeof(int)) * (size_t)cols;
}

constexpr size_t ZQ_SMEM_MAX = 200 * 1024;   // (one CTA per SM)
// a step's work beside the columns, in columns; time of CTAs that share an SM
constexpr double ZQ_STEP = 16.0, ZQ_SHARED = 1.5;

bool zqr_ok(int rows, int cols) { return zq_smem_bytes(rows, cols) <= ZQ_SMEM_MAX; }

template <bool PIV>
static int zqr_launch(ia_context *ctx, int rows, int cols, double2 *A, int lda, long long sA, double2 *tau, int *perm,
                      int batch)
{
    const size_t smem = zq_smem_bytes(rows, cols);
    auto kern = rows <= 256    ? zqr_cluster_kernel<8, 2, PIV>
                : rows <= 768  ? zqr_cluster_kernel<24, 2, PIV>
                : rows <= 1280 ? zqr_cluster_kernel<40, 4, PIV>
                               : zqr_cluster_kernel<0, 1, PIV>;
    IA_CUDA_TRY(allow_shared<(int)ZQ_SMEM_MAX>(kern));
    // The cluster size of least waves (cols / c + ZQ_STEP) among those with a
    // column per warp: a step's columns over the CTAs, plus what each CTA does for
    // itself (reflector, barrier: as long as about 16 columns of the update: 64
    // to 256 columns).  A cluster stays inside one GPC, so fewer run at once than c *
    // batch SMs hold: 46 of 3, 28 of 5, 15 of 8.  Two waves of larger
    // clusters can then beat one: 48 bins of 1280 x 192 44.3 ms with 2, 56.4 with
    // 3, 39.6 with 5; 90 bins 79.1 with 1, 59.5 with 3.  Up to 768 rows (and
    // streamed) two CTAs fit an SM; sharing it costs up to 1.6: 48 bins of 256 x
    // 256 17.9 ms with 3 (two clusters on shared SMs), 15.4 with 2 (none), 12.1
    // with 5 (all); 64 bins 15.4 with 2, 14.4 with 4.
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(ZQ_THREADS);
    lc.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    int cs = 1;
    double least = 0.0;
    for (int c : {8, 6, 5, 4, 3, 2, 1}) {
        if (c > 1 && c * ZQ_WARPS > cols) continue;
        lc.gridDim = dim3((unsigned)(c * batch));
        at[0].val.clusterDim.x = c;
        int alone = 0, fit = 0;   // clusters at once, a CTA per SM and as many as fit
        lc.dynamicSmemBytes = ZQ_SMEM_MAX;
        if (c * batch <= ctx->sm_count) IA_CUDA_TRY(cudaOccupancyMaxActiveClusters(&alone, kern, &lc));
        const double one = (double)cols / c + ZQ_STEP;
        if (alone >= batch) {   // no smaller cluster is faster than one wave of these
            if (!least || one < least) cs = c;
            break;
        }
        lc.dynamicSmemBytes = smem;
        IA_CUDA_TRY(cudaOccupancyMaxActiveClusters(&fit, kern, &lc));
        if (fit < 1) continue;
        const double cost = one * ((batch + fit - 1) / fit) * (c * fit > ctx->sm_count ? ZQ_SHARED : 1.0);
        if (!least || cost < least) {
            least = cost;
            cs = c;
        }
    }
    lc.dynamicSmemBytes = smem;
    lc.gridDim = dim3((unsigned)(cs * batch));
    at[0].val.clusterDim.x = cs;
    IA_CUDA_TRY(cudaLaunchKernelEx(&lc, kern, rows, cols, A, lda, sA, tau, perm));
    IA_LAUNCH_CHECK(ctx);
    return IA_OK;
}

// R of the column-pivoted QR in place, unmoved columns: R(i, k) at
// A(i, perm[k]), i <= k; what stands below is not meaningful
int zqr_pivoted_batched(ia_context *ctx, int rows, int cols, double2 *A, int lda, long long sA, int *perm, int batch)
{
    return zqr_launch<true>(ctx, rows, cols, A, lda, sA, nullptr, perm, batch);
}

// R above the diagonal, reflectors (v(j) = 1) below, tau (may be null) as
// LAPACK's zgeqrf
int zqr_plain_batched(ia_context *ctx, int rows, int cols, double2 *A, int lda, long long sA, double2 *tau, int batch)
{
    return zqr_launch<false>(ctx, rows, cols, A, lda, sA, tau, nullptr, batch);
}

}  // namespace ia
