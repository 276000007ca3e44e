// Start of the FP64 one-sided Jacobi iteration (wide_solve.cu): M = R K with K
// unitary and the columns of M nearly orthogonal.
//
// On R (here the lower triangular factor R^H of the pivoted QR) the FP64 Jacobi
// takes 8 to 11 sweeps, nearly all pairs rotating in all but the last
// two or three, on the FP64 pipe (two FMA per clock and SM; 20 FMA per row of a
// rotated pair, 8 of a tested one).  Here the rotations are found in FP32 and
// the FP64 work is products on the tensor cores (10 BF16 slices, zgemm_tc):
//   1. FP32 Jacobi of R scaled by a power of two; the rotations are recorded and
//      then applied to J;
//   2. J's polar factor in FP64: with E = I - J^H J (|E|_F ~ 2e-4 in FP32),
//      J <- J + J (E / 2 + 3 E^2 / 8 + E^2 (5 E / 16 + 35 E^2 / 128)), unitary to
//      |E|^5 (cf. Higham, Functions of Matrices, ch. 8);  M = R J: couplings
//      |m_i^H m_j| / |m_i||m_j| ~ 1e-5;
//   3. three times: G = M^H M, T_ij = G_ij / (G_jj - G_ii) anti-Hermitian, the
//      first-order rotation that removes G_ij, with the large entries (near-equal
//      norms) left out; M <- M K, K = (I + T)(I - T^2)^(-1/2), the polar factor of
//      I + T, by its series: to T^11 in the first step (|T| <= 0.05), to T^4 in
//      the second (|T| <= 6e-4), to T^2 in the third (|T| <= 5e-6).  Each step
//      squares the couplings; the third clears the smallest columns, whose
//      products the large ones hide before the first;
//   4. what is left -- near-equal singular values, columns at the rounding level
//      of the largest -- in FP64 sweeps over the pairs that G = M^H M shows above
//      the Jacobi's test, G anew for each: a sweep costs its rotations and a
//      barrier per round, not a dot product per pair.
// A bin is done when none of its pairs is above the test; the FP64 Jacobi runs
// those that are not (none, as a rule) as before; a bin whose J is not usable starts from R itself.
// K is unitary to FP64 rounding, so the decomposition is normwise backward
// stable; a small column of M carries that rounding of the large ones, so
// U^H b is formed from U = M / sigma instead of being carried along.
// (Mixed-precision Jacobi SVD: Gao, Ma, Shao 2022; Hermitian refinement: Ogita
// and Aishima 2018.)
#include "ia_common.cuh"
#include "ia_internal.h"

namespace ia {

// Sizes that take the start.  GCV solves of N x 4 N operators whose singular values
// fall to the rounding level (the start's worst case: the tail's pairs still rotate),
// without and with it, ms: N = 64, 1 bin 4.74 / 2.54, 150 bins 14.7 / 6.0, 512 bins
// 55.7 / 19.5; 120: 15.7 / 6.3, 77.7 / 26.1, 308 / 90; 192: 43.4 / 14.7, 310 / 83;
// 256: 88 / 27.6, 851 / 176; monopole operators gain more (64: 512 bins 55.5 / 17.4;
// 120: 266 / 54).  Below 64 it would pay too (48: 3.15 / 2.08, 512 bins 26.7 / 11.3;
// 40: 2.50 / 1.91, 17.7 / 9.3): the line is where an earlier form of the start was
// level, and small arrays keep the digits they have.  The upper end is the recorded
// rotations' 128 slots.
constexpr int JS_MIN_N = 64, JS_MAX_N = 256;
constexpr int JS_FP32_SWEEPS = 12;
constexpr double JS_MAX_D = 1e-3;      // largest |D (I - J^H J) D^-1|_F: 63/256 of its fifth power = 2.5e-16
constexpr float JS_MAX_T1 = 0.05f;     // largest |D T D^-1|_F of the first step: 231/1024 |T|^12 = 6e-17
constexpr float JS_MAX_T2 = 6e-4f;     // of the second: 3/8 |T|^5 = 3e-17
constexpr float JS_MAX_T3 = 5e-6f;     // of the third: |T|^3 / 2 = 6e-17
// flagged sweeps: they rotate a few pairs at the rounding level
constexpr int JS_FLAG_SWEEPS = 2;
constexpr int JS_THREADS = 512;

bool jacobi_precondition_ok(int N) { return N >= JS_MIN_N && N <= JS_MAX_N && tc_fp64_ok(N); }

// The FP32 Jacobi's units: |R(0, 0)| (the pivoted R's largest entry) between 2^54
// and 2^55, so that squared norms lie below 256 * 2^110 and columns down to 1e-33
// of the largest still rotate (the squares of 3e-17 of it, in units of R(0, 0),
// already near FP32's underflow: order-15 HELS then keeps hundreds of unrotated
// pairs at the rounding level).  1 for a zero or non-finite R(0, 0).
__device__ __forceinline__ double js_scale(const double2 *R)
{
    const double a = fmax(fabs(R[0].x), fabs(R[0].y));
    const int e = (int)((__double_as_longlong(a) >> 52) & 0x7FF);
    return e > 0 && e < 0x7FF ? ldexp(1.0, min(1022 + 55 - e, 1023)) : 1.0;
}

// exponent of the largest component of a column held by a warp (biased exponents
// in, this lane's largest): its size as a power of two; 0 for zero and non-finite
// columns
__device__ __forceinline__ int js_column_exponent(int e)
{
    for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    return e == 0 || e == 0x7FF ? 0 : min(max(e - 1023, -1000), 1000);
}
__device__ __forceinline__ int js_biased_exponent(double2 v)
{
    return max((__double2hiint(v.x) >> 20) & 0x7FF, (__double2hiint(v.y) >> 20) & 0x7FF);
}

// Y (N x N FP32) = R's first N rows in the FP32 Jacobi's units, M = R D^-1, E the
// exponents of D.  A warp per column.
__global__ void js_init_kernel(int ld, int N, const double2 *__restrict__ R, float2 *__restrict__ Y,
                               double2 *__restrict__ M, int *__restrict__ E)
{
    const int f = blockIdx.y, lane = threadIdx.x & 31, j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (j >= N) return;
    R += (size_t)f * ld * N;
    const double sc = js_scale(R);
    R += (size_t)j * ld;
    Y += ((size_t)f * N + j) * N;
    M += ((size_t)f * N + j) * N;
    int e = 0;
    for (int i = lane; i < N; i += 32) {
        const double2 v = R[i];
        Y[i] = make_float2((float)(v.x * sc), (float)(v.y * sc));
        e = max(e, js_biased_exponent(v));
    }
    e = js_column_exponent(e);
    const double d = ldexp(1.0, -e);
    for (int i = lane; i < N; i += 32) M[i] = zscale(R[i], d);
    if (lane == 0) E[(size_t)f * N + j] = e;
}

// J = D X D^-1, Jt = D^-1 X D (both from the FP32 X)
__global__ void js_widen_kernel(int N, const float2 *__restrict__ X, const int *__restrict__ E,
                                double2 *__restrict__ J, double2 *__restrict__ Jt)
{
    const int f = blockIdx.y;
    const size_t o = (size_t)f * N * N;
    E += (size_t)f * N;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N * N; e += gridDim.x * blockDim.x) {
        const int c = e / N, r = e - c * N, s = min(max(E[r] - E[c], -1000), 1000);
        const double2 v = make_double2((double)X[o + e].x, (double)X[o + e].y);
        J[o + e] = zscale(v, __hiloint2double((1023 + s) << 20, 0));
        Jt[o + e] = zscale(v, __hiloint2double((1023 - s) << 20, 0));
    }
}

__device__ __forceinline__ double js_block_sum(double v, double *red)
{
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < JS_THREADS / 32; ++w) t += red[w];
    __syncthreads();
    return t;
}

// E = D J^H J D^-1 -> I - E; a bin where that is too large (or not a number) gets
// J = I, E = 0.  One CTA per bin.
__global__ void __launch_bounds__(JS_THREADS) js_defect_kernel(int N, double2 *E, double2 *J)
{
    __shared__ double red[JS_THREADS / 32];
    const int f = blockIdx.x;
    E += (size_t)f * N * N;
    J += (size_t)f * N * N;
    double s = 0.0;
    for (int e = threadIdx.x; e < N * N; e += JS_THREADS) {
        const int c = e / N, r = e - c * N;
        double2 d = E[e];
        d = make_double2((r == c ? 1.0 : 0.0) - d.x, -d.y);
        E[e] = d;
        s += zabs2(d);
    }
    s = js_block_sum(s, red);
    if (s <= JS_MAX_D * JS_MAX_D) return;
    for (int e = threadIdx.x; e < N * N; e += JS_THREADS) {
        const int c = e / N, r = e - c * N;
        E[e] = make_double2(0.0, 0.0);
        J[e] = make_double2(r == c ? 1.0 : 0.0, 0.0);
    }
}

// Z = a X + b Y
__global__ void js_combine_kernel(size_t count, double a, const double2 *__restrict__ X, double b, const double2 *Y,
                                  double2 *Z)
{
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x)
        Z[e] = make_double2(fma(a, X[e].x, b * Y[e].x), fma(a, X[e].y, b * Y[e].y));
}

// 1 / x to ~20 bits (T only has to be accurate to the couplings it leaves)
__device__ __forceinline__ double js_rcp(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

// Columns scaled by powers of two to a largest component in [1, 2): X <- X D^-1,
// E += the exponents of D.  A warp per column.
__global__ void js_normalize_kernel(int N, double2 *__restrict__ X, int *__restrict__ E)
{
    const int f = blockIdx.y, lane = threadIdx.x & 31, j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (j >= N) return;
    X += ((size_t)f * N + j) * N;
    int e = 0;
    for (int i = lane; i < N; i += 32) e = max(e, js_biased_exponent(X[i]));
    e = js_column_exponent(e);
    const double sc = ldexp(1.0, -e);
    for (int i = lane; i < N; i += 32) X[i] = zscale(X[i], sc);
    if (lane == 0) E[(size_t)f * N + j] += e;
}

// X <- X D
__global__ void js_unscale_kernel(int N, double2 *__restrict__ X, const int *__restrict__ E)
{
    const int f = blockIdx.y, lane = threadIdx.x & 31, j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (j >= N) return;
    X += ((size_t)f * N + j) * N;
    const double sc = ldexp(1.0, E[(size_t)f * N + j]);
    for (int i = lane; i < N; i += 32) X[i] = zscale(X[i], sc);
}

// G = (M D^-1)^H (M D^-1) -> D T D^-1 in place, T_ij = (D G D)_ij / ((D G D)_jj -
// (D G D)_ii) anti-Hermitian (each pair is computed once).  The larger of the pair's
// two entries, t = G_ij max(d_i, d_j)^2 / ((D G D)_jj - (D G D)_ii), is kept where
// |t| <= theta, the largest of 5e-2, 1e-2 .. 1e-7 with |D T D^-1|_F <= limit; the
// other is -conj(t) times the squared ratio of the sizes.  One CTA per bin.
constexpr int JS_NT = 7;
__host__ __device__ constexpr float js_theta2(int q)
{
    return q == 0 ? 2.5e-3f : q == 1 ? 1e-4f : q == 2 ? 1e-6f : q == 3 ? 1e-8f : q == 4 ? 1e-10f : q == 5 ? 1e-12f : 1e-14f;
}

__global__ void __launch_bounds__(JS_THREADS) js_rotation_kernel(int N, float limit, const int *E, double2 *G)
{
    extern __shared__ double js_g[];   // N: diag(D G D); N: d; N: 1 / d, relative to the largest d
    double *w = js_g + N, *wi = w + N;
    __shared__ float red[JS_NT][JS_THREADS / 32];
    __shared__ int s_emax;
    const int f = blockIdx.x;
    G += (size_t)f * N * N;
    E += (size_t)f * N;
    if (threadIdx.x == 0) s_emax = -4000;
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += JS_THREADS) atomicMax(&s_emax, E[i]);
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += JS_THREADS) {
        w[i] = ldexp(1.0, E[i] - s_emax);
        wi[i] = ldexp(1.0, s_emax - E[i]);
        js_g[i] = G[i + (size_t)i * N].x * w[i] * w[i];
    }
    __syncthreads();
    // |T_ij|^2 and its sums in FP32: they only choose theta (below 1e-19 they
    // underflow, and count as nothing)
    auto size2 = [](double2 t) { const float x = (float)t.x, y = (float)t.y; return x * x + y * y; };
    float s[JS_NT];
#pragma unroll
    for (int q = 0; q < JS_NT; ++q) s[q] = 0.f;
    for (int e = threadIdx.x; e < N * N; e += JS_THREADS) {
        const int j = e / N, i = e - j * N;
        if (i >= j) continue;
        const double2 g = G[e];
        const double d = fmax(w[i], w[j]), q = js_rcp(js_g[j] - js_g[i]) * (d * d);
        const double2 t = make_double2(g.x * q, g.y * q);
        const float m = size2(t);
        // a zero gap, a NaN and an infinity fail every comparison
        if (m <= js_theta2(0)) {
            G[e] = t;
#pragma unroll
            for (int k = 0; k < JS_NT; ++k)
                if (m <= js_theta2(k)) s[k] += m;
        } else {
            G[e] = make_double2(0.0, 0.0);
        }
    }
    float keep = -1.f;   // largest |T_ij|^2 kept
#pragma unroll
    for (int q = 0; q < JS_NT; ++q) {
        float v = s[q];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < JS_NT; ++q) {
        float t = 0.f;
        for (int v = 0; v < JS_THREADS / 32; ++v) t += red[q][v];
        if (keep < 0.f && 2.f * t <= limit * limit) keep = js_theta2(q);
    }
    for (int e = threadIdx.x; e < N * N; e += JS_THREADS) {
        const int j = e / N, i = e - j * N;
        if (i > j) continue;
        if (i == j) {
            G[e] = make_double2(0.0, 0.0);
            continue;
        }
        double2 t = G[e];
        if (!(size2(t) <= keep)) t = make_double2(0.0, 0.0);
        const bool up = w[i] >= w[j];
        const double u = up ? w[j] * wi[i] : w[i] * wi[j];
        const double2 small = zscale(t, u * u);
        G[e] = up ? t : small;
        const double2 o = up ? small : t;
        G[j + (size_t)i * N] = make_double2(-o.x, o.y);
    }
}

// The FP64 Jacobi's test on every pair, from G = M^H M: flags[i + j N] (i < j) for
// a pair to rotate, done[f] when there is none.  One CTA per bin.
__global__ void __launch_bounds__(JS_THREADS) js_flags_kernel(int N, double tol, const double2 *G,
                                                              unsigned char *flags, int *done)
{
    extern __shared__ double js_g[];   // N: column norms
    const int f = blockIdx.x;
    G += (size_t)f * N * N;
    flags += (size_t)f * N * N;
    for (int i = threadIdx.x; i < N; i += JS_THREADS) js_g[i] = sqrt(G[i + (size_t)i * N].x);
    __syncthreads();
    int any = 0;
    for (int e = threadIdx.x; e < N * N; e += JS_THREADS) {
        const int j = e / N, i = e - j * N;
        const double b = tol * js_g[i] * js_g[j];
        const bool rot = i < j && zabs2(G[e]) > b * b;
        flags[e] = rot ? 1 : 0;
        any |= rot ? 1 : 0;
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) done[f] = !any;
}

size_t jacobi_precondition_ws_bytes(int N, int batch)
{
    const size_t nn = (size_t)N * N * batch;
    const size_t prod = zgemm_tc_ws_bytes(N, N, N, batch), start = jacobi_start_ws_bytes(N, JS_FP32_SWEEPS, batch);
    return 5 * ws_round(16 * nn) + ws_round(nn) + ws_round(4 * (size_t)N * batch) + (prod > start ? prod : start) + 2048;
}

int jacobi_precondition_batched(ia_context *ctx, int N, const double2 *R, int ldr, double2 *M, int *done, int batch,
                                int *info, WsCursor cur)
{
    const long long nn = (long long)N * N;
    const size_t count = (size_t)nn * batch;
    float2 *Y = cur.take<float2>(2 * count);
    double2 *J = cur.take<double2>(count), *D = cur.take<double2>(count), *Q = cur.take<double2>(count),
            *P = cur.take<double2>(count);
    unsigned char *flags = cur.take<unsigned char>(count);
    int *E = cur.take<int>((size_t)N * batch);
    if (cur.off > cur.cap) return IA_ERR_ALLOC;
    int st;
    int blocks = (int)((nn + 255) / 256);
    if (blocks > 64) blocks = 64;
    const dim3 grid(blocks, batch), cols((N + 7) / 8, batch);
    const size_t want = (count + 255) / 256, cap = (size_t)ctx->sm_count * 8;
    const int flat = (int)(want < cap ? want : cap);
    // C = op(A) B + beta C, N x N
    auto prod = [&](Op opa, const double2 *A, const double2 *B, double beta, double2 *C) {
        return zgemm_tc(ctx, opa, OP_N, N, N, N, 1.0, A, N, nn, B, N, nn, beta, C, N, nn, batch, info, cur);
    };
    auto combine = [&](double a, const double2 *X, double b, const double2 *Z, double2 *W) -> int {
        js_combine_kernel<<<flat, 256, 0, ctx->stream>>>(count, a, X, b, Z, W);
        IA_LAUNCH_CHECK(ctx);
        return IA_OK;
    };
    js_init_kernel<<<cols, 256, 0, ctx->stream>>>(ldr, N, R, Y, M, E);
    IA_LAUNCH_CHECK(ctx);
    if ((st = jacobi_start_batched(ctx, N, Y, Y + count, batch, JS_FP32_SWEEPS, cur))) return st;
    js_widen_kernel<<<grid, 256, 0, ctx->stream>>>(N, Y + count, E, J, P);
    IA_LAUNCH_CHECK(ctx);
    // J to its polar factor, M = R J
    double2 *S = reinterpret_cast<double2 *>(Y);   // (Y and J in FP32: N^2 FP64 pairs)
    if ((st = prod(OP_C, P, J, 0.0, D))) return st;
    js_defect_kernel<<<batch, JS_THREADS, 0, ctx->stream>>>(N, D, J);
    IA_LAUNCH_CHECK(ctx);
    if ((st = prod(OP_N, D, D, 0.0, Q))) return st;
    if ((st = combine(0.5, D, 0.375, Q, P))) return st;
    if ((st = combine(0.3125, D, 35.0 / 128.0, Q, S))) return st;
    if ((st = prod(OP_N, Q, S, 1.0, P))) return st;
    if ((st = prod(OP_N, J, P, 1.0, J))) return st;
    if ((st = prod(OP_N, M, J, 0.0, M))) return st;
    const size_t nsm = sizeof(double) * (size_t)N;
    // T of M, on M with its columns scaled
    auto rotation = [&](float limit) -> int {
        js_normalize_kernel<<<cols, 256, 0, ctx->stream>>>(N, M, E);
        IA_LAUNCH_CHECK(ctx);
        if ((st = prod(OP_C, M, M, 0.0, D))) return st;
        js_rotation_kernel<<<batch, JS_THREADS, 3 * nsm, ctx->stream>>>(N, limit, E, D);
        IA_LAUNCH_CHECK(ctx);
        return IA_OK;
    };
    // first step: p = (I - T^2)^(-1/2) - I to (T^2)^5, P = T + p + T p
    if ((st = rotation(JS_MAX_T1))) return st;
    {
        // D = T, Q = T^2, J = T^4, P = T^6, then P = 5/16 Q + 35/128 J + 63/256 P
        double2 *T = D;
        if ((st = prod(OP_N, T, T, 0.0, Q))) return st;
        if ((st = prod(OP_N, Q, Q, 0.0, J))) return st;
        if ((st = prod(OP_N, Q, J, 0.0, P))) return st;
        if ((st = combine(35.0 / 128.0, J, 63.0 / 256.0, P, P))) return st;
        if ((st = combine(5.0 / 16.0, Q, 1.0, P, P))) return st;
        if ((st = combine(0.5, Q, 0.375, J, S))) return st;
        if ((st = prod(OP_N, J, P, 1.0, S))) return st;      // p
        if ((st = combine(1.0, T, 1.0, S, P))) return st;
        if ((st = prod(OP_N, T, S, 1.0, P))) return st;
        if ((st = prod(OP_N, M, P, 1.0, M))) return st;
    }
    // second step: P = T + T^2 / 2 + T^2 (T / 2 + 3 T^2 / 8)
    if ((st = rotation(JS_MAX_T2))) return st;
    if ((st = prod(OP_N, D, D, 0.0, Q))) return st;
    if ((st = combine(0.5, D, 0.375, Q, J))) return st;
    if ((st = combine(1.0, D, 0.5, Q, P))) return st;
    if ((st = prod(OP_N, Q, J, 1.0, P))) return st;
    if ((st = prod(OP_N, M, P, 1.0, M))) return st;
    // third step: P = T + T^2 / 2
    if ((st = rotation(JS_MAX_T3))) return st;
    if ((st = prod(OP_N, D, D, 0.0, Q))) return st;
    if ((st = combine(1.0, D, 0.5, Q, P))) return st;
    if ((st = prod(OP_N, M, P, 1.0, M))) return st;
    js_unscale_kernel<<<cols, 256, 0, ctx->stream>>>(N, M, E);
    IA_LAUNCH_CHECK(ctx);
    // sweeps over the pairs above the test
    for (int it = 0; it < JS_FLAG_SWEEPS; ++it) {
        if ((st = prod(OP_C, M, M, 0.0, D))) return st;
        js_flags_kernel<<<batch, JS_THREADS, nsm, ctx->stream>>>(N, jacobi_tol_fp64(N), D, flags, done);
        IA_LAUNCH_CHECK(ctx);
        if ((st = jacobi_flagged_batched(ctx, N, M, batch, done, flags))) return st;
    }
    return IA_OK;
}

}  // namespace ia
