// FP64 building blocks behind the reference's `_double` entry points
// (include/potrf/double_blocked_potrf.h:57-103, include/getrf/
// double_blocked_getrf.h:37-74 and the SYRK / TRSM / GEMM twins).  The
// drivers in api_potrf.cu and api_getrf.cu are templates over the scalar
// type; this file gives them the FP64 overloads of their primitives:
//
//   gemm_sub / gemm_sub_tn   C -= op(A) op(B), FP64 FMA: 128x128x8 tiles with
//                            8x8 outputs per thread for large updates, the
//                            small-update kernel (gemm_small.cu) below, 64x64x16
//                            tiles for TN; lower-triangle mode
//   trsm_rlt / trsm_llu      recursive TRSMs on the leaves of trsm_block.cu
//                            (diagonal tiles and inverses: panel_kernels.cu)
//   potrf_diag, syrk_lower   recursive diagonal Cholesky, lower SYRK
//   getrf_panel              recursive LU panel on the leaves of getf2_cluster.cu
//                            and getf2_grid.cu
//   apply_moves              composed row moves, gathered through scratch
#include <algorithm>
#include <cfloat>
#include <climits>

#include "internal.h"

namespace hdbf {
namespace {

constexpr int kL = 64;  // leaf / diagonal-block order

inline int split64(int n)
{
    int h = (n / 2 + kL - 1) / kL * kL;
    if (h <= 0 || h >= n) h = std::max(1, n - kL);
    return h;
}

// ------------------------------------------------------------------ GEMM
// Large updates: 128x128x8 tiles, 256 threads, 8x8 outputs per thread in the split layout
// (rows ty*4 + {0..3} and 64 + ty*4 + {0..3}, columns likewise with tx), so
// every fragment is two 16-byte shared-memory loads; the next k-tile is
// copied into the other shared-memory buffer with 8-byte cp.async (zero fill
// outside the matrix) while the current one is consumed.
constexpr int GBM = 128, GBN = 128, GBK = 8, GTHR = 256, GLD = GBM + 4;

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem, bool valid)
{
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(s), "l"(gmem),
                 "r"(valid ? 8 : 0)
                 : "memory");
}

// MODE 0: C -= A B^T (A M x K, B N x K); 1: C -= A B (B K x N);
// 2: C -= A^T B (A stored K x M, B K x N).  TRI: only entries with row >= col
// (local to C) are written and tiles wholly above the diagonal are skipped.
template <int MODE, bool TRI>
__global__ void __launch_bounds__(GTHR, 1) dgemm_sub_kernel(int M, int N, int K,
                                                            const double* __restrict__ A,
                                                            long long lda,
                                                            const double* __restrict__ B,
                                                            long long ldb, double* C,
                                                            long long ldc, int tiles_m)
{
    __shared__ __align__(16) double As[2][GBK][GLD];  // As[buf][k][m]
    __shared__ __align__(16) double Bs[2][GBK][GLD];  // Bs[buf][k][n]
    const int tile = blockIdx.x;
    const int m0 = (tile % tiles_m) * GBM, n0 = (tile / tiles_m) * GBN;
    if (TRI && n0 >= m0 + GBM) return;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    double acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0;
    auto issue = [&](int buf, int k0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int q = tid + e * GTHR;
            int m, k;
            if (MODE == 2) { k = q & 7; m = q >> 3; }
            else { m = q & 127; k = q >> 7; }
            const int gm = m0 + m, gk = k0 + k;
            const bool va = gm < M && gk < K;
            const double* pa =
                va ? (MODE == 2 ? A + (long long)gm * lda + gk : A + (long long)gk * lda + gm) : A;
            cp_async8(&As[buf][k][m], pa, va);
            int nn, kk;
            if (MODE == 0) { nn = q & 127; kk = q >> 7; }
            else { kk = q & 7; nn = q >> 3; }
            const int gn = n0 + nn, gk2 = k0 + kk;
            const bool vb = gn < N && gk2 < K;
            const double* pb =
                vb ? (MODE == 0 ? B + (long long)gk2 * ldb + gn : B + (long long)gn * ldb + gk2)
                   : B;
            cp_async8(&Bs[buf][kk][nn], pb, vb);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int nk = (K + GBK - 1) / GBK;
    issue(0, 0);
    for (int kt = 0; kt < nk; ++kt) {
        const int cur = kt & 1;
        if (kt + 1 < nk) issue(cur ^ 1, (kt + 1) * GBK);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GBK; ++k) {
            double a[8], b[8];
            const double2* ap = reinterpret_cast<const double2*>(&As[cur][k][ty * 4]);
            const double2* ap2 = reinterpret_cast<const double2*>(&As[cur][k][64 + ty * 4]);
            const double2* bp = reinterpret_cast<const double2*>(&Bs[cur][k][tx * 4]);
            const double2* bp2 = reinterpret_cast<const double2*>(&Bs[cur][k][64 + tx * 4]);
            const double2 a0 = ap[0], a1 = ap[1], a2 = ap2[0], a3 = ap2[1];
            const double2 b0 = bp[0], b1 = bp[1], b2 = bp2[0], b3 = bp2[1];
            a[0] = a0.x; a[1] = a0.y; a[2] = a1.x; a[3] = a1.y;
            a[4] = a2.x; a[5] = a2.y; a[6] = a3.x; a[7] = a3.y;
            b[0] = b0.x; b[1] = b0.y; b[2] = b1.x; b[3] = b1.y;
            b[4] = b2.x; b[5] = b2.y; b[6] = b3.x; b[7] = b3.y;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int c = n0 + (j < 4 ? tx * 4 + j : 64 + tx * 4 + (j - 4));
        if (c >= N) continue;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + (i - 4));
            if (r < M && (!TRI || r >= c)) C[(long long)c * ldc + r] -= acc[i][j];
        }
    }
}

template <int MODE, bool TRI>
void dgemm_launch(cudaStream_t s, int M, int N, int K, const double* A, long long lda,
                  const double* B, long long ldb, double* C, long long ldc)
{
    const int tm = (M + GBM - 1) / GBM, tn = (N + GBN - 1) / GBN;
    dgemm_sub_kernel<MODE, TRI><<<(unsigned)((long long)tm * tn), GTHR, 0, s>>>(
        M, N, K, A, lda, B, ldb, C, ldc, tm);
}

// 64x64x16 tiles, 4x4 outputs per thread, register-staged prefetch: the
// tall, narrow updates of the panels and TRSM recursions (more CTAs).
constexpr int SBM = 64, SBN = 64, SBK = 16, STHR = 256;

// MODE 0: C -= A B^T (A M x K, B N x K); 1: C -= A B (B K x N);
// 2: C -= A^T B (A stored K x M, B K x N).  TRI: only entries with row >= col
// (local to C) are written and tiles wholly above the diagonal are skipped.
template <int MODE, bool TRI>
__global__ void __launch_bounds__(STHR) dgemm_sub64_kernel(int M, int N, int K,
                                                         const double* __restrict__ A,
                                                         long long lda,
                                                         const double* __restrict__ B,
                                                         long long ldb, double* C, long long ldc,
                                                         int tiles_m)
{
    __shared__ double As[SBK][SBM + 1];
    __shared__ double Bs[SBK][SBN + 1];
    const int tile = blockIdx.x;
    const int m0 = (tile % tiles_m) * SBM, n0 = (tile / tiles_m) * SBN;
    if (TRI && n0 >= m0 + SBM) return;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    double ra[4], rb[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int q = tid + e * STHR;
            int m, k;
            if (MODE == 2) { k = q & 15; m = q >> 4; }
            else { m = q & 63; k = q >> 6; }
            const int gm = m0 + m, gk = k0 + k;
            double v = 0.0;
            if (gm < M && gk < K)
                v = MODE == 2 ? A[(long long)gm * lda + gk] : A[(long long)gk * lda + gm];
            ra[e] = v;
            int nn, kk;
            if (MODE == 0) { nn = q & 63; kk = q >> 6; }
            else { kk = q & 15; nn = q >> 4; }
            const int gn = n0 + nn, gk2 = k0 + kk;
            double w = 0.0;
            if (gn < N && gk2 < K)
                w = MODE == 0 ? B[(long long)gk2 * ldb + gn] : B[(long long)gn * ldb + gk2];
            rb[e] = w;
        }
    };
    auto stash = [&]() {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int q = tid + e * STHR;
            if (MODE == 2) As[q & 15][q >> 4] = ra[e];
            else As[q >> 6][q & 63] = ra[e];
            if (MODE == 0) Bs[q >> 6][q & 63] = rb[e];
            else Bs[q & 15][q >> 4] = rb[e];
        }
    };
    const int nk = (K + SBK - 1) / SBK;
    fetch(0);
    for (int kt = 0; kt < nk; ++kt) {
        stash();
        __syncthreads();
        if (kt + 1 < nk) fetch((kt + 1) * SBK);
#pragma unroll
        for (int k = 0; k < SBK; ++k) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[k][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = n0 + tx + 16 * j;
        if (c >= N) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = m0 + ty + 16 * i;
            if (r < M && (!TRI || r >= c)) C[(long long)c * ldc + r] -= acc[i][j];
        }
    }
}

template <int MODE, bool TRI>
void dgemm_launch64(cudaStream_t s, int M, int N, int K, const double* A, long long lda,
                  const double* B, long long ldb, double* C, long long ldc)
{
    const int tm = (M + SBM - 1) / SBM, tn = (N + SBN - 1) / SBN;
    dgemm_sub64_kernel<MODE, TRI><<<(unsigned)((long long)tm * tn), STHR, 0, s>>>(
        M, N, K, A, lda, B, ldb, C, ldc, tm);
}

// The small-update kernel's split (gemm_small.cu), or 0 where 64 x 64 x 16 tiles are
// faster.  Both have the same tiles and are bound by the FP64 pipe: the small kernel
// takes 1.17 times as long per step of K (0.075 us), the other 6 us (80 steps) more to
// start, and only the small one splits K.  4096 x 1024 x 1000: 652 us, 544 in 64 x 64 x
// 16 tiles; 2048 x 64 x 512: 27 us, 54.  Tall updates of up to three tile columns and
// one tile per SM are slower in the latter than the steps say (8192 x 64 x 2048: 232
// us, 187; 1536 x 384 x 2048, as many tiles: 177, 187).  Without 16-byte accesses (!vec)
// the small kernel takes 1.25 times as long a step, the other 60 steps more a tile
// (2048 x 2048 x 128 with odd leading dimensions: 109 us, 162).
int small_split64(const hdbf_context* ctx, int M, int N, int K, bool tri, bool vec)
{
    const int S = gemm_small_split(ctx, M, N, K);
    if (S == 0 || (N <= 192 && tile_count(M, N, 64, false) <= ctx->sm_count)) return S;
    const long long kc = ((K + S - 1) / S + 7) / 8 * 8;
    const double small = (vec ? 1.17 : 1.25) * (double)small_waves(ctx, M, N, tri, S) * kc;
    const double other = (double)small_waves(ctx, M, N, tri, 1) * (vec ? K : K + 60) + 80.0;
    return small < other ? S : 0;
}

hdbf_status dgemm(hdbf_context* ctx, int mode, bool lower_only, int M, int N, int K,
                  const double* A, long long lda, const double* B, long long ldb, double* C,
                  long long ldc)
{
    if (M <= 0 || N <= 0 || K <= 0) return HDBF_STATUS_SUCCESS;
    if (!A || !B || !C) return HDBF_STATUS_INVALID_VALUE;
    if (lower_only && mode != 0) return HDBF_STATUS_INVALID_VALUE;
    const long long tiles = (long long)((M + SBM - 1) / SBM) * ((N + SBN - 1) / SBN);
    if (tiles > 0x7fffffffLL) return HDBF_STATUS_NOT_SUPPORTED;
    double flops = 2.0 * (double)M * N * K;
    if (lower_only) {
        const double d = (double)(M < N ? M : N);
        flops = 2.0 * (double)K * (d * (double)M - d * (d - 1.0) / 2.0);
    }
    ProfScope prof(ctx, kClsGemm, flops, 8.0 * ((double)M * K + (double)N * K + 2.0 * M * N), M,
                   N, K);
    cudaStream_t s = ctx->stream;
    if (mode != 2) {
        auto even = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
        const bool vec = even(A) && even(B) && lda % 2 == 0 && ldb % 2 == 0;
        const int S = small_split64(ctx, M, N, K, lower_only, vec);
        if (S > 0) return gemm_small(ctx, mode == 1, lower_only, S, M, N, K, A, lda, B, ldb, C, ldc);
    }
    // 128x128 tiles only when they still give two waves of CTAs (one per SM)
    const long long big_tiles = (long long)((M + GBM - 1) / GBM) * ((N + GBN - 1) / GBN);
    if (big_tiles >= 2LL * ctx->sm_count) {
        if (mode == 0) {
            if (lower_only) dgemm_launch<0, true>(s, M, N, K, A, lda, B, ldb, C, ldc);
            else dgemm_launch<0, false>(s, M, N, K, A, lda, B, ldb, C, ldc);
        } else if (mode == 1) {
            dgemm_launch<1, false>(s, M, N, K, A, lda, B, ldb, C, ldc);
        } else {
            dgemm_launch<2, false>(s, M, N, K, A, lda, B, ldb, C, ldc);
        }
    } else if (mode == 0) {
        if (lower_only) dgemm_launch64<0, true>(s, M, N, K, A, lda, B, ldb, C, ldc);
        else dgemm_launch64<0, false>(s, M, N, K, A, lda, B, ldb, C, ldc);
    } else if (mode == 1) {
        dgemm_launch64<1, false>(s, M, N, K, A, lda, B, ldb, C, ldc);
    } else {
        dgemm_launch64<2, false>(s, M, N, K, A, lda, B, ldb, C, ldc);
    }
    ctx->launches++;
    return last_cuda(ctx);
}

// ------------------------------------------------------------- TRSM recursion
hdbf_status trsm_rlt_rec64(hdbf_context* ctx, int rows, int cols, const double* L,
                           long long ldl, double* B, long long ldb, const double* inv)
{
    if (cols <= llu_block_max_rows()) return rlt_block(ctx, rows, cols, L, ldl, inv, B, ldb);
    const int c1 = split64(cols);
    const int c2 = cols - c1;
    HDBF_TRY(trsm_rlt_rec64(ctx, rows, c1, L, ldl, B, ldb, inv));
    HDBF_TRY(dgemm(ctx, 0, false, rows, c2, c1, B, ldb, L + c1, ldl, B + (long long)c1 * ldb,
                   ldb));
    return trsm_rlt_rec64(ctx, rows, c2, L + (long long)c1 * ldl + c1, ldl,
                          B + (long long)c1 * ldb, ldb, inv + (long long)(c1 / kL) * kL * kL);
}

hdbf_status trsm_llu_rec64(hdbf_context* ctx, int rows, int cols, const double* L,
                           long long ldl, double* B, long long ldb, const double* inv)
{
    if (rows <= llu_block_max_rows()) return llu_block(ctx, rows, cols, L, ldl, inv, B, ldb);
    const int r1 = split64(rows);
    const int r2 = rows - r1;
    HDBF_TRY(trsm_llu_rec64(ctx, r1, cols, L, ldl, B, ldb, inv));
    HDBF_TRY(dgemm(ctx, 1, false, r2, cols, r1, L + r1, ldl, B, ldb, B + r1, ldb));
    return trsm_llu_rec64(ctx, r2, cols, L + (long long)r1 * ldl + r1, ldl, B + r1, ldb,
                          inv + (long long)(r1 / kL) * kL * kL);
}

// --------------------------------------------------------------- row moves
// Gather every moved source row of nc columns into scratch, then scatter to
// the targets (sources and targets are the same row set).
__global__ void dgather_rows_kernel(const double* A, long long lda, int nc, const int* src,
                                    const int* count, int cap, double* temp)
{
    const int cnt = min(*count, cap);
    const long long total = (long long)nc * cnt;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(e / cnt), q = (int)(e - (long long)c * cnt);
        temp[(long long)c * cap + q] = A[(long long)c * lda + src[q]];
    }
}

__global__ void dscatter_rows_kernel(double* A, long long lda, int nc, const int* tgt,
                                     const int* count, int cap, const double* temp)
{
    const int cnt = min(*count, cap);
    const long long total = (long long)nc * cnt;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(e / cnt), q = (int)(e - (long long)c * cnt);
        A[(long long)c * lda + tgt[q]] = temp[(long long)c * cap + q];
    }
}

}  // namespace

hdbf_status gemm_sub(hdbf_context* ctx, bool nn, bool lower_only, int M, int N, int K,
                     const double* A, long long lda, const double* B, long long ldb, double* C,
                     long long ldc)
{
    return dgemm(ctx, nn ? 1 : 0, lower_only, M, N, K, A, lda, B, ldb, C, ldc);
}

hdbf_status gemm_sub_tn(hdbf_context* ctx, int M, int N, int K, const double* A, long long lda,
                        const double* B, long long ldb, double* C, long long ldc)
{
    return dgemm(ctx, 2, false, M, N, K, A, lda, B, ldb, C, ldc);
}

hdbf_status trsm_rlt(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                     double* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    HDBF_TRY(ensure_ws(ctx, ws_order<double>(cols)));
    double* inv = reinterpret_cast<double*>(ws_inv(ctx));
    HDBF_TRY(tri_inv64(ctx, cols, L, ldl, false, inv));
    return trsm_rlt_rec64(ctx, rows, cols, L, ldl, B, ldb, inv);
}

hdbf_status trsm_rlt_ready(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                           double* B, long long ldb)
{
    if (cols > kL) return trsm_rlt(ctx, rows, cols, L, ldl, B, ldb);
    return rlt_block(ctx, rows, cols, L, ldl, reinterpret_cast<double*>(ws_inv(ctx)), B, ldb);
}

hdbf_status trsm_llu(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                     double* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    HDBF_TRY(ensure_ws(ctx, ws_order<double>(rows)));
    double* inv = reinterpret_cast<double*>(ws_inv(ctx));
    HDBF_TRY(tri_inv64(ctx, rows, L, ldl, true, inv));
    return trsm_llu_rec64(ctx, rows, cols, L, ldl, B, ldb, inv);
}

hdbf_status syrk_lower(hdbf_context* ctx, int n, int k, const double* A, long long lda,
                       double* C, long long ldc)
{
    return dgemm(ctx, 0, true, n, n, k, A, lda, A, lda, C, ldc);
}

hdbf_status potrf_diag(hdbf_context* ctx, int n, double* A, long long lda, int* info,
                       int info_base, bool last)
{
    if (n <= 0) return HDBF_STATUS_SUCCESS;
    HDBF_TRY(ensure_ws(ctx, ws_order<double>(n)));
    if (n <= kL)
        return potf2_small(ctx, n, A, lda, info, info_base,
                           last ? nullptr : reinterpret_cast<double*>(ws_inv(ctx)));
    const int n1 = split64(n);
    const int n2 = n - n1;
    double* A21 = A + n1;
    double* A22 = A + (long long)n1 * lda + n1;
    HDBF_TRY(potrf_diag(ctx, n1, A, lda, info, info_base, false));
    HDBF_TRY(trsm_rlt_ready(ctx, n2, n1, A, lda, A21, lda));
    HDBF_TRY(syrk_lower(ctx, n2, n1, A21, lda, A22, lda));
    return potrf_diag(ctx, n2, A22, lda, info, info_base + n1, last);
}

hdbf_status apply_moves(hdbf_context* ctx, double* A, long long lda, int ncols, const int* src,
                        const int* tgt, const int* count, int max_moves, double* temp,
                        long long temp_cols)
{
    if (ncols <= 0 || max_moves <= 0) return HDBF_STATUS_SUCCESS;
    if (!temp || temp_cols <= 0) return HDBF_STATUS_INVALID_VALUE;
    ProfScope prof(ctx, kClsMoves, 0.0, 16.0 * (double)max_moves * ncols);
    for (long long c = 0; c < ncols; c += temp_cols) {
        const int nc = (int)((ncols - c) < temp_cols ? (ncols - c) : temp_cols);
        const long long total = (long long)nc * max_moves;
        const int grid = (int)((total + 255) / 256 < 65535 ? (total + 255) / 256 : 65535);
        dgather_rows_kernel<<<grid, 256, 0, ctx->stream>>>(A + c * lda, lda, nc, src, count,
                                                           max_moves, temp);
        dscatter_rows_kernel<<<grid, 256, 0, ctx->stream>>>(A + c * lda, lda, nc, tgt, count,
                                                            max_moves, temp);
        ctx->launches += 2;
    }
    return last_cuda(ctx);
}

// Recursive (Toledo/Gustavson) LU of an m x w FP64 panel; leaves as in the FP32
// panel.
hdbf_status getrf_panel(hdbf_context* ctx, int m, int w, double* A, long long lda, int* ipiv,
                        int ipiv_add, int* info, int info_base, bool pivot, const GetrfWs& ws)
{
    if (m <= 0 || w <= 0) return HDBF_STATUS_SUCCESS;
    const int held = panel_cluster_leaf(ctx, m, (int)sizeof(double));
    const int leaf = held > 0 ? held : getf2_grid_leaf(ctx, m, (int)sizeof(double));
    if (leaf < 1) return HDBF_STATUS_NOT_SUPPORTED;
    if (w <= leaf) {
        if (held > 0) return getf2_cluster(ctx, m, w, A, lda, ipiv, ipiv_add, info, info_base, pivot);
        return getf2_grid(ctx, m, w, A, lda, ipiv, ipiv_add, info, info_base, pivot);
    }
    const int w1 = std::max(leaf, w / 2 / leaf * leaf);
    const int w2 = w - w1;
    HDBF_TRY(getrf_panel(ctx, m, w1, A, lda, ipiv, ipiv_add, info, info_base, pivot, ws));
    double* A12 = A + (long long)w1 * lda;
    if (pivot)
        HDBF_TRY(panel_swaps(ctx, A, lda, ipiv, w1, ipiv_add, m, w1, w2, info, ws));
    HDBF_TRY(trsm_llu(ctx, w1, w2, A, lda, A12, lda));
    HDBF_TRY(dgemm(ctx, 1, false, m - w1, w2, w1, A + w1, lda, A12, lda, A12 + w1, lda));
    HDBF_TRY(getrf_panel(ctx, m - w1, w2, A12 + w1, lda, pivot ? ipiv + w1 : nullptr,
                         ipiv_add + w1, info, info_base + w1, pivot, ws));
    if (pivot)
        HDBF_TRY(panel_swaps(ctx, A + w1, lda, ipiv + w1, w2, ipiv_add + w1, m - w1, 0, w1, info, ws));
    return HDBF_STATUS_SUCCESS;
}

}  // namespace hdbf
