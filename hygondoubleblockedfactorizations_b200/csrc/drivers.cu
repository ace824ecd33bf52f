// Host-side building blocks: recursive diagonal Cholesky, recursive TRSMs,
// SYRK, recursive GETRF panel.  Everything is enqueued on ctx->stream; no
// host synchronisation.
#include <algorithm>

#include "internal.h"

namespace hdbf {

namespace {
constexpr int kDiagLeaf = 64;   // potf2_small / trsm_*_small leaf order
constexpr int kClusterLeaf = 32;  // leaf width when the cluster panel kernel is forced

// Split point for a recursion on `n` columns with `leaf`-aligned halves.
inline int split_at(int n, int leaf)
{
    int h = (n / 2 + leaf - 1) / leaf * leaf;
    if (h <= 0 || h >= n) h = std::max(1, n - leaf);
    return h;
}
}  // namespace

hdbf_status potrf_diag(hdbf_context* ctx, int n, float* A, long long lda, int* info,
                       int info_base, bool last)
{
    if (n <= 0) return HDBF_STATUS_SUCCESS;
    HDBF_TRY(ensure_ws(ctx, n));
    if (n <= kDiagLeaf)
        return potf2_small(ctx, n, A, lda, info, info_base, last ? nullptr : ws_inv(ctx));
    if (n <= potrf_block_max_n())
        return potrf_block(ctx, n, A, lda, info, info_base, nullptr, 0, last);
    const int n1 = split_at(n, kDiagLeaf);
    const int n2 = n - n1;
    float* A21 = A + n1;
    float* A22 = A + (long long)n1 * lda + n1;
    HDBF_TRY(potrf_diag(ctx, n1, A, lda, info, info_base, false));
    HDBF_TRY(trsm_rlt_ready(ctx, n2, n1, A, lda, A21, lda));
    HDBF_TRY(syrk_lower(ctx, n2, n1, A21, lda, A22, lda));
    return potrf_diag(ctx, n2, A22, lda, info, info_base + n1, last);
}

namespace {
// Recursive right/lower/transposed solve with precomputed 64x64 block inverses
// (inv holds the blocks of L starting at block `blk`).
hdbf_status trsm_rlt_rec(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                         float* B, long long ldb, const float* inv)
{
    if (cols <= llu_block_max_rows()) return rlt_block(ctx, rows, cols, L, ldl, inv, B, ldb);
    const int c1 = split_at(cols, kDiagLeaf);
    const int c2 = cols - c1;
    HDBF_TRY(trsm_rlt_rec(ctx, rows, c1, L, ldl, B, ldb, inv));
    // B2 -= X1 * L21^T, L21 = L(c1:cols, 0:c1)
    HDBF_TRY(sgemm_sub(ctx, false, false, rows, c2, c1, B, ldb, L + c1, ldl,
                       B + (long long)c1 * ldb, ldb));
    return trsm_rlt_rec(ctx, rows, c2, L + (long long)c1 * ldl + c1, ldl,
                        B + (long long)c1 * ldb, ldb, inv + (long long)(c1 / kDiagLeaf) * 4096);
}

hdbf_status trsm_llu_rec(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                         float* B, long long ldb, const float* inv)
{
    if (rows <= llu_block_max_rows()) return llu_block(ctx, rows, cols, L, ldl, inv, B, ldb);
    const int r1 = split_at(rows, kDiagLeaf);
    const int r2 = rows - r1;
    HDBF_TRY(trsm_llu_rec(ctx, r1, cols, L, ldl, B, ldb, inv));
    // B2 -= L21 * X1
    HDBF_TRY(sgemm_sub(ctx, true, false, r2, cols, r1, L + r1, ldl, B, ldb, B + r1, ldb));
    return trsm_llu_rec(ctx, r2, cols, L + (long long)r1 * ldl + r1, ldl, B + r1, ldb,
                        inv + (long long)(r1 / kDiagLeaf) * 4096);
}
}  // namespace

// B(rows x cols) <- B * L^{-T}: invert the 64x64 diagonal blocks of L once,
// then recurse on column halves with GEMM updates; leaves are small GEMMs
// with the inverted blocks (no serial dependency chains).
hdbf_status trsm_rlt(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                     float* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    HDBF_TRY(ensure_ws(ctx, cols));
    float* inv = ws_inv(ctx);
    HDBF_TRY(tri_inv64(ctx, cols, L, ldl, false, inv));
    return trsm_rlt_rec(ctx, rows, cols, L, ldl, B, ldb, inv);
}

hdbf_status trsm_rlt_ready(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                           float* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    // The recursion of a larger diagonal block reuses the inverse table.
    if (cols > potrf_block_max_n()) return trsm_rlt(ctx, rows, cols, L, ldl, B, ldb);
    return trsm_rlt_rec(ctx, rows, cols, L, ldl, B, ldb, ws_inv(ctx));
}

// B(rows x cols) <- L^{-1} B, L unit lower, same scheme on row halves.
hdbf_status trsm_llu(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                     float* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    HDBF_TRY(ensure_ws(ctx, rows));
    float* inv = ws_inv(ctx);
    HDBF_TRY(tri_inv64(ctx, rows, L, ldl, true, inv));
    return trsm_llu_rec(ctx, rows, cols, L, ldl, B, ldb, inv);
}

hdbf_status syrk_lower(hdbf_context* ctx, int n, int k, const float* A, long long lda,
                       float* C, long long ldc)
{
    return sgemm_sub(ctx, false, true, n, n, k, A, lda, A, lda, C, ldc);
}

hdbf_status getrf_workspace(hdbf_context* ctx, int n, GetrfWs* ws)
{
    HDBF_TRY(ensure_ws(ctx, n));
    ws->src = ws_src(ctx);
    ws->tgt = ws_tgt(ctx);
    ws->gperm = ws_gperm(ctx);
    ws->temp = ws_temp(ctx);
    ws->temp_cols = 64;
    ws->count = ctx->dev_small + kSmallMoveCount;
    return HDBF_STATUS_SUCCESS;
}

// A part's interchanges on columns [c0, c0 + nc) of its rows.
template <class T>
static hdbf_status panel_swaps_t(hdbf_context* ctx, T* A, long long lda, const int* ipiv, int k,
                                 int ipiv_add, int m, int c0, int nc, int* info, const GetrfWs& ws)
{
    const hdbf_status st = swap_rows(ctx, A, lda, ipiv, k, ipiv_add, m, c0, nc, 0, 0, info);
    if (st != HDBF_STATUS_NOT_SUPPORTED) return st;
    HDBF_TRY(compose_swaps(ctx, ipiv, k, ipiv_add, m, ws.src, ws.tgt, ws.count, ws.gperm, info));
    return apply_moves(ctx, A + (long long)c0 * lda, lda, nc, ws.src, ws.tgt, ws.count,
                       std::min(m, 2 * k), reinterpret_cast<T*>(ws.temp), ws.temp_cols);
}
hdbf_status panel_swaps(hdbf_context* ctx, float* A, long long lda, const int* ipiv, int k,
                        int ipiv_add, int m, int c0, int nc, int* info, const GetrfWs& ws)
{
    return panel_swaps_t(ctx, A, lda, ipiv, k, ipiv_add, m, c0, nc, info, ws);
}
hdbf_status panel_swaps(hdbf_context* ctx, double* A, long long lda, const int* ipiv, int k,
                        int ipiv_add, int m, int c0, int nc, int* info, const GetrfWs& ws)
{
    return panel_swaps_t(ctx, A, lda, ipiv, k, ipiv_add, m, c0, nc, info, ws);
}

// Leaf width for the cluster panel kernel at height m, 0 for the grid-wide one.
// The cluster has the cheaper columns while a thread has one row (512 threads a
// CTA, m <= 8192): 1.3-1.8 us against the grid's 1.9-2.0 us.  Above, its columns
// cost as much or more (2.4 and 4.6 us at m = 16384 and 30000) and its leaves
// narrow to 64 columns and fewer, each merge of two (swaps, TRSM, GEMM) ~40 us more.
// FP32 LU: leaves of 256 bytes up to m = 13300 / up to 8192 / none: n = 8192 25.4 /
// 25.4 / 25.6 ms, n = 32768 260.3 / 257-259 / 257.4 ms.
int panel_cluster_leaf(hdbf_context* ctx, int m, int elem)
{
    if (ctx->panel_mode == 1) return 0;
    const int leaf = getf2_cluster_leaf(ctx, m, elem);
    if (ctx->panel_mode == 2 || leaf * elem >= 512) return leaf;
    return leaf * elem >= 256 && m <= 512 * ctx->cluster_max ? leaf : 0;
}

// Recursive (Toledo/Gustavson) LU of an m x w panel.  A leaf is as wide as one
// cluster can hold at this height, or the grid above that and where the grid-wide
// kernel is forced, at most the handle's panel-leaf width (32 when the cluster
// kernel is forced).  ipiv
// receives (local row + 1 + ipiv_add) for the panel's w columns.
hdbf_status getrf_panel(hdbf_context* ctx, int m, int w, float* A, long long lda, int* ipiv,
                        int ipiv_add, int* info, int info_base, bool pivot, const GetrfWs& ws)
{
    if (m <= 0 || w <= 0) return HDBF_STATUS_SUCCESS;
    const int held = panel_cluster_leaf(ctx, m, (int)sizeof(float));
    const int widest = ctx->panel_mode == 2 ? kClusterLeaf : ctx->panel_leaf;
    const int leaf =
        std::min(held > 0 ? held : getf2_grid_leaf(ctx, m, (int)sizeof(float)), widest);
    if (leaf < 1) return HDBF_STATUS_NOT_SUPPORTED;
    if (w <= leaf) {
        if (held > 0) return getf2_cluster(ctx, m, w, A, lda, ipiv, ipiv_add, info, info_base, pivot);
        return getf2_grid(ctx, m, w, A, lda, ipiv, ipiv_add, info, info_base, pivot);
    }
    const int w1 = split_at(w, leaf);
    const int w2 = w - w1;
    HDBF_TRY(getrf_panel(ctx, m, w1, A, lda, ipiv, ipiv_add, info, info_base, pivot, ws));
    float* A12 = A + (long long)w1 * lda;
    if (pivot)
        HDBF_TRY(panel_swaps(ctx, A, lda, ipiv, w1, ipiv_add, m, w1, w2, info, ws));
    HDBF_TRY(trsm_llu(ctx, w1, w2, A, lda, A12, lda));
    HDBF_TRY(sgemm_sub(ctx, true, false, m - w1, w2, w1, A + w1, lda, A12, lda, A12 + w1, lda));
    HDBF_TRY(getrf_panel(ctx, m - w1, w2, A12 + w1, lda, pivot ? ipiv + w1 : nullptr,
                         ipiv_add + w1, info, info_base + w1, pivot, ws));
    if (pivot)
        HDBF_TRY(panel_swaps(ctx, A + w1, lda, ipiv + w1, w2, ipiv_add + w1, m - w1, 0, w1, info, ws));
    return HDBF_STATUS_SUCCESS;
}

}  // namespace hdbf
