// LAPACK row interchanges of a panel applied to other columns in one launch,
// straight from the pivots (up to 512 swaps), FP32 and FP64.
//
// Replaces apply_panel_pivots_kernel (src/getrf/getrf_pivot_kernels.hip:14-45).
// The panels of the LU recursion swap after every leaf and every merge, so what
// counts is latency: composing the swaps in one launch (sort, scans, one CTA: 12-14
// us) and applying the moves in another (14-25 us) took longer than the arithmetic
// between them.  Here every CTA composes the swaps itself: position x (a
// diagonal row 0 .. k-1, or a pivot row >= k) ends up with the row found by
// undoing the swaps from the last one on, a compare and two selects per swap out
// of shared memory, all 2k positions in parallel.  A pivot row that appears
// several times gets the same row several times.  Then columns move eight at a
// time: every source of a column is read into registers before a barrier, the
// targets are written after it.  128 swaps on 128 columns: 5 us (27 before).
#include <algorithm>

#include "internal.h"

namespace hdbf {
namespace {

constexpr int kMaxSwaps = 512;
constexpr int kThr = 256;
constexpr int kCols = 8;  // columns per pass

template <class T, int NP>
__global__ void __launch_bounds__(kThr)
swap_rows_kernel(T* A, long long lda, const int* __restrict__ ipiv, int k, int minus, int m, int c0,
                 int n0, int c1, int n1, int cols_per_cta, int* info, int* err)
{
    __shared__ __align__(16) int piv[kMaxSwaps];
    const int tid = threadIdx.x;
    int bad = 0;
    for (int i = tid; i < (k + 3) / 4 * 4; i += kThr) {
        const int b = i < k ? ipiv[i] - 1 - minus : i;  // padding: a swap of nothing
        if (i < k && (b < i || b >= m)) bad = 1;
        piv[i] = b;
    }
    if (__syncthreads_or(bad)) {  // a pivot outside [row, m): move nothing
        if (tid == 0 && blockIdx.x == 0) {
            if (info) atomicExch(info, -1);
            atomicCAS(err, 0, kErrBadPivot);
        }
        return;
    }
    int pos[NP], src[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int x = tid + kThr * p;
        pos[p] = x < k ? x : (x < 2 * k ? piv[x - k] : -1);
        if (x >= k && pos[p] < k) pos[p] = -1;  // a diagonal row: already there
        src[p] = pos[p];
    }
    for (int t = (k + 3) / 4 * 4 - 4; t >= 0; t -= 4) {
        const int4 q = *reinterpret_cast<const int4*>(piv + t);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            src[p] = src[p] == t + 3 ? q.w : (src[p] == q.w ? t + 3 : src[p]);
            src[p] = src[p] == t + 2 ? q.z : (src[p] == q.z ? t + 2 : src[p]);
            src[p] = src[p] == t + 1 ? q.y : (src[p] == q.y ? t + 1 : src[p]);
            src[p] = src[p] == t ? q.x : (src[p] == q.x ? t : src[p]);
        }
    }
    const int first = blockIdx.x * cols_per_cta, last = min(first + cols_per_cta, n0 + n1);
    for (int c = first; c < last; c += kCols) {
        T v[NP][kCols];
#pragma unroll
        for (int u = 0; u < kCols; ++u) {
            const int cc = c + u;
            const T* a = A + (long long)(cc < n0 ? c0 + cc : c1 + cc - n0) * lda;
#pragma unroll
            for (int p = 0; p < NP; ++p)
                v[p][u] = (cc < last && src[p] != pos[p]) ? a[src[p]] : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kCols; ++u) {
            const int cc = c + u;
            T* a = A + (long long)(cc < n0 ? c0 + cc : c1 + cc - n0) * lda;
#pragma unroll
            for (int p = 0; p < NP; ++p)
                if (cc < last && src[p] != pos[p]) a[pos[p]] = v[p][u];
        }
    }
}

template <class T>
hdbf_status swap_rows_t(hdbf_context* ctx, T* A, long long lda, const int* ipiv, int k, int minus,
                        int m, int c0, int n0, int c1, int n1, int* info)
{
    if (k <= 0 || m <= 0) return HDBF_STATUS_SUCCESS;
    if (k > m) return HDBF_STATUS_INVALID_VALUE;
    if (k > kMaxSwaps || !ctx->dev_small) return HDBF_STATUS_NOT_SUPPORTED;
    n0 = std::max(n0, 0);
    n1 = std::max(n1, 0);
    const int n = n0 + n1;
    if (n == 0) return HDBF_STATUS_SUCCESS;
    // The composition is paid once per CTA, 10 us at 256 swaps and 20 at 512 (four
    // positions a thread): up to four CTAs per SM, two above 128 swaps, one above 256,
    // but four again where the moves take longer than that.  384 swaps on 4096 columns:
    // 63 us with four, 34 with one, 45 composed once and gathered (compose_swaps,
    // apply_moves); on 8192 columns 95, 99 and 152.
    const int one = kCols * ctx->sm_count;
    const int per_sm = k <= 128 || (k > 256 && n > 5 * one) ? 4 : (k <= 256 ? 2 : 1);
    const int passes = std::max(1, (n + per_sm * one - 1) / (per_sm * one));
    // FP32 gathers of a few thousand columns: 512 swaps on 3000 columns 36 us here, 32
    // composed once; on 1500 and on 6000 columns 28 and 66 here, 28 and 73.
    if (sizeof(T) == 4 && k > 448 && n > one && n <= 4 * one) return HDBF_STATUS_NOT_SUPPORTED;
    const int per = kCols * passes;
    const unsigned grid = (unsigned)((n + per - 1) / per);
    int* err = ctx->dev_small + kSmallErr;
    ProfScope prof(ctx, kClsMoves, 0.0, 4.0 * sizeof(T) * k * (double)n, k, n, m);
    if (2 * k <= kThr)
        swap_rows_kernel<T, 1><<<grid, kThr, 0, ctx->stream>>>(A, lda, ipiv, k, minus, m, c0, n0, c1,
                                                               n1, per, info, err);
    else if (k <= kThr)
        swap_rows_kernel<T, 2><<<grid, kThr, 0, ctx->stream>>>(A, lda, ipiv, k, minus, m, c0, n0, c1,
                                                               n1, per, info, err);
    else
        swap_rows_kernel<T, 4><<<grid, kThr, 0, ctx->stream>>>(A, lda, ipiv, k, minus, m, c0, n0, c1,
                                                               n1, per, info, err);
    ctx->launches++;
    return last_cuda(ctx);
}

}  // namespace

hdbf_status swap_rows(hdbf_context* ctx, float* A, long long lda, const int* ipiv, int k, int minus,
                      int m, int c0, int n0, int c1, int n1, int* info)
{
    return swap_rows_t(ctx, A, lda, ipiv, k, minus, m, c0, n0, c1, n1, info);
}
hdbf_status swap_rows(hdbf_context* ctx, double* A, long long lda, const int* ipiv, int k, int minus,
                      int m, int c0, int n0, int c1, int n1, int* info)
{
    return swap_rows_t(ctx, A, lda, ipiv, k, minus, m, c0, n0, c1, n1, info);
}

}  // namespace hdbf
