// Diagonal-block Cholesky and small triangular-solve kernels.
//
// potf2_small replaces rocsolver_spotrf on the diagonal block
// (src/potrf/double_blocked_potrf.cpp:34-56, call :334) at the leaf of this
// library's recursive diagonal factorization; tri_inv64 inverts the
// diagonal blocks for the TRSM leaves (trsm_block.cu) and the solves.
#include <cfloat>

#include "internal.h"
#include "tile64.cuh"

namespace hdbf {
namespace {

constexpr int kLeaf = 64;
constexpr int kTileWords =  // tile, inverse, scratch and reciprocals
    2 * kLeaf * tile64::kLd + tile64::kScratch + kLeaf;
template <class T>  // dynamic part
constexpr size_t kTileSmem = sizeof(T) == 4 ? 0 : sizeof(T) * (size_t)kTileWords;

// Cholesky of an n x n (n <= 64) lower block, one CTA (chol64), and, with inv,
// the inverse of its factor in tri_inv64's layout, so that the panel solve
// which follows needs no launch of its own for it.
// Pivot test and info follow LAPACK xPOTRF: the first column whose updated
// diagonal is not > 0 (or is NaN) stops the factorization, its value is left
// in place, and info = info_base + j + 1 (first failure wins).  A block whose
// info is already non-zero is left untouched, and inv is then the inverse of the
// block as it stands, so that the panel solve depends on the matrix alone.
template <class T>
__global__ void __launch_bounds__(tile64::kThreads, 1)
potf2_kernel(int n, T* A, long long lda, int* info, int info_base, T* inv)
{
    // FP32 fits the static limit
    __shared__ __align__(16) float fixed[sizeof(T) == 4 ? kTileWords : 4];
    extern __shared__ __align__(16) unsigned char sm_raw[];
    T* S = sizeof(T) == 4 ? reinterpret_cast<T*>(fixed) : reinterpret_cast<T*>(sm_raw);
    T* W = S + kLeaf * tile64::kLd;
    T* X = W + kLeaf * tile64::kLd;
    T* rd = X + tile64::kScratch;
    __shared__ int s_fail;
    // read by every thread before thread 0 may write it behind load_lower's barrier
    const bool done = info && *reinterpret_cast<volatile int*>(info) != 0;
    if (done && !inv) return;
    tile64::load_lower<false>(S, A, lda, n, false);
    __syncthreads();
    if (!done) {
        const int fail = tile64::chol64(S, n, &s_fail);
        tile64::store_lower(A, S, lda, n);
        if (fail >= 0 && threadIdx.x == 0 && info) atomicCAS(info, 0, info_base + fail + 1);
    }
    if (inv) {
        tile64::inv64<tile64::kReciprocal>(S, W, X, rd);
        tile64::store_inv(inv, W, false);
    }
}

// Inverses of the 64x64 diagonal blocks of a lower-triangular n x n matrix
// (unit or non-unit diagonal), one CTA per block (inv64).
// out[b*4096 + c*64 + r] = inv(L_bb)(r, c); a partial last block is padded
// with the identity.
// mode 0: lower non-unit, 1: lower unit, 2: upper non-unit (the upper block
// U is inverted as (U^T)^{-1} and stored transposed).
template <class T>
__global__ void __launch_bounds__(tile64::kThreads, 1)
tri_inv64_kernel(int n, const T* __restrict__ L, long long ldl, int mode, T* out)
{
    // FP32 fits the static limit
    __shared__ __align__(16) float fixed[sizeof(T) == 4 ? kTileWords : 4];
    extern __shared__ __align__(16) unsigned char sm_raw[];
    T* S = sizeof(T) == 4 ? reinterpret_cast<T*>(fixed) : reinterpret_cast<T*>(sm_raw);
    T* W = S + kLeaf * tile64::kLd;
    T* X = W + kLeaf * tile64::kLd;
    T* rd = X + tile64::kScratch;
    const int base = blockIdx.x * kLeaf;
    tile64::load_lower<false>(S, L + (long long)base * ldl + base, ldl, min(kLeaf, n - base),
                              mode == 2);
    __syncthreads();
    if (mode == 1) tile64::inv64<tile64::kUnit>(S, W, X, rd);
    else if (mode == 2) tile64::inv64<tile64::kCorrected>(S, W, X, rd);
    else tile64::inv64<tile64::kReciprocal>(S, W, X, rd);
    tile64::store_inv(out + (long long)blockIdx.x * kLeaf * kLeaf, W, mode == 2);
}

// B(rows x cols) <- inv * B for rows <= 64 (inv = L^{-1} of the leaf block):
// CTA = 64 x 64 tile of B, thread = 4 x 4 outputs, in place.
__global__ void __launch_bounds__(256) llu_apply_kernel(int rows, int cols,
                                                        const float* __restrict__ inv, float* B,
                                                        long long ldb, int trans)
{
    __shared__ __align__(16) float Is[kLeaf][kLeaf];  // Is[k][r] = inv(r, k)
    __shared__ __align__(16) float Bs[kLeaf][kLeaf];  // Bs[k][c] = B(k, c0 + c)
    const int tid = threadIdx.x;
    const long long c0 = (long long)blockIdx.x * kLeaf;
    for (int idx = tid; idx < kLeaf * kLeaf; idx += 256) {
        const int k = idx >> 6, r = idx & 63;
        Is[k][r] = trans ? inv[r * kLeaf + k] : inv[idx];
        const int c = idx >> 6, kk = idx & 63;
        Bs[kk][c] = (kk < rows && c0 + c < cols) ? B[(c0 + c) * ldb + kk] : 0.f;
    }
    __syncthreads();
    const int ty = tid >> 4, tx = tid & 15;
    float acc[4][4] = {};
#pragma unroll 16
    for (int k = 0; k < kLeaf; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(&Is[k][ty * 4]);
        const float4 b = *reinterpret_cast<const float4*>(&Bs[k][tx * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w};
        const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const long long c = c0 + tx * 4 + j;
        if (c >= cols) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty * 4 + i;
            if (r < rows) B[c * ldb + r] = acc[i][j];
        }
    }
}

}  // namespace

namespace {
template <class T>
hdbf_status potf2_t(hdbf_context* ctx, int n, T* A, long long lda, int* info, int info_base, T* inv)
{
    if (n <= 0) return HDBF_STATUS_SUCCESS;
    if (n > kLeaf) return HDBF_STATUS_INVALID_VALUE;
    ProfScope prof(ctx, kClsPotf2, (double)n * n * n / 3.0, 2.0 * sizeof(T) * n * n);
    potf2_kernel<T><<<1, tile64::kThreads, kTileSmem<T>, ctx->stream>>>(n, A, lda, info, info_base,
                                                                        inv);
    ctx->launches++;
    return last_cuda(ctx);
}
template <class T>
hdbf_status tri_inv64_t(hdbf_context* ctx, int n, const T* L, long long ldl, int mode, T* out)
{
    if (n <= 0) return HDBF_STATUS_SUCCESS;
    const int blocks = (n + kLeaf - 1) / kLeaf;
    ProfScope prof(ctx, kClsTrsmInv, (double)blocks * kLeaf * kLeaf * kLeaf / 3.0,
                   2.0 * sizeof(T) * blocks * kLeaf * kLeaf);
    tri_inv64_kernel<T><<<blocks, tile64::kThreads, kTileSmem<T>, ctx->stream>>>(n, L, ldl, mode,
                                                                                 out);
    ctx->launches++;
    return last_cuda(ctx);
}
}  // namespace

void configure_tile_kernels(hdbf_context*)
{
    cudaFuncSetAttribute(potf2_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kTileSmem<double>);
    cudaFuncSetAttribute(tri_inv64_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kTileSmem<double>);
    cudaGetLastError();
}

hdbf_status potf2_small(hdbf_context* ctx, int n, float* A, long long lda, int* info,
                        int info_base, float* inv)
{
    return potf2_t(ctx, n, A, lda, info, info_base, inv);
}
hdbf_status potf2_small(hdbf_context* ctx, int n, double* A, long long lda, int* info,
                        int info_base, double* inv)
{
    return potf2_t(ctx, n, A, lda, info, info_base, inv);
}

hdbf_status tri_inv64(hdbf_context* ctx, int n, const float* L, long long ldl, bool unit,
                      float* out)
{
    return tri_inv64_t(ctx, n, L, ldl, unit ? 1 : 0, out);
}
hdbf_status tri_inv64(hdbf_context* ctx, int n, const double* L, long long ldl, bool unit,
                      double* out)
{
    return tri_inv64_t(ctx, n, L, ldl, unit ? 1 : 0, out);
}

hdbf_status tri_inv64_mode(hdbf_context* ctx, int n, const float* L, long long ldl, int mode,
                           float* out)
{
    return tri_inv64_t(ctx, n, L, ldl, mode, out);
}

hdbf_status llu_apply_t(hdbf_context* ctx, int rows, int cols, const float* inv, float* B,
                        long long ldb, bool trans)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    if (rows > kLeaf) return HDBF_STATUS_INVALID_VALUE;
    const long long grid = ((long long)cols + kLeaf - 1) / kLeaf;
    ProfScope prof(ctx, kClsTrsmL, 2.0 * kLeaf * kLeaf * (double)cols, 8.0 * rows * cols);
    llu_apply_kernel<<<(unsigned)grid, 256, 0, ctx->stream>>>(rows, cols, inv, B, ldb,
                                                               trans ? 1 : 0);
    ctx->launches++;
    return last_cuda(ctx);
}

}  // namespace hdbf
