// Leaves of the recursive TRSMs, up to four 64 x 64 diagonal blocks at once:
// left/lower/unit B <- L^{-1} B (rows <= 256) and right/lower/transposed
// B <- B L^{-T} (cols <= 256).  They replace the reference's trsm_left_lower_unit
// (src/getrf/getrf_npvt_internal.h:42-88) and rocblas_strsm at the leaves of its
// right-side TRSM (src/trsm/right_lower_trsm.cpp:24-37).
//
// A CTA keeps a slice of B (all rows, or all columns) in shared memory and runs
// the block forward substitution with the inverted diagonal blocks D_i:
//     X_i = D_i (B_i - sum_{j<i} L_ij X_j)       (and its transpose on the right).
// The order of the L and D tiles is known from the start, so they come through
// a three-deep cp.async ring while earlier ones are multiplied (4 x 4 or smaller
// register tiles, packed FP32 FMAs); before, each of the ten tile products of a
// 256-wide block waited for its own loads (57 us at 7500 x 256, now 33; 19 us
// at 2000 x 64, now 7.5).  The slice width falls when wider slices would not give
// every SM a CTA.
#include "internal.h"

namespace hdbf {
namespace {

constexpr int kT = 64;
constexpr int kThr = 256;
constexpr int kMaxW = 256;   // rows (left) / columns (right) of the solved block
constexpr int kRing = 3;
constexpr int kTile = kT * kT;
constexpr int kLdL = kMaxW + 4;  // left: pitch of a column of X

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void copy16(float* dst, const float* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src, bool have)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(have ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// 64 columns of 64 contiguous floats: dst[c * pitch + r] = src[c * ld + r], zero
// outside rows x cols.
__device__ __forceinline__ void copy_tile(float* dst, int pitch, const float* src, long long ld,
                                          int rows, int cols)
{
    const bool vec = rows == kT && cols == kT && ld % 4 == 0 &&
                     (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
    if (vec) {
#pragma unroll
        for (int u = 0; u < kTile / 4 / kThr; ++u) {
            const int q = threadIdx.x + u * kThr, c = q >> 4, r = (q & 15) * 4;
            copy16(dst + c * pitch + r, src + (long long)c * ld + r);
        }
    } else {
#pragma unroll
        for (int u = 0; u < kTile / kThr; ++u) {
            const int q = threadIdx.x + u * kThr, c = q >> 6, r = q & 63;
            const bool have = r < rows && c < cols;
            copy4(dst + c * pitch + r, have ? src + (long long)c * ld + r : src, have);
        }
    }
}

// Tile t of the substitution: (i, j) with j < i the block L_ij, j == i the
// inverse D_i; i = 0, 1, ... and within it j = 0 .. i.
__device__ __forceinline__ void tile_at(int t, int& i, int& j)
{
    i = 0;
    while (t > i) t -= ++i;
    j = t;
}

__device__ __forceinline__ unsigned long long pack2(float x, float y)
{
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    return v;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a,
                                     unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// ------------------------------------------------------------------- right
// CTA: 16 RP rows of B, all columns.  X[c * 16 RP + r].  Thread: RP rows
// (RP * (tid & 15)) x 4 columns (4 * (tid >> 4)) of a 64-column block.
template <int RP>
__global__ void __launch_bounds__(kThr) rlt_block_kernel(int rows, int cols,
                                                         const float* __restrict__ L, long long ldl,
                                                         const float* __restrict__ inv, float* B,
                                                         long long ldb)
{
    constexpr int RT = 16 * RP;  // rows of the slice
    extern __shared__ __align__(16) float sm[];
    const int nb = (cols + kT - 1) / kT, nt = nb * (nb + 1) / 2;
    const int ring = min(nt, kRing);
    float* tiles = sm;
    float* X = sm + ring * kTile;
    const int tid = threadIdx.x, ty = tid & 15, tx = tid >> 4;
    const long long r0 = (long long)blockIdx.x * RT;
    const int nr = (int)min((long long)RT, (long long)rows - r0);
    auto fetch = [&](int t) {
        if (t < nt) {
            int i, j;
            tile_at(t, i, j);
            float* dst = tiles + (t % ring) * kTile;
            if (i == j) copy_tile(dst, kT, inv + (long long)i * kTile, kT, kT, kT);
            else  // [k][c] = L(64 i + c, 64 j + k)
                copy_tile(dst, kT, L + (long long)(j * kT) * ldl + i * kT, ldl,
                          min(kT, cols - i * kT), kT);
        }
        commit();
    };
    {
        const bool vec = nr == RT && ldb % 4 == 0 && (reinterpret_cast<uintptr_t>(B + r0) & 15u) == 0;
        const int total = nb * kT * RT;
        if (vec) {
            for (int q = tid * 4; q < total; q += kThr * 4) {
                const int c = q / RT, r = q % RT;
                if (c < cols) copy16(X + q, B + (long long)c * ldb + r0 + r);
                else *reinterpret_cast<float4*>(X + q) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        } else {
            for (int q = tid; q < total; q += kThr) {
                const int c = q / RT, r = q % RT;
                const bool have = r < nr && c < cols;
                copy4(X + q, have ? B + (long long)c * ldb + r0 + r : B, have);
            }
        }
    }
    fetch(0);
    if (ring > 1) fetch(1); else commit();
    int t = 0;
    for (int i = 0; i < nb; ++i) {
        unsigned long long acc[4][(RP + 1) / 2];
        float a1[4];  // RP == 1
        for (int j = 0; j <= i; ++j, ++t) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();  // tile t and X are there; tile t - 1 and X_i's old reads are done
            if (ring > 2) fetch(t + 2); else commit();
            if (j == 0) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float* x = X + (i * kT + tx * 4 + c) * RT + ty * RP;
                    if (RP == 1) a1[c] = i == 0 ? 0.f : x[0];
#pragma unroll
                    for (int h = 0; h < RP / 2; ++h)
                        acc[c][h] = i == 0 ? 0ull : *reinterpret_cast<const unsigned long long*>(x + 2 * h);
                }
            }
            const float* b = tiles + (t % ring) * kTile + tx * 4;
            const float* x = X + j * kT * RT + ty * RP;
            if (j == i && i > 0) {  // B_i - sum back into X_i, then times D_i
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float* o = X + (i * kT + tx * 4 + c) * RT + ty * RP;
                    if (RP == 1) o[0] = a1[c], a1[c] = 0.f;
#pragma unroll
                    for (int h = 0; h < RP / 2; ++h) {
                        *reinterpret_cast<unsigned long long*>(o + 2 * h) = acc[c][h];
                        acc[c][h] = 0ull;
                    }
                }
                __syncthreads();
            }
            const float sign = j == i ? 1.f : -1.f;
#pragma unroll 8
            for (int k = 0; k < kT; ++k) {
                const float4 bv = *reinterpret_cast<const float4*>(b + k * kT);
                const float bb[4] = {sign * bv.x, sign * bv.y, sign * bv.z, sign * bv.w};
                if (RP == 1) {
                    const float xv = x[k * RT];
#pragma unroll
                    for (int c = 0; c < 4; ++c) a1[c] = fmaf(xv, bb[c], a1[c]);
                }
#pragma unroll
                for (int h = 0; h < RP / 2; ++h) {
                    const unsigned long long xv =
                        *reinterpret_cast<const unsigned long long*>(x + k * RT + 2 * h);
#pragma unroll
                    for (int c = 0; c < 4; ++c) fma2(acc[c][h], xv, pack2(bb[c], bb[c]));
                }
            }
            if (j == i) {
                if (i + 1 < nb) __syncthreads();  // X_i is still being read
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int col = i * kT + tx * 4 + c;
                    float v[RP];
                    if (RP == 1) v[0] = a1[c];
#pragma unroll
                    for (int h = 0; h < RP / 2; ++h) {
                        const float2 p = unpack2(acc[c][h]);
                        v[2 * h] = p.x;
                        v[(2 * h + 1) % RP] = p.y;
                    }
#pragma unroll
                    for (int e = 0; e < RP; ++e) {
                        if (i + 1 < nb) X[col * RT + ty * RP + e] = col < cols ? v[e] : 0.f;
                        if (col < cols && ty * RP + e < nr)
                            B[(long long)col * ldb + r0 + ty * RP + e] = v[e];
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// -------------------------------------------------------------------- left
// CTA: 16 CP columns of B, all rows.  X[n * kLdL + k].  Thread: 4 rows
// (4 * (tid & 15)) of a 64-row block x CP columns (CP * (tid >> 4)).
template <int CP>
__global__ void __launch_bounds__(kThr) llu_block_kernel(int rows, int cols,
                                                         const float* __restrict__ L, long long ldl,
                                                         const float* __restrict__ inv, float* B,
                                                         long long ldb)
{
    constexpr int CT = 16 * CP;
    extern __shared__ __align__(16) float sm[];
    const int nb = (rows + kT - 1) / kT, nt = nb * (nb + 1) / 2;
    const int ring = min(nt, kRing);
    float* tiles = sm;
    float* X = sm + ring * kTile;
    const int tid = threadIdx.x, ty = tid & 15, tx = tid >> 4;
    const long long c0 = (long long)blockIdx.x * CT;
    const int nc = (int)min((long long)CT, (long long)cols - c0);
    auto fetch = [&](int t) {
        if (t < nt) {
            int i, j;
            tile_at(t, i, j);
            float* dst = tiles + (t % ring) * kTile;
            if (i == j) copy_tile(dst, kT, inv + (long long)i * kTile, kT, kT, kT);
            else  // [k][m] = L(64 i + m, 64 j + k)
                copy_tile(dst, kT, L + (long long)(j * kT) * ldl + i * kT, ldl,
                          min(kT, rows - i * kT), kT);
        }
        commit();
    };
    {
        const int len = nb * kT;
        const bool vec = rows == len && ldb % 4 == 0 && (reinterpret_cast<uintptr_t>(B) & 15u) == 0;
        if (vec) {
            for (int q = tid * 4; q < CT * len; q += kThr * 4) {
                const int n = q / len, k = q - n * len;
                if (n < nc) copy16(X + n * kLdL + k, B + (c0 + n) * ldb + k);
                else *reinterpret_cast<float4*>(X + n * kLdL + k) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        } else {
            for (int q = tid; q < CT * len; q += kThr) {
                const int n = q / len, k = q - n * len;
                const bool have = n < nc && k < rows;
                copy4(X + n * kLdL + k, have ? B + (c0 + n) * ldb + k : B, have);
            }
        }
    }
    fetch(0);
    if (ring > 1) fetch(1); else commit();
    int t = 0;
    for (int i = 0; i < nb; ++i) {
        unsigned long long acc[CP][2];  // [column][row pair]
        for (int j = 0; j <= i; ++j, ++t) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            if (ring > 2) fetch(t + 2); else commit();
            if (j == 0) {
#pragma unroll
                for (int c = 0; c < CP; ++c) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(
                        X + (tx * CP + c) * kLdL + i * kT + ty * 4);
                    acc[c][0] = i == 0 ? 0ull : v.x;
                    acc[c][1] = i == 0 ? 0ull : v.y;
                }
            }
            const float* a = tiles + (t % ring) * kTile + ty * 4;
            if (j == i && i > 0) {
#pragma unroll
                for (int c = 0; c < CP; ++c) {
                    ulonglong2 v;
                    v.x = acc[c][0];
                    v.y = acc[c][1];
                    *reinterpret_cast<ulonglong2*>(X + (tx * CP + c) * kLdL + i * kT + ty * 4) = v;
                    acc[c][0] = acc[c][1] = 0ull;
                }
                __syncthreads();
            }
            const float sign = j == i ? 1.f : -1.f;
            const float* x = X + tx * CP * kLdL + j * kT;
#pragma unroll 4
            for (int k = 0; k < kT; k += 4) {
                float4 xv[CP];
#pragma unroll
                for (int c = 0; c < CP; ++c)
                    xv[c] = *reinterpret_cast<const float4*>(x + c * kLdL + k);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(a + (k + q) * kT);
#pragma unroll
                    for (int c = 0; c < CP; ++c) {
                        const float e = sign * (q == 0 ? xv[c].x : q == 1 ? xv[c].y
                                                       : q == 2 ? xv[c].z : xv[c].w);
                        fma2(acc[c][0], av.x, pack2(e, e));
                        fma2(acc[c][1], av.y, pack2(e, e));
                    }
                }
            }
            if (j == i) {
                if (i + 1 < nb) __syncthreads();
#pragma unroll
                for (int c = 0; c < CP; ++c) {
                    const int n = tx * CP + c;
                    const float2 p = unpack2(acc[c][0]), q = unpack2(acc[c][1]);
                    const float v[4] = {p.x, p.y, q.x, q.y};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int r = i * kT + ty * 4 + e;
                        if (i + 1 < nb) X[n * kLdL + r] = r < rows ? v[e] : 0.f;
                        if (r < rows && n < nc) B[(c0 + n) * ldb + r] = v[e];
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Dynamic shared memory for nb diagonal blocks; one block needs no more than the
// default limit, so a launch without a configured handle may take it.
template <int RP>
size_t rlt_smem(int nb)
{
    const int nt = nb * (nb + 1) / 2;
    return sizeof(float) * ((size_t)(nt < kRing ? nt : kRing) * kTile + (size_t)nb * kT * 16 * RP);
}
template <int CP>
size_t llu_smem(int nb)
{
    const int nt = nb * (nb + 1) / 2;
    return sizeof(float) * ((size_t)(nt < kRing ? nt : kRing) * kTile + (size_t)16 * CP * kLdL);
}

template <int RP>
void rlt_launch(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                const float* inv, float* B, long long ldb)
{
    const unsigned grid = (unsigned)(((long long)rows + 16 * RP - 1) / (16 * RP));
    rlt_block_kernel<RP><<<grid, kThr, rlt_smem<RP>((cols + kT - 1) / kT), ctx->stream>>>(
        rows, cols, L, ldl, inv, B, ldb);
}
template <int CP>
void llu_launch(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                const float* inv, float* B, long long ldb)
{
    const unsigned grid = (unsigned)(((long long)cols + 16 * CP - 1) / (16 * CP));
    llu_block_kernel<CP><<<grid, kThr, llu_smem<CP>((rows + kT - 1) / kT), ctx->stream>>>(
        rows, cols, L, ldl, inv, B, ldb);
}

}  // namespace

int llu_block_max_rows() { return kMaxW; }

void configure_trsm_block_kernels(hdbf_context*)
{
    const int nb = kMaxW / kT;
    cudaFuncSetAttribute(rlt_block_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rlt_smem<4>(nb));
    cudaFuncSetAttribute(rlt_block_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rlt_smem<2>(nb));
    cudaFuncSetAttribute(rlt_block_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rlt_smem<1>(nb));
    cudaFuncSetAttribute(llu_block_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)llu_smem<4>(nb));
    cudaFuncSetAttribute(llu_block_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)llu_smem<2>(nb));
    cudaFuncSetAttribute(llu_block_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)llu_smem<1>(nb));
    cudaGetLastError();
}

// B(rows x cols) <- B L^{-T} for non-unit lower L (cols <= 256); inv holds the
// 64x64 diagonal-block inverses of L (tri_inv64 layout).
hdbf_status rlt_block(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                      const float* inv, float* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    if (cols > kMaxW) return HDBF_STATUS_INVALID_VALUE;
    ProfScope prof(ctx, kClsTrsmR, (double)cols * cols * rows, 8.0 * (double)rows * cols, rows,
                   cols, (cols + kT - 1) / kT);
    // 64 rows per CTA when that gives two thirds of the SMs one, else 32, else 16
    const long long full = 2LL * ctx->sm_count / 3 * 64;
    if (rows >= full) rlt_launch<4>(ctx, rows, cols, L, ldl, inv, B, ldb);
    else if (2LL * rows >= full) rlt_launch<2>(ctx, rows, cols, L, ldl, inv, B, ldb);
    else rlt_launch<1>(ctx, rows, cols, L, ldl, inv, B, ldb);
    ctx->launches++;
    return last_cuda(ctx);
}

// B(rows x cols) <- L^{-1} B for unit lower L (rows <= 256); inv holds the
// 64x64 unit-lower diagonal-block inverses of L (tri_inv64 layout).
hdbf_status llu_block(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                      const float* inv, float* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    if (rows > kMaxW) return HDBF_STATUS_INVALID_VALUE;
    ProfScope prof(ctx, kClsTrsmL, (double)rows * rows * cols, 8.0 * (double)rows * cols, rows,
                   cols, (rows + kT - 1) / kT);
    const long long full = 2LL * ctx->sm_count / 3 * 64;  // as rlt_block
    if (cols >= full) llu_launch<4>(ctx, rows, cols, L, ldl, inv, B, ldb);
    else if (2LL * cols >= full) llu_launch<2>(ctx, rows, cols, L, ldl, inv, B, ldb);
    else llu_launch<1>(ctx, rows, cols, L, ldl, inv, B, ldb);
    ctx->launches++;
    return last_cuda(ctx);
}

}  // namespace hdbf
