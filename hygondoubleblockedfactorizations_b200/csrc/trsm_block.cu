// Leaves of the recursive TRSMs, up to four 64 x 64 diagonal blocks at once:
// left/lower/unit B <- L^{-1} B (rows <= 256) and right/lower/transposed
// B <- B L^{-T} (cols <= 256).  They replace the reference's trsm_left_lower_unit
// (src/getrf/getrf_npvt_internal.h:42-88) and rocblas_strsm at the leaves of its
// right-side TRSM (src/trsm/right_lower_trsm.cpp:24-37).
//
// A CTA keeps a slice of B (all rows, or all columns) in shared memory and runs
// the block forward substitution with the inverted diagonal blocks D_i:
//     X_i = D_i (B_i - sum_{j<i} L_ij X_j)       (and its transpose on the right).
// Each product L_ij X_j is summed from zero and then subtracted from what is left
// of B_i: FMAs straight onto B_i would round every term at the size of B_i (five
// times the error at 256 columns where the off-diagonal part is small).
// The order of the L and D tiles is known from the start, so they come through
// a three-deep cp.async ring while earlier ones are multiplied (4 x 4 or smaller
// register tiles, packed FP32 FMAs); before, each of the ten tile products of a
// 256-wide block waited for its own loads (57 us at 7500 x 256, now 33; 19 us
// at 2000 x 64, now 7.5).  The slice width falls when wider slices would not give
// every SM a CTA.  FP32 and FP64.
#include "internal.h"
#include "pair.cuh"

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
__device__ __forceinline__ void copy16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src)
                 : "memory");
}
template <class T>
__device__ __forceinline__ void copy1(T* dst, const T* src, bool have)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_addr(dst)), "l"(src),
                 "n"(sizeof(T)), "r"(have ? (int)sizeof(T) : 0)
                 : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <class T>
constexpr int kVec = 16 / (int)sizeof(T);  // elements of a 16-byte copy
template <class T>
__device__ __forceinline__ void zero16(T* p)
{
    *reinterpret_cast<uint4*>(p) = make_uint4(0u, 0u, 0u, 0u);
}

// 64 columns of 64 contiguous values: dst[c * 64 + r] = src[c * ld + r], zero
// outside rows x cols.
template <class T>
__device__ __forceinline__ void copy_tile(T* dst, const T* src, long long ld, int rows, int cols)
{
    constexpr int V = kVec<T>, PER = kT / V;
    const bool vec = rows == kT && cols == kT && ld % V == 0 &&
                     (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
    if (vec) {
#pragma unroll
        for (int u = 0; u < kT * PER / kThr; ++u) {
            const int q = threadIdx.x + u * kThr, c = q / PER, r = (q % PER) * V;
            copy16(dst + c * kT + r, src + (long long)c * ld + r);
        }
    } else {
#pragma unroll
        for (int u = 0; u < kTile / kThr; ++u) {
            const int q = threadIdx.x + u * kThr, c = q >> 6, r = q & 63;
            const bool have = r < rows && c < cols;
            copy1(dst + c * kT + r, have ? src + (long long)c * ld + r : src, have);
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

// ------------------------------------------------------------------- right
// acc[c][e] = sum_k x[k * ldx + e] b[k * 64 + c] over 64 of K.
template <class T, int RP>
__device__ __forceinline__ void right_product(T acc[4][RP], const T* x, int ldx, const T* b)
{
    if (RP == 1) {
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c][0] = T(0);
#pragma unroll 8
        for (int k = 0; k < kT; ++k) {
            T bv[4];
            Two<T> lo, hi;
            load_pairs(b + k * kT, lo, hi);
            lo.get(bv[0], bv[1]);
            hi.get(bv[2], bv[3]);
            const T xv = x[k * ldx];
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[c][0] = ::fma(xv, bv[c], acc[c][0]);
        }
    } else {
        Two<T> s[4][RP / 2 > 0 ? RP / 2 : 1];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < RP / 2; ++h) s[c][h] = Two<T>::zero();
#pragma unroll 8
        for (int k = 0; k < kT; ++k) {
            T bv[4];
            Two<T> lo, hi;
            load_pairs(b + k * kT, lo, hi);
            lo.get(bv[0], bv[1]);
            hi.get(bv[2], bv[3]);
            Two<T> xv[RP / 2 > 0 ? RP / 2 : 1];
#pragma unroll
            for (int h = 0; h < RP / 2; ++h)
                xv[h] = *reinterpret_cast<const Two<T>*>(x + k * ldx + 2 * h);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const Two<T> bb = Two<T>::make(bv[c], bv[c]);
#pragma unroll
                for (int h = 0; h < RP / 2; ++h) s[c][h].fma(xv[h], bb);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int h = 0; h < RP / 2; ++h) s[c][h].get(acc[c][2 * h], acc[c][(2 * h + 1) % RP]);
    }
}

// CTA: 16 RP rows of B, all columns.  X[c * 16 RP + r].  Thread: RP rows
// (RP * (tid & 15)) x 4 columns (4 * (tid >> 4)) of a 64-column block.
template <class T, int RP>
__global__ void __launch_bounds__(kThr) rlt_block_kernel(int rows, int cols,
                                                         const T* __restrict__ L, long long ldl,
                                                         const T* __restrict__ inv, T* B,
                                                         long long ldb)
{
    constexpr int RT = 16 * RP;  // rows of the slice
    extern __shared__ __align__(16) unsigned char sm_raw[];
    T* sm = reinterpret_cast<T*>(sm_raw);
    const int nb = (cols + kT - 1) / kT, nt = nb * (nb + 1) / 2;
    const int ring = min(nt, kRing);
    T* tiles = sm;
    T* X = sm + ring * kTile;
    const int tid = threadIdx.x, ty = tid & 15, tx = tid >> 4;
    const long long r0 = (long long)blockIdx.x * RT;
    const int nr = (int)min((long long)RT, (long long)rows - r0);
    auto fetch = [&](int t) {
        if (t < nt) {
            int i, j;
            tile_at(t, i, j);
            T* dst = tiles + (t % ring) * kTile;
            if (i == j) copy_tile(dst, inv + (long long)i * kTile, kT, kT, kT);
            else  // [k][c] = L(64 i + c, 64 j + k)
                copy_tile(dst, L + (long long)(j * kT) * ldl + i * kT, ldl,
                          min(kT, cols - i * kT), kT);
        }
        commit();
    };
    {
        constexpr int V = kVec<T>;
        const bool vec = nr == RT && ldb % V == 0 && (reinterpret_cast<uintptr_t>(B + r0) & 15u) == 0;
        const int total = nb * kT * RT;
        if (vec) {
            for (int q = tid * V; q < total; q += kThr * V) {
                const int c = q / RT, r = q % RT;
                if (c < cols) copy16(X + q, B + (long long)c * ldb + r0 + r);
                else zero16(X + q);
            }
        } else {
            for (int q = tid; q < total; q += kThr) {
                const int c = q / RT, r = q % RT;
                const bool have = r < nr && c < cols;
                copy1(X + q, have ? B + (long long)c * ldb + r0 + r : B, have);
            }
        }
    }
    fetch(0);
    if (ring > 1) fetch(1); else commit();
    int t = 0;
    for (int i = 0; i < nb; ++i) {
        T acc[4][RP], rest[4][RP];  // rest: B_i less the products so far
        for (int j = 0; j <= i; ++j, ++t) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();  // tile t and X are there; tile t - 1 and X_i's old reads are done
            if (ring > 2) fetch(t + 2); else commit();
            if (j == 0 && i > 0) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < RP; ++e)
                        rest[c][e] = X[(i * kT + tx * 4 + c) * RT + ty * RP + e];
            }
            const T* b = tiles + (t % ring) * kTile + tx * 4;
            const T* x = X + j * kT * RT + ty * RP;
            if (j == i && i > 0) {  // B_i - sum back into X_i, then times D_i
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < RP; ++e)
                        X[(i * kT + tx * 4 + c) * RT + ty * RP + e] = rest[c][e];
                __syncthreads();
            }
            right_product<T, RP>(acc, x, RT, b);
            if (j < i) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < RP; ++e) rest[c][e] -= acc[c][e];
            }
            if (j == i) {
                if (i + 1 < nb) __syncthreads();  // X_i is still being read
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int col = i * kT + tx * 4 + c;
#pragma unroll
                    for (int e = 0; e < RP; ++e) {
                        if (i + 1 < nb) X[col * RT + ty * RP + e] = col < cols ? acc[c][e] : T(0);
                        if (col < cols && ty * RP + e < nr)
                            B[(long long)col * ldb + r0 + ty * RP + e] = acc[c][e];
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
template <class T, int CP>
__global__ void __launch_bounds__(kThr) llu_block_kernel(int rows, int cols,
                                                         const T* __restrict__ L, long long ldl,
                                                         const T* __restrict__ inv, T* B,
                                                         long long ldb)
{
    constexpr int CT = 16 * CP;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    T* sm = reinterpret_cast<T*>(sm_raw);
    const int nb = (rows + kT - 1) / kT, nt = nb * (nb + 1) / 2;
    const int ring = min(nt, kRing);
    T* tiles = sm;
    T* X = sm + ring * kTile;
    const int tid = threadIdx.x, ty = tid & 15, tx = tid >> 4;
    const long long c0 = (long long)blockIdx.x * CT;
    const int nc = (int)min((long long)CT, (long long)cols - c0);
    auto fetch = [&](int t) {
        if (t < nt) {
            int i, j;
            tile_at(t, i, j);
            T* dst = tiles + (t % ring) * kTile;
            if (i == j) copy_tile(dst, inv + (long long)i * kTile, kT, kT, kT);
            else  // [k][m] = L(64 i + m, 64 j + k)
                copy_tile(dst, L + (long long)(j * kT) * ldl + i * kT, ldl,
                          min(kT, rows - i * kT), kT);
        }
        commit();
    };
    {
        constexpr int V = kVec<T>;
        const int len = nb * kT;
        const bool vec = rows == len && ldb % V == 0 && (reinterpret_cast<uintptr_t>(B) & 15u) == 0;
        if (vec) {
            for (int q = tid * V; q < CT * len; q += kThr * V) {
                const int n = q / len, k = q - n * len;
                if (n < nc) copy16(X + n * kLdL + k, B + (c0 + n) * ldb + k);
                else zero16(X + n * kLdL + k);
            }
        } else {
            for (int q = tid; q < CT * len; q += kThr) {
                const int n = q / len, k = q - n * len;
                const bool have = n < nc && k < rows;
                copy1(X + n * kLdL + k, have ? B + (c0 + n) * ldb + k : B, have);
            }
        }
    }
    fetch(0);
    if (ring > 1) fetch(1); else commit();
    int t = 0;
    const Two<T> minus = Two<T>::make(T(-1), T(-1));
    for (int i = 0; i < nb; ++i) {
        Two<T> acc[CP][2], rest[CP][2];  // [column][row pair]; rest as on the right
        for (int j = 0; j <= i; ++j, ++t) {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            if (ring > 2) fetch(t + 2); else commit();
            if (j == 0 && i > 0) {
#pragma unroll
                for (int c = 0; c < CP; ++c)
                    load_pairs(X + (tx * CP + c) * kLdL + i * kT + ty * 4, rest[c][0], rest[c][1]);
            }
            const T* a = tiles + (t % ring) * kTile + ty * 4;
            if (j == i && i > 0) {
#pragma unroll
                for (int c = 0; c < CP; ++c)
                    store_pairs(X + (tx * CP + c) * kLdL + i * kT + ty * 4, rest[c][0], rest[c][1]);
                __syncthreads();
            }
#pragma unroll
            for (int c = 0; c < CP; ++c) acc[c][0] = acc[c][1] = Two<T>::zero();
            const T* x = X + tx * CP * kLdL + j * kT;
#pragma unroll 4
            for (int k = 0; k < kT; k += 4) {
                T xv[CP][4];
#pragma unroll
                for (int c = 0; c < CP; ++c) {
                    Two<T> lo, hi;
                    load_pairs(x + c * kLdL + k, lo, hi);
                    lo.get(xv[c][0], xv[c][1]);
                    hi.get(xv[c][2], xv[c][3]);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    Two<T> a0, a1;
                    load_pairs(a + (k + q) * kT, a0, a1);
#pragma unroll
                    for (int c = 0; c < CP; ++c) {
                        const Two<T> ee = Two<T>::make(xv[c][q], xv[c][q]);
                        acc[c][0].fma(a0, ee);
                        acc[c][1].fma(a1, ee);
                    }
                }
            }
            if (j < i) {
#pragma unroll
                for (int c = 0; c < CP; ++c)
#pragma unroll
                    for (int h = 0; h < 2; ++h) rest[c][h].fma(acc[c][h], minus);
            }
            if (j == i) {
                if (i + 1 < nb) __syncthreads();
#pragma unroll
                for (int c = 0; c < CP; ++c) {
                    const int n = tx * CP + c;
                    T v[4];
                    acc[c][0].get(v[0], v[1]);
                    acc[c][1].get(v[2], v[3]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int r = i * kT + ty * 4 + e;
                        if (i + 1 < nb) X[n * kLdL + r] = r < rows ? v[e] : T(0);
                        if (r < rows && n < nc) B[(c0 + n) * ldb + r] = v[e];
                    }
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Dynamic shared memory for nb diagonal blocks; one FP32 block needs no more than
// the default limit, so a launch without a configured handle may take it.
template <class T, int RP>
size_t rlt_smem(int nb)
{
    const int nt = nb * (nb + 1) / 2;
    return sizeof(T) * ((size_t)(nt < kRing ? nt : kRing) * kTile + (size_t)nb * kT * 16 * RP);
}
template <class T, int CP>
size_t llu_smem(int nb)
{
    const int nt = nb * (nb + 1) / 2;
    return sizeof(T) * ((size_t)(nt < kRing ? nt : kRing) * kTile + (size_t)16 * CP * kLdL);
}

template <class T, int RP>
void rlt_launch(hdbf_context* ctx, int rows, int cols, const T* L, long long ldl, const T* inv, T* B,
                long long ldb)
{
    const unsigned grid = (unsigned)(((long long)rows + 16 * RP - 1) / (16 * RP));
    rlt_block_kernel<T, RP><<<grid, kThr, rlt_smem<T, RP>((cols + kT - 1) / kT), ctx->stream>>>(
        rows, cols, L, ldl, inv, B, ldb);
}
template <class T, int CP>
void llu_launch(hdbf_context* ctx, int rows, int cols, const T* L, long long ldl, const T* inv, T* B,
                long long ldb)
{
    const unsigned grid = (unsigned)(((long long)cols + 16 * CP - 1) / (16 * CP));
    llu_block_kernel<T, CP><<<grid, kThr, llu_smem<T, CP>((rows + kT - 1) / kT), ctx->stream>>>(
        rows, cols, L, ldl, inv, B, ldb);
}

template <class T, int P>
void configure_one()
{
    const int nb = kMaxW / kT;
    cudaFuncSetAttribute(rlt_block_kernel<T, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rlt_smem<T, P>(nb));
    cudaFuncSetAttribute(llu_block_kernel<T, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)llu_smem<T, P>(nb));
}

template <class T>
hdbf_status rlt_block_t(hdbf_context* ctx, int rows, int cols, const T* L, long long ldl,
                        const T* inv, T* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    if (cols > kMaxW) return HDBF_STATUS_INVALID_VALUE;
    ProfScope prof(ctx, kClsTrsmR, (double)cols * cols * rows, 2.0 * sizeof(T) * rows * cols, rows,
                   cols, (cols + kT - 1) / kT);
    // 64 rows per CTA when that gives two thirds of the SMs one, else 32, else 16
    const long long full = 2LL * ctx->sm_count / 3 * 64;
    if (rows >= full) rlt_launch<T, 4>(ctx, rows, cols, L, ldl, inv, B, ldb);
    else if (2LL * rows >= full) rlt_launch<T, 2>(ctx, rows, cols, L, ldl, inv, B, ldb);
    else rlt_launch<T, 1>(ctx, rows, cols, L, ldl, inv, B, ldb);
    ctx->launches++;
    return last_cuda(ctx);
}

template <class T>
hdbf_status llu_block_t(hdbf_context* ctx, int rows, int cols, const T* L, long long ldl,
                        const T* inv, T* B, long long ldb)
{
    if (rows <= 0 || cols <= 0) return HDBF_STATUS_SUCCESS;
    if (rows > kMaxW) return HDBF_STATUS_INVALID_VALUE;
    ProfScope prof(ctx, kClsTrsmL, (double)rows * rows * cols, 2.0 * sizeof(T) * rows * cols, rows,
                   cols, (rows + kT - 1) / kT);
    const long long full = 2LL * ctx->sm_count / 3 * 64;  // as rlt_block
    if (cols >= full) llu_launch<T, 4>(ctx, rows, cols, L, ldl, inv, B, ldb);
    else if (2LL * cols >= full) llu_launch<T, 2>(ctx, rows, cols, L, ldl, inv, B, ldb);
    else llu_launch<T, 1>(ctx, rows, cols, L, ldl, inv, B, ldb);
    ctx->launches++;
    return last_cuda(ctx);
}

}  // namespace

int llu_block_max_rows() { return kMaxW; }

void configure_trsm_block_kernels(hdbf_context*)
{
    configure_one<float, 4>();
    configure_one<float, 2>();
    configure_one<float, 1>();
    configure_one<double, 4>();
    configure_one<double, 2>();
    configure_one<double, 1>();
    cudaGetLastError();
}

// B(rows x cols) <- B L^{-T} for non-unit lower L (cols <= 256); inv holds the
// 64x64 diagonal-block inverses of L (tri_inv64 layout).
hdbf_status rlt_block(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                      const float* inv, float* B, long long ldb)
{
    return rlt_block_t(ctx, rows, cols, L, ldl, inv, B, ldb);
}
hdbf_status rlt_block(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                      const double* inv, double* B, long long ldb)
{
    return rlt_block_t(ctx, rows, cols, L, ldl, inv, B, ldb);
}

// B(rows x cols) <- L^{-1} B for unit lower L (rows <= 256); inv holds the
// 64x64 unit-lower diagonal-block inverses of L (tri_inv64 layout).
hdbf_status llu_block(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                      const float* inv, float* B, long long ldb)
{
    return llu_block_t(ctx, rows, cols, L, ldl, inv, B, ldb);
}
hdbf_status llu_block(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                      const double* inv, double* B, long long ldb)
{
    return llu_block_t(ctx, rows, cols, L, ldl, inv, B, ldb);
}

}  // namespace hdbf
