// FP32 and FP64 updates that do not fill the machine with 128 x 128 tiles:
//     C -= A * B^T  (NT: A is M x K, B is N x K)  or  C -= A * B  (NN: B is K x N),
// column-major, the whole of C or its lower triangle.
//
// These are the inner updates of the panels (N = 64 .. 256, K <= 1024).  They
// sit on the factorizations' serial chain and were bound by latency: the 128 x
// 128 x 8 kernel waits for one global load per 8 of K (1200 cycles a slab) on a
// few SMs.  Here a CTA owns a 64 x 64 tile (256 threads, 4 x 4 entries each,
// packed FP32 FMAs), operands come in slabs of 32 of K through a four-deep
// cp.async ring, and a cluster of S CTAs shares a tile's K: each sums its own
// range, then every CTA adds up its share of the columns from the S partial
// tiles in distributed shared memory, in K order, and subtracts it from C -- one
// launch, no scratch in global memory, results independent of timing.
// M = 2048, N = 64, K = 512: 40 us before, 9 us now; M = 192, N = 64, K = 192:
// 22 us, 6 us.  The FP64 twins' inner updates took 32 us on their 64 x 64 kernel.
#include <algorithm>

#include "internal.h"
#include "pair.cuh"

namespace hdbf {
namespace {

constexpr int kT = 64;      // tile
constexpr int kKB = 32;     // K per slab
constexpr int kThr = 256;
constexpr int kFold = 8;    // slabs per partial sum: FP32 error as small as a K split's
template <class T>
constexpr int kStages = sizeof(T) == 4 ? 4 : 3;
template <class T>
constexpr int kVec = 16 / (int)sizeof(T);  // elements of a 16-byte copy
constexpr int kLdN = 36;    // pitch of a k-contiguous B slab (NN): 16-byte rows, spread banks
constexpr int kSlabA = kKB * kT;
constexpr int kSlabB = kT * kLdN;  // the larger of the two layouts
constexpr int kLdP = kT + 4;       // pitch of a partial tile
template <class T>
constexpr size_t kSmem = sizeof(T) * kStages<T> * (size_t)(kSlabA + kSlabB);
static_assert(kT * kLdP <= 3 * (kSlabA + kSlabB), "partial tile fits over the ring");

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// 16 bytes, of which the first `bytes` are read and the rest are zero.
__device__ __forceinline__ void copy16(void* dst, const void* src, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(bytes)
                 : "memory");
}
template <class T>
__device__ __forceinline__ void copy1(T* dst, const T* src, bool have)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_addr(dst)), "l"(src),
                 "n"(sizeof(T)), "r"(have ? (int)sizeof(T) : 0)
                 : "memory");
}

// Slab of an operand whose rows are contiguous: dst[k * 64 + r] = src(r0 + r, k).
template <bool VEC, class T>
__device__ __forceinline__ void slab_rows(T* dst, const T* src, long long ld, int r0, int rows,
                                          int k0, int k1)
{
    if (VEC) {
        constexpr int V = kVec<T>, PER = kT / V;
#pragma unroll
        for (int u = 0; u < kKB * PER / kThr; ++u) {
            const int q = threadIdx.x + u * kThr, k = q / PER, r = (q % PER) * V;
            const int left = (k0 + k < k1) ? min(V, rows - r0 - r) : 0;
            copy16(dst + k * kT + r, left > 0 ? src + (long long)(k0 + k) * ld + r0 + r : src,
                   left > 0 ? (int)sizeof(T) * left : 0);
        }
    } else {
#pragma unroll
        for (int u = 0; u < kKB * kT / kThr; ++u) {
            const int q = threadIdx.x + u * kThr, k = q >> 6, r = q & 63;
            const bool have = k0 + k < k1 && r0 + r < rows;
            copy1(dst + k * kT + r, have ? src + (long long)(k0 + k) * ld + r0 + r : src, have);
        }
    }
}
// Slab of an operand whose K is contiguous: dst[c * kLdN + k] = src(k, c0 + c).
template <bool VEC, class T>
__device__ __forceinline__ void slab_cols(T* dst, const T* src, long long ld, int c0, int cols,
                                          int k0, int k1)
{
    if (VEC) {
        constexpr int V = kVec<T>, PER = kKB / V;
#pragma unroll
        for (int u = 0; u < kT * PER / kThr; ++u) {
            const int q = threadIdx.x + u * kThr, c = q / PER, k = (q % PER) * V;
            const int left = c0 + c < cols ? min(V, k1 - k0 - k) : 0;
            copy16(dst + c * kLdN + k, left > 0 ? src + (long long)(c0 + c) * ld + k0 + k : src,
                   left > 0 ? (int)sizeof(T) * left : 0);
        }
    } else {
#pragma unroll
        for (int u = 0; u < kKB * kT / kThr; ++u) {
            const int q = threadIdx.x + u * kThr, c = q >> 5, k = q & 31;
            const bool have = k0 + k < k1 && c0 + c < cols;
            copy1(dst + c * kLdN + k, have ? src + (long long)(c0 + c) * ld + k0 + k : src, have);
        }
    }
}

__device__ __forceinline__ float peer_load(uint32_t addr, float)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ double peer_load(uint32_t addr, double)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
    return v;
}

template <class T, bool NN, bool VEC, bool TRI>
__global__ void __launch_bounds__(kThr)
gemm_small_kernel(int M, int N, int K, const T* __restrict__ A, long long lda,
                  const T* __restrict__ B, long long ldb, T* __restrict__ C, long long ldc,
                  int tiles_m, int kc, const unsigned* range)
{
    extern __shared__ __align__(16) unsigned char sm_raw[];
    if (range && !split_range_bad(range)) return;  // done on the tensor cores
    T* sm = reinterpret_cast<T*>(sm_raw);
    constexpr int kSt = kStages<T>;
    int S, split;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(S));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(split));
    const int tile = blockIdx.x / S;
    const int m0 = (tile % tiles_m) * kT, n0 = (tile / tiles_m) * kT;
    if (TRI && m0 + kT <= n0) return;  // the whole cluster
    const int tid = threadIdx.x;
    const int ty = tid & 15, tx = tid >> 4;  // rows ty * 4 + i; columns tx * 4 + j (NN: tx + 16 j)
    const int k0 = split * kc, k1 = min(K, k0 + kc);
    const int slabs = k1 > k0 ? (k1 - k0 + kKB - 1) / kKB : 0;
    auto As = [&](int st) { return sm + st * (kSlabA + kSlabB); };
    auto Bs = [&](int st) { return sm + st * (kSlabA + kSlabB) + kSlabA; };
    auto fetch = [&](int s) {
        if (s < slabs) {
            const int k = k0 + s * kKB;
            slab_rows<VEC>(As(s % kSt), A, lda, m0, M, k, k1);
            if (NN) slab_cols<VEC>(Bs(s % kSt), B, ldb, n0, N, k, k1);
            else slab_rows<VEC>(Bs(s % kSt), B, ldb, n0, N, k, k1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < kSt - 1; ++s) fetch(s);

    auto col_of = [&](int j) { return NN ? tx + 16 * j : tx * 4 + j; };
    T c_old[4][4];  // this thread's entries of C, in flight during the products
    if (S == 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = m0 + ty * 4 + i, c = n0 + col_of(j);
                c_old[j][i] = (r < M && c < N && (!TRI || r >= c))
                                  ? __ldcg(C + (long long)c * ldc + r)
                                  : T(0);
            }
    }
    Two<T> acc[4][2];  // [column][row pair]
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = Two<T>::zero();
    Two<T> total[4][2];  // FP32: sums of 256 of K each
#pragma unroll
    for (int j = 0; j < 4; ++j) total[j][0] = total[j][1] = Two<T>::zero();
    auto fold = [&]() {
        const Two<T> one = Two<T>::make(T(1), T(1));
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                total[j][h].fma(acc[j][h], one);
                acc[j][h] = Two<T>::zero();
            }
    };
    for (int s = 0; s < slabs; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kSt - 2) : "memory");
        __syncthreads();
        fetch(s + kSt - 1);
        const T* a = As(s % kSt) + ty * 4;
        const T* b = Bs(s % kSt);
#pragma unroll 2
        for (int kk = 0; kk < kKB; kk += 4) {
            T bv[4][4];  // NT: [k][column]; NN: [column][k]
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                Two<T> lo, hi;
                load_pairs(NN ? b + (tx + 16 * q) * kLdN + kk : b + (kk + q) * kT + tx * 4, lo, hi);
                lo.get(bv[q][0], bv[q][1]);
                hi.get(bv[q][2], bv[q][3]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                Two<T> a0, a1;
                load_pairs(a + (kk + q) * kT, a0, a1);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const T x = NN ? bv[j][q] : bv[q][j];
                    const Two<T> xx = Two<T>::make(x, x);
                    acc[j][0].fma(a0, xx);
                    acc[j][1].fma(a1, xx);
                }
            }
        }
        if (sizeof(T) == 4 && s % kFold == kFold - 1) fold();
    }
    if (sizeof(T) == 4) fold();
    Two<T>(&sums)[4][2] = sizeof(T) == 4 ? total : acc;
    T p[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        sums[j][0].get(p[j][0], p[j][1]);
        sums[j][1].get(p[j][2], p[j][3]);
    }
    if (S == 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = m0 + ty * 4 + i, c = n0 + col_of(j);
                if (r < M && c < N && (!TRI || r >= c))
                    C[(long long)c * ldc + r] = c_old[j][i] - p[j][i];
            }
        return;
    }
    // Partial tile over the ring, P[c * kLdP + r]; then this CTA's columns.
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) store_pairs(sm + col_of(j) * kLdP + ty * 4, sums[j][0], sums[j][1]);
    const int per = kT / S;  // columns of this CTA: 256 threads = 64 rows x 4 columns at a time
    const int row = tid & 63, r = m0 + row;
    T old[8];  // S >= 2: at most 32 columns
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int cl = (tid >> 6) + 4 * q, c = n0 + split * per + cl;
        old[q] = (cl < per && r < M && c < N && (!TRI || r >= c))
                     ? __ldcg(C + (long long)c * ldc + r)
                     : T(0);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    T sum[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) sum[q] = T(0);
    const uint32_t base = smem_addr(sm);
    for (int s = 0; s < S; ++s) {
        uint32_t peer;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(base), "r"(s));
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int cl = (tid >> 6) + 4 * q;
            if (cl < per) {
                const T v = peer_load(
                    peer + (uint32_t)sizeof(T) * (uint32_t)((split * per + cl) * kLdP + row), T(0));
                sum[q] = s == 0 ? v : sum[q] + v;
            }
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int cl = (tid >> 6) + 4 * q, c = n0 + split * per + cl;
        if (cl < per && r < M && c < N && (!TRI || r >= c)) C[(long long)c * ldc + r] = old[q] - sum[q];
    }
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // partials stay until read
}

template <class T, bool NN, bool VEC, bool TRI>
cudaError_t launch(cudaStream_t st, int S, int M, int N, int K, const T* A, long long lda,
                   const T* B, long long ldb, T* C, long long ldc, const unsigned* range)
{
    const int tm = (M + kT - 1) / kT, tn = (N + kT - 1) / kT;
    const int kc = ((K + S - 1) / S + 7) / 8 * 8;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tm * tn * S));
    cfg.blockDim = dim3(kThr);
    cfg.dynamicSmemBytes = kSmem<T>;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = S;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, gemm_small_kernel<T, NN, VEC, TRI>, M, N, K, A, lda, B, ldb, C,
                              ldc, tm, kc, range);
}

template <class T, bool NN, bool VEC, bool TRI>
void configure_one()
{
    cudaFuncSetAttribute(gemm_small_kernel<T, NN, VEC, TRI>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem<T>);
}
template <class T>
void configure_type()
{
    configure_one<T, false, false, false>();
    configure_one<T, false, false, true>();
    configure_one<T, false, true, false>();
    configure_one<T, false, true, true>();
    configure_one<T, true, false, false>();
    configure_one<T, true, true, false>();
}

template <class T>
hdbf_status gemm_small_t(hdbf_context* ctx, bool nn, bool lower, int S, int M, int N, int K,
                         const T* A, long long lda, const T* B, long long ldb, T* C, long long ldc,
                         const unsigned* range = nullptr)
{
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const bool vec = al(A) && al(B) && lda % kVec<T> == 0 && ldb % kVec<T> == 0;
    cudaStream_t s = ctx->stream;
    cudaError_t e;
    if (nn)
        e = vec ? launch<T, true, true, false>(s, S, M, N, K, A, lda, B, ldb, C, ldc, range)
                : launch<T, true, false, false>(s, S, M, N, K, A, lda, B, ldb, C, ldc, range);
    else if (lower)
        e = vec ? launch<T, false, true, true>(s, S, M, N, K, A, lda, B, ldb, C, ldc, range)
                : launch<T, false, false, true>(s, S, M, N, K, A, lda, B, ldb, C, ldc, range);
    else
        e = vec ? launch<T, false, true, false>(s, S, M, N, K, A, lda, B, ldb, C, ldc, range)
                : launch<T, false, false, false>(s, S, M, N, K, A, lda, B, ldb, C, ldc, range);
    ctx->launches++;
    if (e != cudaSuccess) {
        cudaGetLastError();
        return HDBF_STATUS_CUDA_ERROR;
    }
    return HDBF_STATUS_SUCCESS;
}

}  // namespace

void configure_gemm_small(hdbf_context*)
{
    configure_type<float>();
    configure_type<double>();
    cudaGetLastError();
}

// CTAs that share a tile's K (1, 2, 4 or 8), or 0 above two 128 x 128 tiles per SM,
// where the larger tiles win for certain; below, the callers compare the two kernels.
int gemm_small_split(const hdbf_context* ctx, int M, int N, int K)
{
    if (!ctx->dev_small) return 0;  // no handle behind this context: kernel not configured
    const long long big = (long long)((M + 127) / 128) * ((N + 127) / 128);
    if (big > 2LL * ctx->sm_count) return 0;
    const long long tiles = (long long)((M + kT - 1) / kT) * ((N + kT - 1) / kT);
    int S = 1;
    // at least 64 of K each, and no more CTAs than two per SM
    while (S < 8 && K / (2 * S) >= 64 && tiles * 2 * S <= 2LL * ctx->sm_count) S *= 2;
    return S;
}

hdbf_status gemm_small(hdbf_context* ctx, bool nn, bool lower, int S, int M, int N, int K,
                       const float* A, long long lda, const float* B, long long ldb, float* C,
                       long long ldc, const unsigned* range)
{
    return gemm_small_t(ctx, nn, lower, S, M, N, K, A, lda, B, ldb, C, ldc, range);
}
hdbf_status gemm_small(hdbf_context* ctx, bool nn, bool lower, int S, int M, int N, int K,
                       const double* A, long long lda, const double* B, long long ldb, double* C,
                       long long ldc)
{
    return gemm_small_t(ctx, nn, lower, S, M, N, K, A, lda, B, ldb, C, ldc);
}

}  // namespace hdbf
