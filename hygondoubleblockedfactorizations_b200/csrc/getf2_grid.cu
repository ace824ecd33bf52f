// Grid-wide GETRF panel leaf: partially pivoted LU of an m x w column block too
// tall for one cluster (getf2_cluster.cu), FP32 and FP64, replacing
// rocsolver_sgetrf's unblocked leaf on the tall panel
// (src/getrf/getrf_pivot_internal.h:17-39).  One cooperative launch, at most one
// CTA per SM.
//
// What bounds it is the exchange of one pivot per column through L2: the CTAs'
// candidates out and back, then the winner's row back, two dependent trips of
// ~0.7 us.  Everything else is kept off that chain:
//   - rows live in registers (thread t owns local rows t, t + 256, ...), shifted by
//     one column per step so that the loop is rolled; a row never moves but
//     carries its position, and is stored to where it ended up once, at the end;
//   - a column's pivot candidate needs only that column, so the rest of the
//     previous step's rank-1 update runs after the candidate is published;
//   - words are published without fences: each 64-bit word is
//     [tag : 32 | value : 32], read whole, and its tag (launch epoch, column)
//     proves its freshness.
// A CTA publishes its candidate's key (magnitude, position) first and the row
// behind it; every CTA reads all keys (thread q watches CTA q), reduces them, and
// reads the winner's row.  Candidates compare as in getf2_cluster.cu (largest |a|,
// lowest position on ties), and every element sees the same operations in the
// same order, so the two kernels agree bit for bit.
// Slots alternate by column parity.  A CTA rewrites a parity only after every CTA
// has published the following column, that is after all of them finished
// reading it.  The last CTA to finish advances the epoch.
// Rows per CTA: 256 (one row a thread) while the SMs hold the panel that way.
// Leaves are as wide as the registers allow: 512 bytes of a row with one row a
// thread, 256 bytes with two or three, 128 bytes with up to six.
// Measured per column (n x n factorization, all heights): 1.9 us at n = 4096, 2.0
// at 32768 (FP32), 2.1 in FP64, against 4.1-6.5 us of a kernel that kept the rows in
// shared memory and swapped them every column; 128 or 192 rows per CTA are 1-3 %
// slower.  The panels of an FP32 LU of order 32768 went from 124 to 64 ms.
// Polls are bounded by the handle's limit; an expired one records a timeout and
// the CTA stops factoring.
#include <algorithm>

#include "getf2_common.cuh"
#include "internal.h"

namespace hdbf {
namespace {

constexpr int kGridThreads = 256;
constexpr int kGridWarps = kGridThreads / 32;
constexpr int kGridMax = 256;   // CTAs: one per thread when the keys are read
constexpr int kHeadWords = 4;   // key words of a slot
constexpr int kRowWords = 128;  // row words of a slot (512 bytes of a row)
constexpr int kSlotWords = kHeadWords + kRowWords;

__device__ __forceinline__ unsigned long long load_word(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_word(unsigned long long* p, unsigned tag, unsigned v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p),
                 "l"(((unsigned long long)tag << 32) | v)
                 : "memory");
}

template <class T>
struct Key {
    Mag<T> mag;
    int row;
    int cta;
};

template <class T, int W>
struct GridSmem {
    alignas(16) T own[W];      // this CTA's candidate row
    alignas(16) T urow[2][W];  // pivot rows of the last two columns, from the diagonal on
    Key<T> warp_key[kGridWarps];
    Key<T> grid_key[kGridWarps];
    int stop_keys, stop_row;  // an expired poll of keys, of the row: each is set and read
                              // between its own two block barriers
};

template <class T, int W, int R>
__global__ void __launch_bounds__(kGridThreads, 1)
getf2_grid_kernel(int m, int w, T* A, long long lda, int rpc, int* ipiv, int ipiv_add, int* info,
                  int info_base, unsigned long long* slots, unsigned* epoch_ptr,
                  unsigned* done_ptr, int* err, int pivot)
{
    constexpr int kWords = W * (int)sizeof(T) / 4;     // words of a row
    constexpr int kKeyWords = 1 + (int)sizeof(T) / 4;  // magnitude, position
    constexpr int V = 16 / (int)sizeof(T);             // values of a 16-byte chunk
    struct alignas(16) Chunk {
        T x[V];
    };
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GridSmem<T, W>& sm = *reinterpret_cast<GridSmem<T, W>*>(smem_raw);
    T* tile = reinterpret_cast<T*>(smem_raw + sizeof(GridSmem<T, W>));  // finished entries
    const int ldt = rpc | 1;

    const int G = gridDim.x, cta = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = cta * rpc;
    const int nr = max(0, min(m, r0 + rpc) - r0);
    const int steps = min(m, w);
    const unsigned epoch = *reinterpret_cast<volatile unsigned*>(epoch_ptr);
    const unsigned limit = spin_limit_of(err);
    auto slot_of = [&](int par, int q) {
        return slots + ((long long)par * kGridMax + q) * kSlotWords;
    };
    // One more fruitless poll; true when it was the last allowed.
    auto expired = [&](unsigned& polls, int& stop) {
        if (++polls >= limit) {
            atomicCAS(err, 0, kErrTimeout);
            stop = 1;
            return true;
        }
        if (polls > 256) __nanosleep(32);
        return false;
    };

    T a[R][W];   // columns J, J + 1, ...; all but the first lack the last step's update
    T l[R];      // that step's multipliers
    int pos[R];  // the row's position; below J once it has been a pivot row
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = tid + kGridThreads * i;
        pos[i] = r < nr ? r0 + r : -1;
        l[i] = T(0);
#pragma unroll
        for (int c = 0; c < W; ++c)
            a[i][c] = (r < nr && c < w) ? A[(long long)c * lda + r0 + r] : T(0);
    }
    if (tid == 0) sm.stop_keys = sm.stop_row = 0;

#pragma unroll 1
    for (int J = 0; J < steps; ++J) {
        const int par = J & 1;
        const unsigned tag = (epoch << 8) | (unsigned)(J + 1);
        unsigned long long* slot = slot_of(par, cta);
        // 1. this CTA's candidate for column J
        Mag<T> mv, vb = 0;
        int mrow, row = INT_MAX;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const Mag<T> b = mag_bits(a[i][0]);
            if ((pivot ? pos[i] >= J : pos[i] == J) &&
                (row == INT_MAX || b > vb || (b == vb && pos[i] < row))) {
                vb = b;
                row = pos[i];
            }
        }
        warp_argmax(vb, row, mv, mrow);
        if (lane == 0) sm.warp_key[warp] = Key<T>{mv, mrow, 0};
        __syncthreads();
        vb = 0;
        row = INT_MAX;
        if (lane < kGridWarps) {
            vb = sm.warp_key[lane].mag;
            row = sm.warp_key[lane].row;
        }
        warp_argmax(vb, row, mv, mrow);
        const unsigned who = __ballot_sync(0xffffffffu, lane < kGridWarps && row == mrow);
        const int from = who ? __ffs(who) - 1 : 0;
        if (warp == from && lane < kKeyWords)
            store_word(slot + lane, tag,
                       lane == kKeyWords - 1 ? (unsigned)mrow
                                             : (unsigned)((unsigned long long)mv >> (32 * lane)));
        // the rest of the previous step's update, behind the key
        if (J > 0) {
            const Chunk* up = reinterpret_cast<const Chunk*>(sm.urow[par ^ 1]);
            const int left = w - J;  // columns from J on
#pragma unroll
            for (int q = 0; q < W / V; ++q) {
                if (q * V > left) break;
                const Chunk u = up[q];
#pragma unroll
                for (int e = 0; e < V; ++e) {
                    const int c = q * V + e;  // column J - 1 + c
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        if (c >= 2) a[i][c - 1] = fma_t(-l[i], u.x[e], a[i][c]);
                    }
                }
            }
        }
        if (warp == from) {  // the candidate's row
#pragma unroll
            for (int i = 0; i < R; ++i) {
                if (pos[i] == mrow) {
#pragma unroll
                    for (int q = 0; q < W / V; ++q) {
                        Chunk x;
#pragma unroll
                        for (int e = 0; e < V; ++e) x.x[e] = a[i][q * V + e];
                        reinterpret_cast<Chunk*>(sm.own)[q] = x;
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int k = lane; k < kWords; k += 32)
                store_word(slot + kHeadWords + k, tag, reinterpret_cast<const unsigned*>(sm.own)[k]);
        }
        // 2. every CTA's key
        vb = 0;
        row = INT_MAX;
        if (tid < G) {
            const unsigned long long* s = slot_of(par, tid);
            unsigned long long v[kKeyWords];
            unsigned polls = 0;
            bool fresh;
            do {
#pragma unroll
                for (int k = 0; k < kKeyWords; ++k) v[k] = load_word(s + k);
                fresh = true;
#pragma unroll
                for (int k = 0; k < kKeyWords; ++k) fresh &= (unsigned)(v[k] >> 32) == tag;
            } while (!fresh && !expired(polls, sm.stop_keys));
            if (fresh) {
                vb = (unsigned)v[0];
                if (sizeof(T) == 8) vb |= (Mag<T>)(v[kKeyWords - 2] << 32);
                row = (int)(unsigned)v[kKeyWords - 1];
            }
        }
        warp_argmax(vb, row, mv, mrow);
        {
            const unsigned b = __ballot_sync(0xffffffffu, row == mrow);
            if (lane == 0) sm.grid_key[warp] = Key<T>{mv, mrow, warp * 32 + __ffs(b) - 1};
        }
        __syncthreads();
        if (sm.stop_keys) break;
        vb = 0;
        row = INT_MAX;
        int src = 0;
        if (lane < kGridWarps) {
            vb = sm.grid_key[lane].mag;
            row = sm.grid_key[lane].row;
            src = sm.grid_key[lane].cta;
        }
        warp_argmax(vb, row, mv, mrow);
        {
            const unsigned b = __ballot_sync(0xffffffffu, lane < kGridWarps && row == mrow);
            src = __shfl_sync(0xffffffffu, src, b ? __ffs(b) - 1 : 0);
        }
        // 3. the winner's row
        if (tid < kWords) {
            const unsigned long long* s = slot_of(par, src) + kHeadWords + tid;
            unsigned long long v;
            unsigned polls = 0;
            while ((unsigned)((v = load_word(s)) >> 32) != tag && !expired(polls, sm.stop_row)) {}
            reinterpret_cast<unsigned*>(sm.urow[par])[tid] = (unsigned)v;
        }
        T rcp = Bits<T>::rcp(Bits<T>::val(mv));
        __syncthreads();
        if (sm.stop_row) break;
        const int p = mrow >= J && mrow < m ? mrow : J;
        const T* urow = sm.urow[par];
        const T piv = urow[0];
        const T u1 = W > 1 ? urow[1] : T(0);
        const bool nz = piv != T(0);
        rcp = piv < T(0) ? -rcp : (piv == piv ? rcp : piv);
        const bool recip = abs_t(piv) >= min_normal(piv) || piv != piv;
#pragma unroll
        for (int i = 0; i < R; ++i) l[i] = a[i][0] * rcp;
        if (!(nz && recip)) {  // a zero or subnormal pivot
#pragma unroll
            for (int i = 0; i < R; ++i) l[i] = nz ? a[i][0] / piv : a[i][0];
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = tid + kGridThreads * i;
            const unsigned b = __ballot_sync(0xffffffffu, pos[i] == p);
            if (b) {  // the pivot row is in this warp: its U entries, a lane per column
                T* x = tile + r - lane + __ffs(b) - 1;
                for (int c = lane; c < w - J; c += 32) x[(J + c) * ldt] = urow[c];
            }
            if (pos[i] == p) pos[i] = J;
            else if (pos[i] == J) pos[i] = p;
            if (pos[i] > J) tile[J * ldt + r] = l[i];
            a[i][0] = fma_t(-l[i], u1, a[i][1]);
        }
        if (cta == 0 && tid == kGridThreads - 1) {
            if (pivot) ipiv[J] = p + 1 + ipiv_add;
            if (!nz && info) atomicCAS(info, 0, info_base + J + 1);
        }
    }
    __syncthreads();
    // Every CTA published the last column, so all rows have long been read.
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = tid + kGridThreads * i;
        if (r < nr) {
            T* x = A + pos[i];
#pragma unroll 8
            for (int c = 0; c < w; ++c) x[(long long)c * lda] = tile[c * ldt + r];
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(done_ptr, 1u) + 1u == (unsigned)G) {
            atomicExch(done_ptr, 0u);
            atomicAdd(epoch_ptr, 1u);
        }
    }
}

template <class T, int W>
size_t grid_smem(int rpc, int w)
{
    return sizeof(GridSmem<T, W>) + sizeof(T) * (size_t)(rpc | 1) * w;
}

// Rows per thread for a leaf of `bytes` bytes of a row.
int grid_rows(int bytes) { return bytes > 256 ? 1 : (bytes > 128 ? 3 : 6); }

template <class T, int BYTES, int R>
cudaError_t launch_grid(hdbf_context* ctx, int G, int rpc, int m, int w, T* A, long long lda,
                        int* ipiv, int ipiv_add, int* info, int info_base, int pivot)
{
    constexpr int W = BYTES / (int)sizeof(T);
    unsigned long long* slots = reinterpret_cast<unsigned long long*>(ws_panel(ctx));
    unsigned* epoch = reinterpret_cast<unsigned*>(ctx->dev_small + kSmallEpoch);
    unsigned* done = reinterpret_cast<unsigned*>(ctx->dev_small + kSmallDone);
    int* err = ctx->dev_small + kSmallErr;
    void* args[] = {&m, &w, &A, &lda, &rpc, &ipiv, &ipiv_add, &info, &info_base,
                    &slots, &epoch, &done, &err, &pivot};
    return cudaLaunchCooperativeKernel((const void*)getf2_grid_kernel<T, W, R>, dim3(G),
                                       dim3(kGridThreads), args, grid_smem<T, W>(rpc, w),
                                       ctx->stream);
}

template <class T>
hdbf_status getf2_grid_t(hdbf_context* ctx, int m, int w, T* A, long long lda, int* ipiv,
                         int ipiv_add, int* info, int info_base, bool pivot)
{
    if (m <= 0 || w <= 0) return HDBF_STATUS_SUCCESS;
    if (w > getf2_grid_leaf(ctx, m, (int)sizeof(T))) return HDBF_STATUS_NOT_SUPPORTED;
    HDBF_TRY(ensure_ws(ctx, 64));
    const int bytes = w * (int)sizeof(T);
    const int most = grid_rows(bytes) * kGridThreads;
    const int target = std::min(ctx->panel_rows > 0 ? ctx->panel_rows : kGridThreads, most);
    const int G = std::min((m + target - 1) / target, std::min(ctx->sm_count, kGridMax));
    const int rpc = (m + G - 1) / G;
    const int piv = pivot ? 1 : 0;
    ProfScope prof(ctx, kClsPanel, (double)m * w * w - (double)w * w * w / 3.0,
                   2.0 * sizeof(T) * m * w);
    cudaError_t e;
#define HDBF_GRID(BYTES, R)                                                                  \
    launch_grid<T, BYTES, R>(ctx, G, rpc, m, w, A, lda, ipiv, ipiv_add, info, info_base, piv)
    if (bytes > 256) e = HDBF_GRID(512, 1);
    else if (rpc <= kGridThreads) e = HDBF_GRID(256, 1);
    else if (bytes > 128) e = rpc <= 2 * kGridThreads ? HDBF_GRID(256, 2) : HDBF_GRID(256, 3);
    else e = rpc <= 3 * kGridThreads ? HDBF_GRID(128, 3) : HDBF_GRID(128, 6);
#undef HDBF_GRID
    ctx->launches++;
    if (e != cudaSuccess) {
        cudaGetLastError();
        return HDBF_STATUS_CUDA_ERROR;
    }
    return HDBF_STATUS_SUCCESS;
}

template <class T>
void configure_grid(hdbf_context* ctx)
{
    const int cap = ctx->max_smem_optin;
    constexpr int E = (int)sizeof(T);
    for (const void* k : {(const void*)getf2_grid_kernel<T, 512 / E, 1>,
                          (const void*)getf2_grid_kernel<T, 256 / E, 1>,
                          (const void*)getf2_grid_kernel<T, 256 / E, 2>,
                          (const void*)getf2_grid_kernel<T, 256 / E, 3>,
                          (const void*)getf2_grid_kernel<T, 128 / E, 3>,
                          (const void*)getf2_grid_kernel<T, 128 / E, 6>})
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
    cudaGetLastError();
}

}  // namespace

void configure_grid_panel(hdbf_context* ctx)
{
    configure_grid<float>(ctx);
    configure_grid<double>(ctx);
}

size_t getf2_grid_scratch_bytes()
{
    return align_up((size_t)2 * kGridMax * kSlotWords * sizeof(unsigned long long), 256);
}

// Widest leaf (a power of two) that the grid holds at height m; 0 when it holds none.
int getf2_grid_leaf(hdbf_context* ctx, int m, int elem)
{
    const int G = std::min(ctx->sm_count, kGridMax);
    for (int bytes = 512; bytes >= 128; bytes /= 2)
        if ((m + G - 1) / G <= grid_rows(bytes) * kGridThreads) return bytes / elem;
    return 0;
}

hdbf_status getf2_grid(hdbf_context* ctx, int m, int w, float* A, long long lda, int* ipiv,
                       int ipiv_add, int* info, int info_base, bool pivot)
{
    return getf2_grid_t(ctx, m, w, A, lda, ipiv, ipiv_add, info, info_base, pivot);
}

hdbf_status getf2_grid(hdbf_context* ctx, int m, int w, double* A, long long lda, int* ipiv,
                       int ipiv_add, int* info, int info_base, bool pivot)
{
    return getf2_grid_t(ctx, m, w, A, lda, ipiv, ipiv_add, info, info_base, pivot);
}

}  // namespace hdbf
