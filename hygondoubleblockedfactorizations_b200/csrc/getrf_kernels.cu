// GETRF pivot composition and row-permutation kernels (FP32).
//
// compose_swaps + apply_moves replace apply_panel_pivots_kernel
// (src/getrf/getrf_pivot_kernels.hip:14-45) and the host-side permutation
// batching (src/getrf/getrf_batched_pivot_internal.h:59-223): a LAPACK swap
// sequence is composed on the GPU into a list of (source, target) row moves,
// then applied to column tiles with a gather into shared memory followed by a
// scatter -- no host round trip.
#include <cfloat>
#include <climits>

#include "internal.h"

namespace hdbf {
namespace {

// ------------------------------------------------------------ compose swaps
constexpr int kComposeThreads = 1024;
constexpr int kComposeMaxK = 4096;  // swaps composed by the sorted-group kernels

__host__ __device__ constexpr int pow2_at_least(int v)
{
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

// Block-wide ordered compaction: items q = 0 .. total-1 in order, item q
// kept when pick(q, &s, &t) is true; kept items are written to src/tgt at
// base + (rank among kept items).  Returns the new base (uniform).
template <class Pick>
__device__ int emit_ordered(int total, int base, int* src, int* tgt, int* warp_tot, int* s_chunk,
                            Pick pick)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int q0 = 0; q0 < total; q0 += kComposeThreads) {
        const int q = q0 + tid;
        int s = 0, t = 0;
        const bool moved = q < total && pick(q, &s, &t);
        const unsigned ball = __ballot_sync(0xffffffffu, moved);
        const int within = __popc(ball & ((1u << lane) - 1u));
        if (lane == 0) warp_tot[warp] = __popc(ball);
        __syncthreads();
        if (tid == 0) {
            int run = 0;
            for (int wv = 0; wv < kComposeThreads / 32; ++wv) {
                const int c = warp_tot[wv];
                warp_tot[wv] = run;
                run += c;
            }
            *s_chunk = run;
        }
        __syncthreads();
        if (moved) {
            src[base + warp_tot[warp] + within] = s;
            tgt[base + warp_tot[warp] + within] = t;
        }
        base += *s_chunk;
        __syncthreads();
    }
    return base;
}

// Composition of a LAPACK swap sequence without replaying it.  Step t
// (t = 0 .. kk-1) exchanges the contents of position x_t = base + t with
// position bt[t] >= x_t.  Position x_t is never touched after step t, and a
// position p >= x_t is touched before step t only by the steps j < t with
// bt[j] = p.  So, with the (bt, t) pairs sorted:
//   prev(t) = the last j < t with bt[j] = bt[t]      (same-target group)
//   g(u)    = the last j < u with bt[j] = x_u        (who filled x_u before step u)
//   V(u)    = content of x_u just before step u = start(x_{root(u)}), root(u)
//             the end of the chain u -> g(u) -> g(g(u)) ... (pointer jumping)
// and the contents after the whole sequence are
//   position x_t:                 prev(t) >= 0 ? V(prev(t)) : start(bt[t])
//   target p >= base + kk (last t of its group): V(t).
// Results: nv[t] (content of x_t), keys[s] the sorted pairs, root[u] the chain
// ends; aux[t] holds prev(t).  start() must stay valid until the caller writes
// the new contents.
template <class Start>
__device__ void compose_sorted(const int* bt, int kk, int base, int P, unsigned long long* keys,
                               int* aux, int* root, int* nv, Start start)
{
    const int tid = threadIdx.x;
    for (int s = tid; s < P; s += kComposeThreads)
        keys[s] = s < kk ? ((unsigned long long)(unsigned)bt[s] << 32) | (unsigned)s : ~0ull;
    for (int u = tid; u < kk; u += kComposeThreads) root[u] = -1;
    __syncthreads();
    // bitonic sort, ascending (b, t)
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < P / 2; i += kComposeThreads) {
                const int lo = 2 * i - (i & (stride - 1));
                const int hi = lo + stride;
                const bool up = (lo & size) == 0;
                const unsigned long long a = keys[lo], b = keys[hi];
                if ((a > b) == up) {
                    keys[lo] = b;
                    keys[hi] = a;
                }
            }
            __syncthreads();
        }
    }
    for (int s = tid; s < kk; s += kComposeThreads) {
        const unsigned long long key = keys[s];
        const int b = (int)(key >> 32), t = (int)(key & 0xffffffffu);
        const bool has_prev = s > 0 && (int)(keys[s - 1] >> 32) == b;
        aux[t] = has_prev ? (int)(keys[s - 1] & 0xffffffffu) : -1;
        const int u = b - base;  // b is the swap-side position of step u
        if (u < kk && t < u) {
            const bool next_in = s + 1 < kk && (int)(keys[s + 1] >> 32) == b;
            if (!next_in || (int)(keys[s + 1] & 0xffffffffu) == u) root[u] = t;
        }
    }
    __syncthreads();
    for (int u = tid; u < kk; u += kComposeThreads)
        if (root[u] < 0) root[u] = u;
    __syncthreads();
    // Pointer jumping: every root[] value is an ancestor, so reading an entry
    // another thread is updating in the same round is harmless; a round in
    // which nothing changes has read only settled values.
    for (;;) {
        int changed = 0;
        for (int u = tid; u < kk; u += kComposeThreads) {
            const int r = root[u], rr = root[r];
            if (rr != r) {
                root[u] = rr;
                changed = 1;
            }
        }
        if (!__syncthreads_or(changed)) break;
    }
    for (int t = tid; t < kk; t += kComposeThreads) {
        const int p = aux[t];
        nv[t] = p >= 0 ? start(base + root[p]) : start(bt[t]);
    }
    __syncthreads();
}

// Shared-memory layout of the sorted-group kernels (after `lead` ints):
// keys[P] (8-byte aligned), then bt, aux, root, nv (kk ints each).
__host__ __device__ inline size_t compose_sorted_bytes(int lead, int kk)
{
    const size_t head = ((size_t)lead * sizeof(int) + 15) / 16 * 16;
    return head + (size_t)pow2_at_least(kk < 1 ? 1 : kk) * 8 + 4 * (size_t)kk * sizeof(int);
}

// Swaps ipiv[0..k) (rows local after subtracting 1 + ipiv_minus) composed
// into the row moves of A(0:m, :): rows [0, k) in order, then the distinct
// pivot rows >= k in increasing order.  Touches O(k) rows only.
__global__ void __launch_bounds__(kComposeThreads)
compose_swaps_kernel(const int* __restrict__ ipiv, int k, int ipiv_minus, int m, int* src,
                     int* tgt, int* count, int* info, int* err)
{
    extern __shared__ __align__(16) unsigned char craw[];
    __shared__ int warp_tot[kComposeThreads / 32];
    __shared__ int s_bad, s_chunk;
    const int P = pow2_at_least(k);
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(craw);
    int* bt = reinterpret_cast<int*>(keys + P);
    int* aux = bt + k;
    int* root = aux + k;
    int* nv = root + k;
    const int tid = threadIdx.x;
    if (tid == 0) s_bad = 0;
    __syncthreads();
    for (int i = tid; i < k; i += kComposeThreads) {
        const int b = ipiv[i] - 1 - ipiv_minus;
        if (b < i || b >= m) s_bad = 1;
        bt[i] = b;
    }
    __syncthreads();
    if (s_bad) {
        if (tid == 0) {
            *count = 0;
            if (info) atomicExch(info, -1);
            atomicCAS(err, 0, kErrBadPivot);
        }
        return;
    }
    compose_sorted(bt, k, 0, P, keys, aux, root, nv, [](int x) { return x; });
    int base = emit_ordered(k, 0, src, tgt, warp_tot, &s_chunk, [&](int q, int* s, int* t) {
        *s = nv[q];
        *t = q;
        return nv[q] != q;
    });
    base = emit_ordered(k, base, src, tgt, warp_tot, &s_chunk, [&](int q, int* s, int* t) {
        const unsigned long long key = keys[q];
        const int b = (int)(key >> 32);
        if (b < k || (q + 1 < k && (int)(keys[q + 1] >> 32) == b)) return false;
        *s = root[(int)(key & 0xffffffffu)];
        *t = b;
        return *s != b;
    });
    if (tid == 0) *count = base;
}

// The same composition by replaying the swaps in one thread, for sequences
// longer than kComposeMaxK: perm[m] (shared memory, or global scratch when
// it does not fit), then the same move order.
__global__ void __launch_bounds__(kComposeThreads)
compose_swaps_serial_kernel(const int* __restrict__ ipiv, int k, int ipiv_minus, int m,
                            int* src, int* tgt, int* count, int* gperm, int use_smem, int* info,
                            int* err)
{
    extern __shared__ int sperm[];
    __shared__ int warp_tot[kComposeThreads / 32];
    __shared__ int s_bad, s_chunk;
    int* perm = use_smem ? sperm : gperm;
    const int tid = threadIdx.x;
    if (tid == 0) s_bad = 0;
    __syncthreads();
    for (int q = tid; q < m; q += kComposeThreads) perm[q] = q;
    for (int i = tid; i < k; i += kComposeThreads) {
        const int b = ipiv[i] - 1 - ipiv_minus;
        if (b < i || b >= m) s_bad = 1;
    }
    __syncthreads();
    if (s_bad) {
        if (tid == 0) {
            *count = 0;
            if (info) atomicExch(info, -1);
            atomicCAS(err, 0, kErrBadPivot);
        }
        return;
    }
    if (tid == 0) {
        for (int i = 0; i < k; ++i) {
            const int b = ipiv[i] - 1 - ipiv_minus;
            const int t = perm[i];
            perm[i] = perm[b];
            perm[b] = t;
        }
    }
    __syncthreads();
    int base = emit_ordered(k, 0, src, tgt, warp_tot, &s_chunk, [&](int q, int* s, int* t) {
        *s = perm[q];
        *t = q;
        return perm[q] != q;
    });
    // pivot rows >= k: each distinct row once, in increasing row order
    base = emit_ordered(m - k, base, src, tgt, warp_tot, &s_chunk, [&](int q, int* s, int* t) {
        *s = perm[k + q];
        *t = k + q;
        return perm[k + q] != k + q;
    });
    if (tid == 0) *count = base;
}

// ------------------------------------------------------------ apply moves
constexpr int kApplyThreads = 256;

// Columns [blockIdx.x*cpc, +cpc): gather every source row into shared memory,
// then scatter to the targets.  Sources and targets are the same row set, so
// reading everything before writing anything is race-free per column.
__global__ void __launch_bounds__(kApplyThreads)
apply_moves_smem_kernel(float* A, long long lda, int ncols, const int* __restrict__ src,
                        const int* __restrict__ tgt, const int* __restrict__ count, int cpc,
                        int cap)
{
    extern __shared__ float buf[];  // cpc * cap values, then cap sources, cap targets
    int* s_src = reinterpret_cast<int*>(buf + (size_t)cpc * cap);
    int* s_tgt = s_src + cap;
    const int cnt = min(*count, cap);
    if (cnt <= 0) return;
    const int c0 = blockIdx.x * cpc;
    const int nc = min(cpc, ncols - c0);
    for (int i = threadIdx.x; i < cnt; i += kApplyThreads) {
        s_src[i] = src[i];
        s_tgt[i] = tgt[i];
    }
    __syncthreads();
    // Flattened (column, move) space, eight independent loads in flight.
    const int total = nc * cnt;
    const float* base = A + (long long)c0 * lda;
    int e = threadIdx.x;
    for (; e + 7 * kApplyThreads < total; e += 8 * kApplyThreads) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int q = e + u * kApplyThreads, cc = q / cnt, i = q - cc * cnt;
            v[u] = base[(long long)cc * lda + s_src[i]];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int q = e + u * kApplyThreads, cc = q / cnt, i = q - cc * cnt;
            buf[cc * cap + i] = v[u];
        }
    }
    for (; e < total; e += kApplyThreads) {
        const int cc = e / cnt, i = e - cc * cnt;
        buf[cc * cap + i] = base[(long long)cc * lda + s_src[i]];
    }
    __syncthreads();
    float* wbase = A + (long long)c0 * lda;
    for (int q = threadIdx.x; q < total; q += kApplyThreads) {
        const int cc = q / cnt, i = q - cc * cnt;
        wbase[(long long)cc * lda + s_tgt[i]] = buf[cc * cap + i];
    }
}

__global__ void gather_rows_kernel(const float* A, long long lda, int ncols,
                                   const int* __restrict__ src, const int* __restrict__ count,
                                   int cap, float* temp)
{
    const int cnt = min(*count, cap);
    const long long total = (long long)cnt * ncols;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % cnt);
        const long long c = idx / cnt;
        temp[c * cap + i] = A[c * lda + src[i]];
    }
}

__global__ void scatter_rows_kernel(float* A, long long lda, int ncols,
                                    const int* __restrict__ tgt, const int* __restrict__ count,
                                    int cap, const float* temp)
{
    const int cnt = min(*count, cap);
    const long long total = (long long)cnt * ncols;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % cnt);
        const long long c = idx / cnt;
        A[c * lda + tgt[i]] = temp[c * cap + i];
    }
}

}  // namespace

// Dynamic shared-memory opt-ins, set once per handle creation (never inside a
// stream capture).
void configure_getrf_kernels(hdbf_context* ctx)
{
    const size_t cap4 = ctx->max_smem_optin > 4096 ? ctx->max_smem_optin - 4096 : 0;
    cudaFuncSetAttribute(compose_swaps_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cap4);
    cudaFuncSetAttribute(compose_swaps_serial_kernel,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap4);
    cudaFuncSetAttribute(apply_moves_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cap4);
    cudaGetLastError();
}

hdbf_status compose_swaps(hdbf_context* ctx, const int* ipiv, int k, int ipiv_minus, int m,
                          int* src, int* tgt, int* count, int* gperm, int* info)
{
    if (k <= 0 || m <= 0) return HDBF_STATUS_SUCCESS;
    if (k > m) return HDBF_STATUS_INVALID_VALUE;
    const size_t cap = ctx->max_smem_optin > 4096 ? ctx->max_smem_optin - 4096 : 0;
    if (k <= kComposeMaxK) {
        const size_t smem = compose_sorted_bytes(0, k);
        ProfScope prof(ctx, kClsCompose, 0.0, 12.0 * k);
        compose_swaps_kernel<<<1, kComposeThreads, smem, ctx->stream>>>(
            ipiv, k, ipiv_minus, m, src, tgt, count, info, ctx->dev_small + kSmallErr);
        ctx->launches++;
        return last_cuda(ctx);
    }
    const size_t smem = (size_t)m * sizeof(int);
    const int use_smem = smem <= cap ? 1 : 0;
    if (!use_smem && !gperm) return HDBF_STATUS_INVALID_VALUE;
    ProfScope prof(ctx, kClsCompose, 0.0, 4.0 * k + 8.0 * m);
    compose_swaps_serial_kernel<<<1, kComposeThreads, use_smem ? smem : 0, ctx->stream>>>(
        ipiv, k, ipiv_minus, m, src, tgt, count, gperm, use_smem, info,
        ctx->dev_small + kSmallErr);
    ctx->launches++;
    return last_cuda(ctx);
}

hdbf_status apply_moves(hdbf_context* ctx, float* A, long long lda, int ncols,
                        const int* src, const int* tgt, const int* count, int max_moves,
                        float* temp, long long temp_cols)
{
    if (ncols <= 0 || max_moves <= 0) return HDBF_STATUS_SUCCESS;
    const size_t per_col = (size_t)max_moves * sizeof(float);
    const size_t idx_bytes = 2 * (size_t)max_moves * sizeof(int);
    const size_t budget = 64 * 1024;
    const size_t hard_cap = ctx->max_smem_optin > 4096 ? ctx->max_smem_optin - 4096 : 0;
    ProfScope prof(ctx, kClsMoves, 0.0, 8.0 * (double)max_moves * ncols);
    if (per_col + idx_bytes <= hard_cap) {
        int cpc = (int)((budget > idx_bytes ? budget - idx_bytes : 0) / per_col);
        if (cpc < 1) cpc = 1;
        if (cpc > 16) cpc = 16;
        const int grid = (ncols + cpc - 1) / cpc;
        apply_moves_smem_kernel<<<grid, kApplyThreads, per_col * cpc + idx_bytes, ctx->stream>>>(
            A, lda, ncols, src, tgt, count, cpc, max_moves);
        ctx->launches++;
        return last_cuda(ctx);
    }
    if (!temp || temp_cols <= 0) return HDBF_STATUS_INVALID_VALUE;
    for (long long c = 0; c < ncols; c += temp_cols) {
        const int nc = (int)((ncols - c) < temp_cols ? (ncols - c) : temp_cols);
        const long long total = (long long)nc * max_moves;
        const int grid = (int)((total + 255) / 256 < 65535 ? (total + 255) / 256 : 65535);
        gather_rows_kernel<<<grid, 256, 0, ctx->stream>>>(A + c * lda, lda, nc, src, count,
                                                          max_moves, temp);
        scatter_rows_kernel<<<grid, 256, 0, ctx->stream>>>(A + c * lda, lda, nc, tgt, count,
                                                           max_moves, temp);
        ctx->launches += 2;
    }
    return last_cuda(ctx);
}

}  // namespace hdbf
