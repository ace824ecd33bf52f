// Cholesky of a diagonal block of order n <= 1024, optionally with the inverse of
// its factor.
//
// Replaces the reference's rocsolver_spotrf call on the diagonal block
// (src/potrf/double_blocked_potrf.cpp:34-56, call :334).  The block is cut
// into 64 x 64 tiles (NT = ceil(n / 64) <= 16) and factored right-looking by one
// thread-block cluster (potrf_cluster_kernel): CTA 0 owns the chain -- factor and
// invert tile (k, k) (tile64.cuh), solve tile (k+1, k) against it, update tile
// (k+1, k+1), all in its shared memory -- and the other CTAs solve the rest of
// column k, then update the trailing tiles while CTA 0 factors the next diagonal
// tile.  Tiles travel through L2 (each is read by several CTAs); two barriers per
// tile column are mbarriers in every CTA's shared memory on which all CTAs arrive
// remotely.  What bounds it is CTA 0's chain, ~15 us a tile (factor 5.9, inverse
// 2.8, products 3.2, the rest loads, stores and barriers): n = 256 57 us, n = 512
// 120 us; with a grid-wide barrier twice per tile column and every step through L2
// it took 96 and 207 us.
// With the inverse requested, W = L^{-1} (lower, the strictly upper tiles zeroed)
// is formed by a second, cooperative launch (tile_inverse_kernel) by recursive
// doubling over tile blocks: for siblings A and C, W(C,A) = -W(C,C) (L(C,A)
// W(A,A)), two GEMM phases per level with bounded grid barriers.
//
// Pivot test and info follow LAPACK xPOTRF: the first column whose updated
// diagonal is not > 0 (or is NaN) stops the factorization and info =
// info_base + column + 1 (first failure wins); a block whose info is already
// non-zero is left untouched.  The inverses of tiles that were not factored are
// those of the tiles as they stand: what the panel solve makes of the rest of the
// matrix then depends on the matrix alone.  Every wait is bounded by the handle's poll limit:
// on expiry the kernel records a timeout and the remaining work is skipped; a
// cluster's CTAs then meet at a hardware barrier, so that none leaves while
// another may still arrive in its shared memory.
#include <algorithm>

#include "internal.h"
#include "pair.cuh"
#include "tile64.cuh"

namespace hdbf {
namespace {

constexpr int kT = 64;        // tile
constexpr int kThreads = 256;
constexpr int kMaxNT = 16;    // n <= 1024
constexpr int kLdS = tile64::kLd;  // padded shared row (float4-aligned)

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

struct Sync {
    unsigned* ctr;
    int* fail;
    int* abort_flag;
    int* err;
    unsigned G;
    unsigned count;  // barriers passed by this CTA
    unsigned limit;  // poll limit (the handle's, spin_limit_of)
};

// Grid barrier: arrive (counter += 1 per CTA), wait until all G CTAs of this
// round arrived.  Bounded; once any CTA gave up, later waits return at once.
__device__ void grid_barrier(Sync& s)
{
    __syncthreads();
    s.count += 1;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(s.ctr, 1u);
        const unsigned target = s.count * s.G;
        unsigned polls = 0;
        while (ld_acquire_u32(s.ctr) < target) {
            if (*reinterpret_cast<volatile int*>(s.abort_flag)) break;
            if (++polls > s.limit) {
                atomicCAS(s.err, 0, kErrTimeout);
                atomicExch(s.abort_flag, 1);
                break;
            }
            if (polls > 64) __nanosleep(64);
        }
        __threadfence();
    }
    __syncthreads();
}

// Two 64 x 64 tiles into shared memory, every global load of the thread in
// flight before the first shared store (the tiles live in L2, so the loads'
// latency, not their bandwidth, sets the cost).  Tile X (X = A, B) is the
// column-major block src (leading dimension ld, entries outside rows x cols
// read as zero); TX = false stores it k-major, dst[k][m] = src(m, k), and
// TX = true transposed, dst[k][n] = src(k, n), both with row pitch kLdS.
struct TileSrc {
    const float* src;
    long long ld;
    int rows, cols;
};
template <bool TA, bool TB>
__device__ __forceinline__ void load_pair(float* dA, TileSrc a, float* dB, TileSrc b)
{
    constexpr int kPer = kT * kT / kThreads;  // 16 elements per thread and tile
    float va[kPer], vb[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int q = threadIdx.x + u * kThreads, c = q >> 6, r = q & 63;
        va[u] = (r < a.rows && c < a.cols) ? __ldcg(a.src + (long long)c * a.ld + r) : 0.f;
        vb[u] = (r < b.rows && c < b.cols) ? __ldcg(b.src + (long long)c * b.ld + r) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int q = threadIdx.x + u * kThreads, c = q >> 6, r = q & 63;
        dA[TA ? r * kLdS + c : c * kLdS + r] = va[u];
        dB[TB ? r * kLdS + c : c * kLdS + r] = vb[u];
    }
}

// acc[i][j] += sum_k As[k][r4 + i] * Bs[k][c4 + j]: rows r4 = 4 (tid & 15) in
// consecutive lanes (whole lines of C), columns c4 = 4 (tid >> 4); packed FMAs.  kmax: a
// multiple of 8, uniform in a warp.
__device__ __forceinline__ void tile_mma(float acc[4][4], const float* As, const float* Bs,
                                         int kmax = kT)
{
    const int r4 = (threadIdx.x & 15) * 4, c4 = (threadIdx.x >> 4) * 4;
    Two<float> s[2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        s[0][j] = Two<float>::make(acc[0][j], acc[1][j]);
        s[1][j] = Two<float>::make(acc[2][j], acc[3][j]);
    }
#pragma unroll 8
    for (int k = 0; k < kmax; ++k) {
        Two<float> a0, a1;
        load_pairs(As + k * kLdS + r4, a0, a1);
        const float4 b = *reinterpret_cast<const float4*>(Bs + k * kLdS + c4);
        const float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const Two<float> bb = Two<float>::make(bv[j], bv[j]);
            s[0][j].fma(a0, bb);
            s[1][j].fma(a1, bb);
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        s[0][j].get(acc[0][j], acc[1][j]);
        s[1][j].get(acc[2][j], acc[3][j]);
    }
}

// ------------------------------------------------------------ cluster kernel
__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Column-major tile src (leading dimension ld, zero outside rows x cols) into
// dst[c * kLdS + r], through L2 only: other CTAs write these tiles.  Whole,
// aligned tiles go by cp.async; the caller commits and waits either way.
__device__ __forceinline__ void fetch_tile(float* dst, TileSrc t)
{
    const bool vec = t.rows == kT && t.cols == kT && t.ld % 4 == 0 &&
                     (reinterpret_cast<uintptr_t>(t.src) & 15u) == 0;
    if (vec) {
#pragma unroll
        for (int u = 0; u < kT * kT / 4 / kThreads; ++u) {
            const int q = threadIdx.x + u * kThreads, c = q >> 4, r = (q & 15) * 4;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                             smem_addr(dst + c * kLdS + r)),
                         "l"(t.src + (long long)c * t.ld + r)
                         : "memory");
        }
    } else {
        float v[kT * kT / kThreads];
#pragma unroll
        for (int u = 0; u < kT * kT / kThreads; ++u) {
            const int q = threadIdx.x + u * kThreads, c = q >> 6, r = q & 63;
            v[u] = (r < t.rows && c < t.cols) ? __ldcg(t.src + (long long)c * t.ld + r) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kT * kT / kThreads; ++u) {
            const int q = threadIdx.x + u * kThreads;
            dst[(q >> 6) * kLdS + (q & 63)] = v[u];
        }
    }
}
__device__ __forceinline__ void fetch_commit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void fetch_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct ClusterSmem {
    float tile[4][kT * kLdS];  // CTA 0: S, W, A(k+1,k), X; others: two pairs of operands
    float X[tile64::kScratch];
    float rd[kT];
    unsigned long long bar[2];
    int fail_col, stop;
};

// All CTAs of the cluster arrive on every CTA's barrier; the wait is bounded.
struct ClusterBarrier {
    ClusterSmem* sm;
    int C;
    unsigned limit;
    int* err;
    unsigned phase[2];
    __device__ void arrive(int b)
    {
        __syncthreads();
        if ((int)threadIdx.x < C)
            asm volatile(
                "{\n\t.reg .b32 ra;\n\t"
                "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
                "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [ra];\n\t}" ::"r"(
                    smem_addr(&sm->bar[b])),
                "r"((int)threadIdx.x)
                : "memory");
    }
    // false: the wait ran out (uniform over the CTA)
    __device__ bool wait(int b)
    {
        unsigned polls = 0;
        bool ok = true;
        for (;;) {
            uint32_t done;
            asm volatile(
                "{\n\t.reg .pred q;\n\t"
                "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 q, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, q;\n\t}"
                : "=r"(done)
                : "r"(smem_addr(&sm->bar[b])), "r"(phase[b] & 1u)
                : "memory");
            if (done) break;
            if (++polls > limit) {
                atomicCAS(err, 0, kErrTimeout);
                ok = false;
                break;
            }
        }
        ++phase[b];
        return __syncthreads_and(ok);
    }
};

__global__ void __launch_bounds__(kThreads, 1)
potrf_cluster_kernel(int n, float* A, long long lda, int* info, int info_base, float* dinv, int last,
                     int* fail, int* err, const int* run_if)
{
    extern __shared__ __align__(16) unsigned char sm_raw[];
    ClusterSmem& sm = *reinterpret_cast<ClusterSmem*>(sm_raw);
    int C, rank;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(C));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int NT = (n + kT - 1) / kT;
    const int tid = threadIdx.x, r4 = (tid & 15) * 4, c4 = (tid >> 4) * 4;
    auto ext = [&](int i) { return min(kT, n - i * kT); };
    auto tile = [&](int i, int j) { return A + (long long)(j * kT) * lda + i * kT; };
    auto src = [&](int i, int j) { return TileSrc{tile(i, j), lda, ext(i), ext(j)}; };
    if (tid == 0) {
        for (int b = 0; b < 2; ++b)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&sm.bar[b])),
                         "r"(C));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sm.stop = (run_if && *reinterpret_cast<const volatile int*>(run_if) == 0) ? 2
                  : (info && *reinterpret_cast<volatile int*>(info) != 0)         ? 1
                                                                                  : 0;
    }
    __syncthreads();
    const int skip = sm.stop;  // the same in every CTA: read before any write
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (skip && rank == 0 && tid == 0) *fail = 1;  // no W either
    if (skip == 2) return;
    int stands = skip ? 0 : NT;  // first tile that is inverted as it stands
    ClusterBarrier bar{&sm, C, spin_limit_of(err), err, {0u, 0u}};
    // One CTA needs no barriers: 0 = column k ready (D_k written, step k - 1 applied),
    // 1 = column k solved.
    const bool solo = C == 1;
    const int kmax = (tid >> 5) * 8 + 8;  // D_k is lower: this warp's columns end there
    float acc[4][4];
    auto clear = [&]() {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    };
    const bool aligned = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15u) == 0;
    auto store_acc = [&](float* T, int rows, int cols) {
        if (aligned && rows == kT && cols == kT) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(T + (long long)(c4 + j) * lda + r4) =
                    make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
            return;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (r4 + i < rows && c4 + j < cols) T[(long long)(c4 + j) * lda + r4 + i] = acc[i][j];
    };
    if (skip) {
    } else if (rank == 0) {
        float *S = sm.tile[0], *W = sm.tile[1], *P = sm.tile[2], *X = sm.tile[3];
        tile64::load_lower<true>(S, A, lda, ext(0), false);
        __syncthreads();
        bool waiting = false;  // arrived on barrier 1, not waited yet
        for (int k = 0; k < NT; ++k) {
            const int f = tile64::chol64(S, ext(k), &sm.fail_col);
            tile64::store_lower(tile(k, k), S, lda, ext(k));
            if (f >= 0 && tid == 0) {
                if (info) atomicCAS(info, 0, info_base + k * kT + f + 1);
                *reinterpret_cast<volatile int*>(fail) = 1;
            }
            // also of a failing tile: its columns before the failing one are valid
            if (!last || k < NT - 1) {
                tile64::inv64<tile64::kReciprocal>(S, W, sm.X, sm.rd);
                tile64::store_inv(dinv + (long long)k * kT * kT, W, false);
            }
            if (!solo) {
                if (waiting && !bar.wait(1)) break;
                waiting = false;
                bar.arrive(0);
                if (!bar.wait(0)) break;
            } else {
                __syncthreads();
            }
            if (f >= 0) stands = k + 1;
            if (f >= 0 || k == NT - 1) break;
            // X = L(k+1, k) = A(k+1, k) D_k^T
            fetch_tile(P, src(k + 1, k));
            fetch_commit();
            float old[4][4];  // tile (k+1, k+1), in flight meanwhile
            const int e = ext(k + 1);
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    old[i][j] = (r4 + i < e && c4 + j <= r4 + i)
                                    ? __ldcg(tile(k + 1, k + 1) + (long long)(c4 + j) * lda + r4 + i)
                                    : (r4 + i == c4 + j ? 1.f : 0.f);
            fetch_wait<0>();
            __syncthreads();
            clear();
            tile_mma(acc, P, W, kmax);
            store_acc(tile(k + 1, k), e, kT);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(X + (c4 + j) * kLdS + r4) =
                    make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
            if (!solo) {
                bar.arrive(1);  // its barrier also orders X
                waiting = true;
            } else {
                __syncthreads();
            }
            clear();
            tile_mma(acc, X, X);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(S + (c4 + j) * kLdS + r4) =
                    make_float4(old[0][j] - acc[0][j], old[1][j] - acc[1][j],
                                old[2][j] - acc[2][j], old[3][j] - acc[3][j]);
            __syncthreads();
        }
    } else {
        const int w = rank - 1, nw = C - 1;
        bool live = true;
        for (int k = 0; k < NT && live; ++k) {
            bar.arrive(0);
            if (!bar.wait(0)) break;
            if (tid == 0) sm.stop = *reinterpret_cast<volatile int*>(fail);
            __syncthreads();
            if (sm.stop) stands = k + 1;
            if (sm.stop || k == NT - 1) break;
            for (int i = k + 2 + w; i < NT; i += nw) {  // L(i, k) = A(i, k) D_k^T
                fetch_tile(sm.tile[0], src(i, k));
                fetch_tile(sm.tile[1], {dinv + (long long)k * kT * kT, kT, kT, kT});
                fetch_commit();
                fetch_wait<0>();
                __syncthreads();
                clear();
                tile_mma(acc, sm.tile[0], sm.tile[1], kmax);
                store_acc(tile(i, k), ext(i), kT);
                __syncthreads();
            }
            bar.arrive(1);
            if (!bar.wait(1)) break;
            // A(i, j) -= L(i, k) L(j, k)^T, pairs in row order after (k+1, k+1); the
            // next pair's operands load during this one's products
            const int rem = NT - 1 - k, pairs = rem * (rem + 1) / 2;
            auto pair_at = [&](int t, int& i, int& j) {
                i = k + 1;
                while (t > i - (k + 1)) {
                    t -= i - k;
                    ++i;
                }
                j = k + 1 + t;
            };
            auto fetch_pair = [&](int t, int slot) {
                if (t < pairs) {
                    int i, j;
                    pair_at(t, i, j);
                    fetch_tile(sm.tile[2 * slot], src(i, k));
                    if (i != j) fetch_tile(sm.tile[2 * slot + 1], src(j, k));
                }
                fetch_commit();
            };
            int slot = 0;
            fetch_pair(1 + w, 0);
            for (int t = 1 + w; t < pairs; t += nw, slot ^= 1) {
                int i, j;
                pair_at(t, i, j);
                float* T = tile(i, j);
                const int ei = ext(i), ej = ext(j);
                float old[4][4];
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int a = 0; a < 4; ++a)
                        old[a][b] = (r4 + a < ei && c4 + b < ej && (i != j || r4 + a >= c4 + b))
                                        ? __ldcg(T + (long long)(c4 + b) * lda + r4 + a)
                                        : 0.f;
                fetch_pair(t + nw, slot ^ 1);
                fetch_wait<1>();
                __syncthreads();
                clear();
                tile_mma(acc, sm.tile[2 * slot], sm.tile[2 * slot + (i != j ? 1 : 0)]);
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int a = 0; a < 4; ++a)
                        if (r4 + a < ei && c4 + b < ej && (i != j || r4 + a >= c4 + b))
                            T[(long long)(c4 + b) * lda + r4 + a] = old[a][b] - acc[a][b];
                __syncthreads();
            }
            fetch_wait<0>();
        }
    }
    for (int i = stands + rank; i < NT - last; i += C) {
        __syncthreads();
        tile64::load_lower<true>(sm.tile[0], tile(i, i), lda, ext(i), false);
        __syncthreads();
        tile64::inv64<tile64::kReciprocal>(sm.tile[0], sm.tile[1], sm.X, sm.rd);
        tile64::store_inv(dinv + (long long)i * kT * kT, sm.tile[1], false);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ------------------------------------------------------------ inverse kernel
__global__ void __launch_bounds__(kThreads, 1)
tile_inverse_kernel(int n, const float* A, long long lda, float* W, long long ldw, const float* dinv,
                    float* Tsc, unsigned* ctr, const int* fail, int* abort_flag, int* err)
{
    __shared__ __align__(16) float As[kT * kLdS];
    __shared__ __align__(16) float Bs[kT * kLdS];
    const int NT = (n + kT - 1) / kT;
    const int cta = blockIdx.x;
    const unsigned G = gridDim.x;
    const int tid = threadIdx.x, r4 = (tid & 15) * 4, c4 = (tid >> 4) * 4;
    Sync sy{ctr, const_cast<int*>(fail), abort_flag, err, G, 0u, spin_limit_of(err)};
    auto tile = [&](int i, int j) { return A + (long long)(j * kT) * lda + i * kT; };
    auto ext = [&](int i) { return min(kT, n - i * kT); };
    if (*fail != 0) return;  // written by the launch before: the same for every CTA

    // W = L^{-1} by recursive doubling over tile blocks: for sibling blocks
    // A = [b, b+s) and C = [b+s, b+2s) (tiles), W(C,A) = -W(C,C) (L(C,A) W(A,A)),
    // T = L(C,A) W(A,A) kept in scratch at the W(C,A) position.
    // Setup: diagonal tiles D_i, strictly upper tiles zero.
    for (int t = cta; t < NT * NT; t += G) {
        const int i = t % NT, j = t / NT;
        if (i < j) {
            for (int q = tid; q < kT * kT; q += kThreads) {
                const int c = q >> 6, r = q & 63;
                if (r < ext(i) && c < ext(j)) W[(long long)(j * kT + c) * ldw + i * kT + r] = 0.f;
            }
        } else if (i == j) {
            const float* D = dinv + (long long)i * kT * kT;
            for (int q = tid; q < kT * kT; q += kThreads) {
                const int c = q >> 6, r = q & 63;
                if (r < ext(i) && c < ext(i))
                    W[(long long)(i * kT + c) * ldw + i * kT + r] = __ldcg(D + c * kT + r);
            }
        }
    }
    grid_barrier(sy);
    auto wt = [&](int i, int j) { return W + (long long)(j * kT) * ldw + i * kT; };
    auto tt = [&](int i, int j) { return Tsc + (long long)(j * kT) * ldw + i * kT; };
    for (int st = 1; st < NT; st *= 2) {
        // tiles (ci, aj) of every pair: C rows [b+st, min(b+2st, NT)), A cols [b, b+st)
        const int npair = (NT + 2 * st - 1) / (2 * st);
        const int per = st * st;
        // phase A: T(ci, aj) = sum_{m=aj}^{b+st-1} L(ci, m) W(m, aj)
        for (int t = cta; t < npair * per; t += G) {
            const int pr = t / per, q = t - pr * per;
            const int b = pr * 2 * st;
            const int ci = b + st + q / st, aj = b + q % st;
            if (ci >= NT) continue;
            float acc[4][4] = {};
            for (int m = aj; m < b + st; ++m) {
                load_pair<false, true>(As, {tile(ci, m), lda, ext(ci), ext(m)}, Bs,
                                       {wt(m, aj), ldw, ext(m), ext(aj)});
                __syncthreads();
                tile_mma(acc, As, Bs);
                __syncthreads();
            }
            float* T = tt(ci, aj);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int bb = 0; bb < 4; ++bb) {
                    const int r = r4 + a, c = c4 + bb;
                    if (r < ext(ci) && c < ext(aj)) T[(long long)c * ldw + r] = acc[a][bb];
                }
        }
        grid_barrier(sy);
        // phase B: W(ci, aj) = -sum_{m=b+st}^{ci} W(ci, m) T(m, aj)
        for (int t = cta; t < npair * per; t += G) {
            const int pr = t / per, q = t - pr * per;
            const int b = pr * 2 * st;
            const int ci = b + st + q / st, aj = b + q % st;
            if (ci >= NT) continue;
            float acc[4][4] = {};
            for (int m = b + st; m <= ci; ++m) {
                load_pair<false, true>(As, {wt(ci, m), ldw, ext(ci), ext(m)}, Bs,
                                       {tt(m, aj), ldw, ext(m), ext(aj)});
                __syncthreads();
                tile_mma(acc, As, Bs);
                __syncthreads();
            }
            float* Wp = wt(ci, aj);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int bb = 0; bb < 4; ++bb) {
                    const int r = r4 + a, c = c4 + bb;
                    if (r < ext(ci) && c < ext(aj)) Wp[(long long)c * ldw + r] = -acc[a][bb];
                }
        }
        grid_barrier(sy);
    }
}

}  // namespace

int potrf_block_max_n() { return kT * kMaxNT; }

hdbf_status potrf_block(hdbf_context* ctx, int n, float* A, long long lda, int* info,
                        int info_base, float* W, long long ldw, bool last)
{
    if (n <= 0) return HDBF_STATUS_SUCCESS;
    if (n > kT * kMaxNT || lda < n || (W && ldw < n)) return HDBF_STATUS_INVALID_VALUE;
    // ws_skinny holds 256 * ws_n floats: >= n * ldw once ws_n >= max(n, ldw * n / 256)
    const long long need = W ? ((long long)ldw * n + 255) / 256 : 0;
    HDBF_TRY(ensure_ws(ctx, (int)std::max<long long>(n, std::max<long long>(need, 64))));
    const int NT = (n + kT - 1) / kT;
    int* sm = ctx->dev_small + kSmallBlockBar;
    if (cudaMemsetAsync(sm, 0, 3 * sizeof(int), ctx->stream) != cudaSuccess) return last_cuda(ctx);
    unsigned* ctr = reinterpret_cast<unsigned*>(sm);
    int* fail = sm + 1;
    int* abort_flag = sm + 2;
    int* err = ctx->dev_small + kSmallErr;
    float* dinv = ws_inv(ctx);
    const double flops = (double)n * n * n / 3.0 + (W ? (double)n * n * n / 3.0 : 0.0);
    ProfScope prof(ctx, kClsPotrfBlock, flops, 8.0 * n * n, n, n, n);
    // Workers for the pairs of a tile column: none for two tiles (CTA 0 does all
    // there is), 3 for three, 7 for four, 15 above.
    int C = NT <= 2 ? 1 : (NT == 3 ? 4 : (NT == 4 ? 8 : 16));
    while (C > std::max(1, ctx->cluster_max)) C /= 2;
    if (C == 2) C = 1;
    if (C == 1 && NT > 2) return HDBF_STATUS_NOT_SUPPORTED;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterSmem);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = C;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, potrf_cluster_kernel, n, A, lda, info, info_base, dinv,
                                       (int)(last && !W), fail, err, ctx->run_if);
    ctx->launches++;
    if (e == cudaSuccess && W) {
        int G = std::min(NT * NT, ctx->sm_count);  // the set-up pass touches NT^2 tiles
        float* Tsc = ws_skinny(ctx);  // n x n scratch (leading dimension ldw)
        const float* Ac = A;
        void* args[] = {&n, &Ac, &lda, &W, &ldw, &dinv, &Tsc, &ctr, &fail, &abort_flag, &err};
        e = cudaLaunchCooperativeKernel((const void*)tile_inverse_kernel, dim3(G), dim3(kThreads),
                                        args, 0, ctx->stream);
        ctx->launches++;
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return HDBF_STATUS_CUDA_ERROR;
    }
    return HDBF_STATUS_SUCCESS;
}

void configure_potrf_block(hdbf_context*)
{
    cudaFuncSetAttribute(potrf_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(ClusterSmem));
    cudaFuncSetAttribute(potrf_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaGetLastError();
}

}  // namespace hdbf
