// GETRF panel leaf on one thread-block cluster: partially pivoted LU of an
// m x w (w <= 128, m <= 32768) column block, FP32 and FP64, replacing
// rocsolver_sgetrf's unblocked leaf on the tall panel
// (src/getrf/getrf_pivot_internal.h:17-39).
//
// What bounds it is the serial chain of one pivot per column, so the whole
// block stays on chip and the exchange of each column stays inside a cluster
// (<= 16 CTAs, <= 16 SMs), where a message takes a fraction of an L2 round
// trip.  The block sits in the cluster's shared memory, a contiguous slice of
// rows per CTA (tile[c * ldt + r], ldt odd).  It is factored in sub-panels of
// NB columns (64 bytes of a row: 16 FP32, 8 FP64) that live in registers,
// thread t owning local rows t, t + TH, ...  Per column:
//   1. every warp finds its candidate (largest |a| over rows at position >= J,
//      lowest position on ties -- LAPACK ISAMAX) with integer warp reductions;
//      its owner lane writes the candidate's row to shared memory;
//   2. after one block barrier a few warps reduce the warps' candidates and
//      push the CTA's one (magnitude, position, NB values) to every CTA of the
//      cluster with st.async, counted in bytes on the receiver's mbarrier: data
//      and flag arrive in one trip, and nothing needs a fence;
//   3. every warp reduces the CTAs' candidates from its own shared memory, and
//      every thread scales and applies the rank-1 update.
// No row moves inside a sub-panel: a row keeps its place and carries its
// position (what LAPACK's swaps so far would have made it), the chosen row
// stores its U entries and the others their multiplier where they are.  The
// registers shift by one column per step, so the loop is rolled and needs no
// selects.
// Two message buffers (column parity) suffice: a CTA sends column J + 1 only
// after a block barrier that follows all its reads of column J, and nobody can
// send column J + 2 without it.
// After a sub-panel, all columns of the tile take its interchanges as at most 2
// NB composed row moves through distributed shared memory; every CTA reads the
// new diagonal rows and solves U12 = L11^{-1} A12 for itself, and every thread
// applies the rank-NB update to its own rows, in column order: the result is
// bit-identical to column-by-column elimination (getf2_grid.cu).
// Measured per column, against the grid-wide kernel's 1.9-2.0 us: 1.3 us at m =
// 1001, 1.5 at 4096, 1.8 at 8192, 2.4 at 16384 (FP32).  The rest is issue and
// fixed latencies: ~300 dependent instructions per warp and column.
// Waits on an mbarrier are bounded by the handle's poll limit; an expired wait
// records a timeout and the CTA runs on without waiting or arriving (a second
// arrival in an incomplete phase is an error), so that every cluster barrier is
// still met.
#include "getf2_common.cuh"
#include "internal.h"

namespace hdbf {
namespace {

constexpr int kClMaxW = 128;
constexpr int kClMaxCluster = 16;
constexpr int kClMaxRows = 2048;  // per CTA: 4 register rows for each of 512 threads

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, int rank)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_arrive()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait()
{
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void push16(uint32_t dst, uint32_t bar, uint4 v)
{
    asm volatile(
        "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, "
        "[%5];" ::"r"(dst),
        "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
        : "memory");
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

template <class T>
struct alignas(16) Vec4 {
    T x[4];
};

template <class T>
constexpr int kNB = 64 / (int)sizeof(T);

// A candidate as it travels: five 16-byte chunks.
template <class T>
struct Cand;
template <>
struct alignas(16) Cand<float> {
    unsigned mag;
    int row;
    int pad[2];
    float x[16];
};
template <>
struct alignas(16) Cand<double> {
    unsigned long long mag;
    int row;
    int pad;
    double x[8];
};

// Magnitude and row of a candidate in one 16-byte load.
__device__ __forceinline__ void load_key(const Cand<float>& c, unsigned& mag, int& row)
{
    const uint2 v = *reinterpret_cast<const uint2*>(&c);
    mag = v.x;
    row = (int)v.y;
}
__device__ __forceinline__ void load_key(const Cand<double>& c, unsigned long long& mag, int& row)
{
    const uint4 v = *reinterpret_cast<const uint4*>(&c);
    mag = ((unsigned long long)v.y << 32) | v.x;
    row = (int)v.z;
}

template <class T>
struct ClusterSmem {
    Cand<T> in[2][kClMaxCluster];  // the cluster's candidates
    Cand<T> own[2][16];            // this CTA's warps' candidates
    T U[kClMaxW / 2][kNB<T>][2];  // U12 of the sub-panel, columns in pairs: U[c / 2][k][c & 1]
    T L[kNB<T>][kNB<T> + 1];      // L11, L[r][k]
    int piv[kNB<T>];              // pivot positions of the sub-panel
    unsigned long long bar[2];
};

// acc(c), acc(c + 1) -= l * (u(c), u(c + 1)): one packed FMA in FP32.
struct Pair32 {
    unsigned long long v;
    __device__ __forceinline__ Pair32(float x, float y)
    {
        asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    }
    __device__ __forceinline__ void fma(Pair32 l, Pair32 u)
    {
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(l.v), "l"(u.v));
    }
    __device__ __forceinline__ void get(float& x, float& y) const
    {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    }
};
struct Pair64 {
    double x, y;
    __device__ __forceinline__ Pair64(double a, double b) : x(a), y(b) {}
    __device__ __forceinline__ void fma(Pair64 l, Pair64 u)
    {
        x = ::fma(l.x, u.x, x);
        y = ::fma(l.y, u.y, y);
    }
    __device__ __forceinline__ void get(double& a, double& b) const
    {
        a = x;
        b = y;
    }
};
template <class T>
struct PairOf {
    using type = Pair32;
};
template <>
struct PairOf<double> {
    using type = Pair64;
};

__device__ __forceinline__ void copy_async(float* dst, const float* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async(double* dst, const double* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src)
                 : "memory");
}

template <class T, int TH, int R>
__global__ void __launch_bounds__(TH, 1)
getf2_cluster_kernel(int m, int w, T* A, long long lda, int rpc, int* ipiv, int ipiv_add, int* info,
                     int info_base, int pivot, int* err)
{
    constexpr int NB = kNB<T>;
    constexpr int NW = TH / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterSmem<T>& sm = *reinterpret_cast<ClusterSmem<T>*>(smem_raw);
    T* tile = reinterpret_cast<T*>(smem_raw + sizeof(ClusterSmem<T>));
    const int ldt = rpc | 1;

    int C, rank;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(C));
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = rank * rpc;
    const int nr = max(0, min(m, r0 + rpc) - r0);
    const unsigned limit = spin_limit_of(err);
    const uint32_t base = smem_addr(smem_raw);
    auto off_of = [&](const void* q) { return smem_addr(q) - base; };
    auto peer_base = [&](int q) { return peer_addr(base, q); };
    bool dead = false;  // an expired wait: run on without waiting

    if (tid == 0) {
        for (int b = 0; b < 2; ++b)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sm.bar[b])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int c = 0; c < w; ++c) {  // the whole slice in flight at once
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = tid + TH * i;
            if (r < nr) copy_async(tile + c * ldt + r, A + (long long)c * lda + r0 + r);
        }
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    cluster_arrive();
    cluster_wait();  // every CTA runs and its barriers are initialised

    const int steps = min(m, w);
    for (int jb = 0; jb < steps; jb += NB) {
        const int nbc = min(NB, w - jb);      // columns of this sub-panel
        const int sb = min(nbc, steps - jb);  // pivots in it
        const int owner = jb / rpc;  // rpc is a multiple of NB: it owns all diagonal rows
        T a[R][NB];
        int pos[R];  // the row's position; below J once it has been a pivot row
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = tid + TH * i;
            pos[i] = r < nr ? r0 + r : -1;
#pragma unroll
            for (int c = 0; c < NB; ++c)
                a[i][c] = (r < nr && c < nbc) ? tile[(jb + c) * ldt + r] : T(0);
        }
        const int dst = lane & 15, ch = tid >> 4;  // sender roles: peer, 16-byte chunk

#pragma unroll 1
        for (int j = 0; j < sb; ++j) {
            const int J = jb + j, par = J & 1;
            // 1. this CTA's candidates for column J
            Mag<T> vb = 0;
            int row = INT_MAX;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const Mag<T> b = mag_bits(a[i][0]);
                if ((pivot ? pos[i] >= J : pos[i] == J) &&
                    (row == INT_MAX || b > vb || (b == vb && pos[i] < row))) {
                    vb = b;
                    row = pos[i];
                }
            }
            Mag<T> mv;
            int mrow;
            warp_argmax(vb, row, mv, mrow);
            if (row == mrow && (row != INT_MAX || lane == 0)) {
                Cand<T>& c = sm.own[par][warp];
                c.mag = mv;
                c.row = mrow;
#pragma unroll
                for (int i = 0; i < R; ++i)
                    if (R == 1 || pos[i] == mrow) {
#pragma unroll
                        for (int q = 0; q < NB; ++q) c.x[q] = a[i][q];
                    }
            }
            if (tid == 0 && C > 1 && !dead)  // every candidate, 80 bytes
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                 smem_addr(&sm.bar[par])),
                             "r"(C * 80)
                             : "memory");
            __syncthreads();
            // 2. the CTA's candidate to every CTA: 16 peers per 16-byte chunk
            int from = 0;
            if (C == 1 || warp < 3) {
                Mag<T> k = 0;
                int kr = INT_MAX;
                if (lane < NW) load_key(sm.own[par][lane], k, kr);
                warp_argmax(k, kr, mv, mrow);
                from = __ffs(__ballot_sync(0xffffffffu, lane < NW && kr == mrow)) - 1;
                if (C > 1 && dst < C && ch < 5)
                    push16(peer_base(dst) + off_of(&sm.in[par][rank]) + 16 * ch,
                           peer_base(dst) + off_of(&sm.bar[par]),
                           reinterpret_cast<const uint4*>(&sm.own[par][from])[ch]);
            }
            // 3. the cluster's candidate
            const T* urow;
            T rcp;
            if (C > 1) {
                if (!dead) {
                    const uint32_t bar = smem_addr(&sm.bar[par]);
                    const uint32_t phase = (J >> 1) & 1;
                    unsigned polls = 0;
                    for (;;) {
                        uint32_t ok;
                        asm volatile(
                            "{\n\t.reg .pred q;\n\t"
                            "mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
                            "selp.u32 %0, 1, 0, q;\n\t}"
                            : "=r"(ok)
                            : "r"(bar), "r"(phase)
                            : "memory");
                        if (ok) break;
                        if (++polls > limit) {
                            atomicCAS(err, 0, kErrTimeout);
                            dead = true;
                            break;
                        }
                    }
                    dead = __any_sync(0xffffffffu, dead);
                }
                Mag<T> k = 0;
                int kr = INT_MAX;
                if (lane < C) load_key(sm.in[par][lane], k, kr);
                rcp = Bits<T>::rcp(Bits<T>::val(k));  // every candidate's, beside the reductions
                warp_argmax(k, kr, mv, mrow);
                const unsigned who = __ballot_sync(0xffffffffu, lane < C && kr == mrow);
                from = who ? __ffs(who) - 1 : 0;
                rcp = __shfl_sync(0xffffffffu, rcp, from);
                urow = sm.in[par][from].x;
            } else {
                urow = sm.own[par][from].x;
                rcp = Bits<T>::rcp(Bits<T>::val(mv));
            }
            const int p = mrow >= J && mrow < m ? mrow : J;
            T u[NB];
#pragma unroll
            for (int c = 0; c < NB; ++c) u[c] = urow[c];
            const T piv = u[0];
            const bool nz = piv != T(0);
            rcp = piv < T(0) ? -rcp : (piv == piv ? rcp : piv);
            const bool recip = abs_t(piv) >= min_normal(piv) || piv != piv;
            T l[R];
#pragma unroll
            for (int i = 0; i < R; ++i) l[i] = a[i][0] * rcp;
            if (!(nz && recip)) {  // a zero or subnormal pivot
#pragma unroll
                for (int i = 0; i < R; ++i) l[i] = nz ? a[i][0] / piv : a[i][0];
            }
#pragma unroll
            for (int i = 0; i < R; ++i) {
                T* x = tile + J * ldt + tid + TH * i;
                if (pos[i] == p) {  // the pivot row: its U entries, in place
#pragma unroll
                    for (int c = 0; c < NB; ++c)
                        if (c < nbc - j) x[c * ldt] = u[c];
                    pos[i] = J;
                } else if (pos[i] == J) {
                    pos[i] = p;
                }
                if (pos[i] > J) x[0] = l[i];
#pragma unroll
                for (int c = 1; c < NB; ++c) a[i][c - 1] = fma_t(-l[i], u[c], a[i][c]);
                a[i][NB - 1] = T(0);
            }
            if (tid == TH - 1) {
                sm.piv[j] = p;
                if (rank == 0) {
                    if (pivot) ipiv[J] = p + 1 + ipiv_add;
                    if (!nz && info) atomicCAS(info, 0, info_base + J + 1);
                }
            }
        }
        __syncthreads();
        cluster_arrive();
        cluster_wait();  // every CTA's rows are in its tile
        // The interchanges, composed: lanes < NB are the diagonal positions, the
        // others the pivot positions; the row that ends up at mv_pos is found
        // by undoing the swaps from the last one on (a position that appears
        // twice gets the same row twice).
        int mv_pos = lane < NB ? jb + lane : (lane < NB + sb ? sm.piv[lane - NB] : -1);
        if (lane >= NB && mv_pos < jb + NB) mv_pos = -1;  // a diagonal position: lanes < NB have it
        int mv_src = mv_pos;
        for (int t = sb - 1; t >= 0; --t) {
            const int q = sm.piv[t];
            mv_src = mv_src == jb + t ? q : (mv_src == q ? jb + t : mv_src);
        }
        // Lane = move, warp = columns: the moves into this
        // CTA's rows, and on every CTA the new diagonal rows from the sub-panel
        // on, from which each takes L11 and solves U12 itself.
        constexpr int kIt = (kClMaxW * 4 / (int)sizeof(T) + NW - 1) / NW;
        const int c1 = jb + nbc;
        const bool top_row = lane < NB;
        const bool moved = mv_pos >= r0 && mv_pos < r0 + nr && mv_src != mv_pos;
        T v[kIt];
        {
            const int q_src = mv_src >= 0 ? mv_src / rpc : 0;
            const uint32_t src = peer_base(q_src) + off_of(tile + (mv_src - q_src * rpc));
#pragma unroll
            for (int k = 0; k < kIt; ++k) {
                const int c = warp + NW * k;
                const bool want =
                    mv_src >= 0 && c < w && ((top_row && c >= jb && lane < sb) || moved);
                v[k] = want ? peer_load(src + (uint32_t)(c * ldt * (int)sizeof(T)), T(0)) : T(0);
            }
        }
        cluster_arrive();
        if (top_row) {
#pragma unroll
            for (int k = 0; k < kIt; ++k) {
                const int c = warp + NW * k;
                if (c >= c1 && c < w) sm.U[(c - c1) >> 1][lane][(c - c1) & 1] = v[k];
                else if (c >= jb && c < c1) sm.L[lane][c - jb] = v[k];
            }
        }
        __syncthreads();
        T x[NB];  // U12 = L11^{-1} A12, a column per thread
        if (c1 + tid < w) {
            T* up = &sm.U[tid >> 1][0][tid & 1];
#pragma unroll
            for (int k = 0; k < NB; ++k) x[k] = up[2 * k];
#pragma unroll
            for (int r = 1; r < NB; ++r) {
                if (r < sb) {
#pragma unroll
                    for (int k = 0; k < r; ++k) x[r] = fma_t(-sm.L[r][k], x[k], x[r]);
                }
                up[2 * r] = x[r];
            }
        }
        cluster_wait();  // everybody has read: rows may change
#pragma unroll
        for (int k = 0; k < kIt; ++k) {
            const int c = warp + NW * k;
            if (moved && c < w && !(top_row && c >= c1)) tile[c * ldt + mv_pos - r0] = v[k];
        }
        if (rank == owner && c1 + tid < w) {
#pragma unroll
            for (int k = 0; k < NB; ++k)
                if (k < sb) tile[(c1 + tid) * ldt + jb - r0 + k] = x[k];
        }
        __syncthreads();
        if (c1 >= w) continue;
        // the rank-NB update of this thread's rows, two columns at a time
        if (jb + sb < m) {
            using P = typename PairOf<T>::type;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int r = tid + TH * i;
                if (r >= nr || r0 + r < jb + sb) continue;
                T nl[NB];
#pragma unroll
                for (int k = 0; k < NB; ++k) nl[k] = -tile[(jb + k) * ldt + r];
                T* xp = tile + c1 * ldt + r;
                for (int c = 0; c + c1 < w; c += 2, xp += 2 * ldt) {
                    const bool two = c + 1 + c1 < w;
                    P acc(xp[0], two ? xp[ldt] : T(0));
                    const Vec4<T>* up = reinterpret_cast<const Vec4<T>*>(sm.U[c >> 1]);
#pragma unroll
                    for (int k = 0; k < NB; k += 2) {
                        const Vec4<T> u = up[k >> 1];
                        acc.fma(P(nl[k], nl[k]), P(u.x[0], u.x[1]));
                        acc.fma(P(nl[k + 1], nl[k + 1]), P(u.x[2], u.x[3]));
                    }
                    T x0, x1;
                    acc.get(x0, x1);
                    xp[0] = x0;
                    if (two) xp[ldt] = x1;
                }
            }
        }
    }
    __syncthreads();
    for (int c0 = 0; c0 < w; c0 += 8) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = tid + TH * i;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (r < nr && c0 + c < w)
                    A[(long long)(c0 + c) * lda + r0 + r] = tile[(c0 + c) * ldt + r];
        }
    }
    if (dead) __nanosleep(200000);  // messages nobody waited for land before the exit
    cluster_arrive();
    cluster_wait();  // no CTA leaves while another may still reach its shared memory
}

// Rows per CTA: a multiple of 16 so that a sub-panel's diagonal rows sit in one CTA.
int cluster_rpc(int m, int C) { return ((m + C - 1) / C + 15) / 16 * 16; }
template <class T>
size_t cluster_smem(int rpc, int w)
{
    return sizeof(ClusterSmem<T>) + sizeof(T) * (size_t)(rpc | 1) * w;
}
size_t cluster_cap(const hdbf_context* ctx)
{
    return ctx->max_smem_optin > 1024 ? ctx->max_smem_optin - 1024 : 0;
}

template <class T, int TH, int R>
cudaError_t launch_cluster(hdbf_context* ctx, int C, size_t smem, int m, int w, T* A, long long lda,
                           int rpc, int* ipiv, int ipiv_add, int* info, int info_base, int pivot)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(TH);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = C;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int* err = ctx->dev_small + kSmallErr;
    return cudaLaunchKernelEx(&cfg, getf2_cluster_kernel<T, TH, R>, m, w, A, lda, rpc, ipiv, ipiv_add,
                              info, info_base, pivot, err);
}

template <class T>
hdbf_status getf2_cluster_t(hdbf_context* ctx, int m, int w, T* A, long long lda, int* ipiv,
                            int ipiv_add, int* info, int info_base, bool pivot)
{
    if (m <= 0 || w <= 0) return HDBF_STATUS_SUCCESS;
    if (w > getf2_cluster_leaf(ctx, m, (int)sizeof(T))) return HDBF_STATUS_NOT_SUPPORTED;
    // One row per thread of 256 where the cluster is large enough for that.
    int C = 1;
    while (C < ctx->cluster_max &&
           (cluster_rpc(m, C) > 256 || cluster_smem<T>(cluster_rpc(m, C), w) > cluster_cap(ctx)))
        C *= 2;
    const int rpc = cluster_rpc(m, C);
    const size_t smem = cluster_smem<T>(rpc, w);
    const int piv = pivot ? 1 : 0;
    ProfScope prof(ctx, kClsPanel, (double)m * w * w - (double)w * w * w / 3.0,
                   2.0 * sizeof(T) * m * w, m, w, C);
    cudaError_t e;
    if (rpc <= 256)
        e = launch_cluster<T, 256, 1>(ctx, C, smem, m, w, A, lda, rpc, ipiv, ipiv_add, info,
                                      info_base, piv);
    else if (rpc <= 512)
        e = launch_cluster<T, 512, 1>(ctx, C, smem, m, w, A, lda, rpc, ipiv, ipiv_add, info,
                                      info_base, piv);
    else if (rpc <= 1024)
        e = launch_cluster<T, 512, 2>(ctx, C, smem, m, w, A, lda, rpc, ipiv, ipiv_add, info,
                                      info_base, piv);
    else
        e = launch_cluster<T, 512, 4>(ctx, C, smem, m, w, A, lda, rpc, ipiv, ipiv_add, info,
                                      info_base, piv);
    ctx->launches++;
    if (e != cudaSuccess) {
        cudaGetLastError();
        return HDBF_STATUS_CUDA_ERROR;
    }
    return HDBF_STATUS_SUCCESS;
}

template <class T, int TH, int R>
int configure_one(hdbf_context* ctx, int best)
{
    auto* k = getf2_cluster_kernel<T, TH, R>;
    const int cap = (int)cluster_cap(ctx);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, cap) != cudaSuccess ||
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    for (; best >= 1; best /= 2) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(best);
        cfg.blockDim = dim3(TH);
        cfg.dynamicSmemBytes = cap;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = best;
        at.val.clusterDim.y = 1;
        at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int clusters = 0;
        const bool ok = cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess &&
                        clusters >= 1;
        cudaGetLastError();
        if (ok) break;
    }
    return best;
}

}  // namespace

// Largest cluster that every instance can launch with the full shared memory.
int configure_cluster_panel(hdbf_context* ctx)
{
    int best = kClMaxCluster;
    best = configure_one<float, 256, 1>(ctx, best);
    best = configure_one<float, 512, 1>(ctx, best);
    best = configure_one<float, 512, 2>(ctx, best);
    best = configure_one<float, 512, 4>(ctx, best);
    best = configure_one<double, 256, 1>(ctx, best);
    best = configure_one<double, 512, 1>(ctx, best);
    best = configure_one<double, 512, 2>(ctx, best);
    best = configure_one<double, 512, 4>(ctx, best);
    return best;
}

// Widest leaf (a power of two, <= 128 FP32 or 64 FP64 columns) that one cluster
// holds at height m; 0 when not even one sub-panel fits.
int getf2_cluster_leaf(hdbf_context* ctx, int m, int elem)
{
    if (ctx->cluster_max < 1) return 0;
    const int rpc = cluster_rpc(m, ctx->cluster_max);
    if (rpc > kClMaxRows) return 0;
    const int widest = kClMaxW * 4 / elem;
    for (int w = widest; w >= 64 / elem; w /= 2) {
        const size_t need = elem == 4 ? cluster_smem<float>(rpc, w) : cluster_smem<double>(rpc, w);
        if (need <= cluster_cap(ctx)) return w;
    }
    return 0;
}

hdbf_status getf2_cluster(hdbf_context* ctx, int m, int w, float* A, long long lda, int* ipiv,
                          int ipiv_add, int* info, int info_base, bool pivot)
{
    return getf2_cluster_t(ctx, m, w, A, lda, ipiv, ipiv_add, info, info_base, pivot);
}

hdbf_status getf2_cluster(hdbf_context* ctx, int m, int w, double* A, long long lda, int* ipiv,
                          int ipiv_add, int* info, int info_base, bool pivot)
{
    return getf2_cluster_t(ctx, m, w, A, lda, ipiv, ipiv_add, info, info_base, pivot);
}

}  // namespace hdbf
