// Batched uneven factor-and-solve in one persistent launch.
//
// Thousands of independent small systems (Cholesky: n <= 512, LU with partial
// pivoting: n <= 768, one right-hand side each) are processed by a grid of
// persistent CTAs (several per SM) that pull matrix indices from a device
// work queue (largest work first, so the tail is short).  Each CTA factors its
// matrix in place, right-looking with panels of PW columns:
//   * the panel (all rows below the diagonal, PW columns) is copied into
//     shared memory and factored there.  Cholesky: sub-panels of 8 columns, whose
//     diagonal block every thread factors in its own registers while it carries
//     its rows along -- three barriers per 8 columns.  LU: sub-panels of 16
//     columns in registers, one barrier per column; no row moves inside a
//     sub-panel (a row carries its position), the interchanges follow as at most
//     32 composed row moves;
//   * LU: the panel's row interchanges are composed into at most 2 PW row
//     moves and applied to the other columns with one gather / scatter per
//     column (every load of a column before its first store); U12 by one thread
//     per column (unit-lower solve against the panel's diagonal block);
//   * the trailing update A22 -= L21 U12 (Cholesky: L21 L21^T, lower part) in
//     items of 128 rows x 8 columns per warp, packed FP32 FMAs, lanes on
//     consecutive rows, so that C moves in whole 128-byte lines and no block
//     barrier is needed (the earlier 8 x 4 tiles per thread scattered every
//     access over 16 columns: 41% of the kernel's time at 13% of the FMA rate);
//   * the right-hand side goes along as one more column (moves, solve against
//     the diagonal block, update), so only the backward substitution is left:
//     32-row blocks, one warp on the diagonal block with reciprocals ready, the
//     other rows' entries loaded while it works.
// The launch shape is a variant: threads per CTA and panel width; the
// shared-memory footprint of the panel width sets the CTAs per SM.
// No reference counterpart (the reference factors one matrix per call); the
// per-matrix arithmetic follows LAPACK's xPOTRF / xGETRF (first maximum
// pivot, reciprocal scaling unless |pivot| < FLT_MIN, info = first failing
// column; LU keeps factoring after a zero pivot, Cholesky stops).
#include <algorithm>
#include <cfloat>
#include <climits>
#include <vector>

#include "internal.h"
#include "tile64.cuh"
#include "hdbf/batched.h"

namespace hdbf {
namespace {

constexpr int kMaxChol = 512;  // largest Cholesky order
constexpr int kMaxLu = 768;    // largest LU order
constexpr int kLdp = kMaxLu + 8;  // panel rows (padding for 8-row register tiles)
constexpr int kNB = 16;           // LU sub-panel
constexpr int kWC = 8;            // columns of a trailing-update item

struct BatchArgs {
    int count;
    const int* order;  // processing order (indices into the arrays below)
    const int* op;     // 0 = POTRF + POTRS, 1 = GETRF + GETRS
    const int* n;
    const int* lda;
    float* const* A;
    float* const* b;
    int* const* ipiv;
    int* info;
    unsigned* queue;
};

// A warp's pivot candidate: magnitude bits, position, its sub-panel row.
struct alignas(16) Cand {
    unsigned mag;
    int pos;
    int pad[2];
    float x[kNB];
};

template <int T, int PW>
struct Smem {
    static constexpr int kW = T / 32;
    float P[(size_t)PW * kLdp];   // panel P[c * kLdp + r], r relative to the panel's first row
    float Ub[kW * PW * kWC];      // a warp's columns of U12: [warp][q][c]
    float x[kMaxLu];              // right-hand side / solution
    Cand cand[2][kW];             // LU: the warps' candidates, by column parity
    float U[kNB][kNB + 1];        // LU: U12 of the sub-panel inside the panel, U[c][k]
    float dots[32];
    int piv[PW];                  // LU: swap rows of the panel's columns
    int item;
};

// Largest magnitude over the warp and the lowest position that has it.
__device__ __forceinline__ void warp_argmax(unsigned vb, int pos, unsigned& mv, int& mp)
{
    mv = __reduce_max_sync(0xffffffffu, vb);
    mp = __reduce_min_sync(0xffffffffu, vb == mv ? pos : INT_MAX);
}
__device__ __forceinline__ unsigned long long pack2(float x, float y)
{
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    return v;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a,
                                     unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// ------------------------------------------------------------ panel kernels
// Pivoted LU of the m x kb panel P (m rows from the diagonal down), kb a multiple
// of kNB or the last panel.  piv[j] receives the panel row swapped with row j.
// Returns the first zero-pivot column + 1 (0: none); the factorization continues
// past it, as xGETF2.  P complete on entry and on return.  R rows per thread.
template <int T, int PW, int R>
__device__ __noinline__ int lu_panel_rows(Smem<T, PW>& s, int m, int kb)
{
    constexpr int NW = T / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int zero = 0;
    const int steps = min(m, kb);
    for (int jb = 0; jb < steps; jb += kNB) {
        const int nbc = min(kNB, kb - jb), sb = min(nbc, steps - jb);
        float a[R][kNB];
        int pos[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = tid + T * i;
            pos[i] = r < m ? r : -1;
#pragma unroll
            for (int c = 0; c < kNB; ++c)
                a[i][c] = (r < m && c < nbc) ? s.P[(jb + c) * kLdp + r] : 0.f;
        }
#pragma unroll 1
        for (int j = 0; j < sb; ++j) {
            const int J = jb + j, par = J & 1;
            unsigned vb = 0;
            int best = INT_MAX;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                // xGETRF's first maximum: a NaN is one on the diagonal (nothing compares
                // above it; its bits are above an infinity's) and loses elsewhere
                const float v = fabsf(a[i][0]);
                const unsigned b = v == v || pos[i] == J ? __float_as_uint(v) : 0u;
                if (pos[i] >= J &&
                    (best == INT_MAX || b > vb || (b == vb && pos[i] < best))) {
                    vb = b;
                    best = pos[i];
                }
            }
            unsigned mv;
            int mp;
            warp_argmax(vb, best, mv, mp);
            if (best == mp && (best != INT_MAX || lane == 0)) {
                Cand& c = s.cand[par][warp];
                c.mag = mv;
                c.pos = mp;
#pragma unroll
                for (int i = 0; i < R; ++i)
                    if (R == 1 || pos[i] == mp) {
#pragma unroll
                        for (int q = 0; q < kNB; ++q) c.x[q] = a[i][q];
                    }
            }
            __syncthreads();
            unsigned k = 0;
            int kp = INT_MAX;
            if (lane < NW) {
                const uint2 key = *reinterpret_cast<const uint2*>(&s.cand[par][lane]);
                k = key.x;
                kp = (int)key.y;
            }
            warp_argmax(k, kp, mv, mp);
            const int from = __ffs(__ballot_sync(0xffffffffu, lane < NW && kp == mp)) - 1;
            const float* urow = s.cand[par][from].x;
            float u[kNB];
#pragma unroll
            for (int c = 0; c < kNB; ++c) u[c] = urow[c];
            const float pv = u[0];
            if (pv == 0.f && zero == 0) zero = J + 1;
            const float rcp = 1.0f / pv;
            const bool plain = fabsf(pv) >= FLT_MIN || pv != pv;
            if (tid == T - 1) s.piv[J] = mp;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                float l = a[i][0] * rcp;
                if (!plain) l = pv != 0.f ? a[i][0] / pv : a[i][0];
                float* x = s.P + J * kLdp + tid + T * i;
                if (pos[i] == mp) {  // the pivot row: its U entries, in place
#pragma unroll
                    for (int c = 0; c < kNB; ++c)
                        if (c < nbc - j) x[c * kLdp] = u[c];
                    pos[i] = J;
                } else if (pos[i] == J) {
                    pos[i] = mp;
                }
                if (pos[i] > J) x[0] = l;
#pragma unroll
                for (int c = 1; c < kNB; ++c) a[i][c - 1] = fmaf(-l, u[c], a[i][c]);
                a[i][kNB - 1] = 0.f;
            }
        }
        __syncthreads();
        // The sub-panel's interchanges on all panel columns, composed: lanes <
        // kNB are its diagonal positions, the others the pivot positions; the
        // row that ends up at mv_pos is found by undoing the swaps.
        int mv_pos = lane < kNB ? jb + lane : (lane < kNB + sb ? s.piv[jb + lane - kNB] : -1);
        if (lane < kNB ? lane >= sb : mv_pos < jb + kNB) mv_pos = -1;
        int mv_src = mv_pos;
        for (int t = sb - 1; t >= 0; --t) {
            const int q = s.piv[jb + t];
            mv_src = mv_src == jb + t ? q : (mv_src == q ? jb + t : mv_src);
        }
        constexpr int kIt = (PW + NW - 1) / NW;
        float v[kIt];
#pragma unroll
        for (int q = 0; q < kIt; ++q) {
            const int c = warp + NW * q;
            v[q] = (c < kb && mv_pos >= 0) ? s.P[c * kLdp + mv_src] : 0.f;
        }
        __syncwarp();  // a column's rows belong to one warp
#pragma unroll
        for (int q = 0; q < kIt; ++q) {
            const int c = warp + NW * q;
            if (c < kb && mv_pos >= 0) s.P[c * kLdp + mv_pos] = v[q];
        }
        __syncthreads();
        const int c1 = jb + nbc;
        if (c1 >= kb || jb + sb >= m) continue;
        // U12 of the panel's remaining columns (at most kNB), a thread each
        if (c1 + tid < kb) {
            float x[kNB];
            float* col = s.P + (c1 + tid) * kLdp + jb;
#pragma unroll
            for (int k = 0; k < kNB; ++k) x[k] = col[k];
#pragma unroll
            for (int k = 0; k < kNB; ++k)
#pragma unroll
                for (int r = k + 1; r < kNB; ++r)
                    x[r] = fmaf(-s.P[(jb + k) * kLdp + jb + r], x[k], x[r]);
#pragma unroll
            for (int k = 0; k < kNB; ++k) s.U[tid][k] = col[k] = x[k];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = tid + T * i;
            if (r >= m || r < jb + kNB) continue;
            float l[kNB];
#pragma unroll
            for (int k = 0; k < kNB; ++k) l[k] = -s.P[(jb + k) * kLdp + r];
            for (int c = 0; c < kb - c1; ++c) {
                float x = s.P[(c1 + c) * kLdp + r];
#pragma unroll
                for (int k = 0; k < kNB; ++k) x = fmaf(l[k], s.U[c][k], x);
                s.P[(c1 + c) * kLdp + r] = x;
            }
        }
        __syncthreads();
    }
    return zero;
}

template <int T, int PW>
__device__ __forceinline__ int lu_panel(Smem<T, PW>& s, int m, int kb)
{
    constexpr int kAll = (kMaxLu + T - 1) / T;
    if (m <= T) return lu_panel_rows<T, PW, 1>(s, m, kb);
    if (kAll > 2 && m <= 2 * T) return lu_panel_rows<T, PW, 2>(s, m, kb);
    return lu_panel_rows<T, PW, kAll>(s, m, kb);
}

// Cholesky of the m x kb panel P (diagonal block on top) from column j0 on, a
// column at a time with IEEE operations: the first failing column + 1, or 0.
// Columns past a failure are left as they are.
template <int T, int PW>
__device__ __noinline__ int chol_panel_careful(Smem<T, PW>& s, int m, int kb, int j0)
{
    const int tid = threadIdx.x;
    for (int j = j0; j < kb; ++j) {
        const float d = s.P[j * kLdp + j];  // final: updated before the last barrier
        if (!(d > 0.f)) return j + 1;       // uniform: every thread read the same value
        const float sd = sqrtf(d);
        const float rcp = 1.0f / sd;
        for (int r = j + 1 + tid; r < m; r += T) {
            const float l = s.P[j * kLdp + r] * rcp;
            s.P[j * kLdp + r] = l;
            if (r < kb) s.dots[r] = l;
        }
        __syncthreads();
        if (tid == 0) s.P[j * kLdp + j] = sd;
        for (int r = j + 1 + tid; r < m; r += T) {
            const float l = s.P[j * kLdp + r];
            const int cmax = min(kb - 1, r);
            for (int c = j + 1; c <= cmax; ++c)
                s.P[c * kLdp + r] = fmaf(-l, s.dots[c], s.P[c * kLdp + r]);
        }
        __syncthreads();
    }
    return 0;
}

// The same in sub-panels of 8 columns: every thread factors the 8 x 8 diagonal
// block in registers and solves its own rows against it, then updates the panel's
// remaining columns of those rows.  A sub-panel with a pivot outside the fast
// range (failed, tiny, huge, NaN) and the rest of the panel go the careful way.
// P complete on entry and on return; a last panel that is no multiple of 8 is
// padded with the identity.
template <int T, int PW>
__device__ int chol_panel(Smem<T, PW>& s, int m, int kb)
{
    constexpr int W = 8;
    constexpr int R = (kMaxChol + T - 1) / T;
    const int tid = threadIdx.x;
    for (int jb = 0; jb < kb; jb += W) {
        float D[W][W];  // D[c][r], r >= c
#pragma unroll
        for (int c = 0; c < W; ++c)
#pragma unroll
            for (int r = c; r < W; ++r)
                D[c][r] = (jb + r < kb) ? s.P[(jb + c) * kLdp + jb + r] : (r == c ? 1.f : 0.f);
        bool ok = true;
        float rs[W];
#pragma unroll
        for (int j = 0; j < W; ++j) {
            ok = ok & tile64::fast_range(D[j][j]);
            tile64::rsqrt_pair(D[j][j], rs[j], D[j][j]);
#pragma unroll
            for (int r = j + 1; r < W; ++r) D[j][r] *= rs[j];
#pragma unroll
            for (int c = j + 1; c < W; ++c)
#pragma unroll
                for (int r = c; r < W; ++r) D[c][r] = fmaf(-D[j][r], D[j][c], D[c][r]);
        }
        if (__syncthreads_or(!ok)) return chol_panel_careful<T, PW>(s, m, kb, jb);
        if (tid == T - 1) {
#pragma unroll
            for (int c = 0; c < W; ++c)
#pragma unroll
                for (int r = c; r < W; ++r)
                    if (jb + r < kb) s.P[(jb + c) * kLdp + jb + r] = D[c][r];
        }
        if (jb + W >= m) break;
        float x[R][W];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = jb + W + tid + T * i;
            if (r >= m) continue;
#pragma unroll
            for (int c = 0; c < W; ++c) x[i][c] = s.P[(jb + c) * kLdp + r];
#pragma unroll
            for (int j = 0; j < W; ++j) {
                x[i][j] *= rs[j];
#pragma unroll
                for (int c = j + 1; c < W; ++c) x[i][c] = fmaf(-x[i][j], D[j][c], x[i][c]);
            }
#pragma unroll
            for (int c = 0; c < W; ++c) s.P[(jb + c) * kLdp + r] = x[i][c];
        }
        __syncthreads();
        if (jb + W < kb) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int r = jb + W + tid + T * i;
                if (r >= m) continue;
                for (int c = jb + W; c < kb; c += 4) {  // four columns (rows of L) at a time
                    if (c > r) break;
                    float y[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) y[e] = c + e < kb ? s.P[(c + e) * kLdp + r] : 0.f;
#pragma unroll
                    for (int k = 0; k < W; ++k) {
                        const float4 l = *reinterpret_cast<const float4*>(s.P + (jb + k) * kLdp + c);
                        y[0] = fmaf(-x[i][k], l.x, y[0]);
                        y[1] = fmaf(-x[i][k], l.y, y[1]);
                        y[2] = fmaf(-x[i][k], l.z, y[2]);
                        y[3] = fmaf(-x[i][k], l.w, y[3]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (c + e < kb && c + e <= r) s.P[(c + e) * kLdp + r] = y[e];
                }
            }
            __syncthreads();
        }
    }
    __syncthreads();
    return 0;
}

// P (m x kb) <-> global A at the panel's top-left corner, a warp per column,
// eight loads in flight per lane; lower: only rows r >= c are stored.
template <int T, int PW, bool TO_SMEM>
__device__ __forceinline__ void move_panel(Smem<T, PW>& s, float* A, long long lda, int m, int kb,
                                           bool lower)
{
    const int lane = threadIdx.x & 31;
    for (int c = threadIdx.x >> 5; c < kb; c += T / 32) {
        float* g = A + (long long)c * lda;
        float* p = s.P + c * kLdp;
        for (int r0 = lower ? c / 32 * 32 : 0; r0 < m; r0 += 256) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int r = r0 + lane + 32 * u;
                v[u] = r < m ? (TO_SMEM ? g[r] : p[r]) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int r = r0 + lane + 32 * u;
                if (r < m && (!lower || r >= c)) (TO_SMEM ? p[r] : g[r]) = v[u];
            }
        }
    }
}

// --------------------------------------------------------- trailing update
// One item: rows r0 + lane + 32 i (i < RI) x 8 columns, C -= A B with A(r, q) =
// a[q * kLdp + r] (shared) and B(q, c) = b[q * ldb + c] (shared, 16-byte aligned
// rows).  lower: only entries with r >= c0 + column are touched.
template <int RI, int PW>
__device__ __forceinline__ void update_item(const float* a, const float* b, int ldb, int kb, float* C,
                                            long long ldc, int r0, int rows, int c0, int cols,
                                            bool lower)
{
    const int lane = threadIdx.x & 31;
    float old[RI][kWC];
#pragma unroll
    for (int c = 0; c < kWC; ++c)
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int r = r0 + lane + 32 * i;
            old[i][c] = (c0 + c < cols && r < rows && (!lower || r >= c0 + c))
                            ? C[(long long)(c0 + c) * ldc + r]
                            : 0.f;
        }
    unsigned long long acc[RI][kWC / 2];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int c = 0; c < kWC / 2; ++c) acc[i][c] = 0ull;
    a += r0 + lane;
#pragma unroll 4
    for (int q = 0; q < kb; ++q) {
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(b + q * ldb);
        const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(b + q * ldb + 4);
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const float x = a[q * kLdp + 32 * i];
            const unsigned long long xx = pack2(x, x);
            fma2(acc[i][0], xx, b0.x);
            fma2(acc[i][1], xx, b0.y);
            fma2(acc[i][2], xx, b1.x);
            fma2(acc[i][3], xx, b1.y);
        }
    }
#pragma unroll
    for (int c = 0; c < kWC; ++c)
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int r = r0 + lane + 32 * i;
            float lo, hi;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc[i][c >> 1]));
            if (c0 + c < cols && r < rows && (!lower || r >= c0 + c))
                C[(long long)(c0 + c) * ldc + r] = old[i][c] - ((c & 1) ? hi : lo);
        }
}

// C (n2 x n2) -= L21 B over all items, warps in turn.  LU: B = U12 in global
// memory (kb rows above C), copied to the warp's own buffer per item; Cholesky: B
// = L21^T from the panel, lower part only.
template <int T, int PW>
__device__ __forceinline__ void trailing_update(Smem<T, PW>& s, int kb, int n2, float* C,
                                                long long ldc, bool lower)
{
    constexpr int NW = T / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int groups = (n2 + kWC - 1) / kWC, blocks = (n2 + 127) / 128;
    float* ub = s.Ub + warp * PW * kWC;
    for (int it = warp; it < groups * blocks; it += NW) {
        const int g = it % groups, blk = it / groups;
        const int c0 = g * kWC, end = min(n2, 128 * blk + 128);
        int r0 = 128 * blk;
        if (lower) r0 = max(r0, c0 / 32 * 32);
        if (r0 >= end) continue;
        const float* b = s.P + kb + c0;
        int ldb = kLdp;
        if (!lower) {
            float v[PW * kWC / 32];
#pragma unroll
            for (int u = 0; u < PW * kWC / 32; ++u) {
                const int e = lane + 32 * u, c = e / PW, q = e % PW;
                v[u] = (c0 + c < n2 && q < kb) ? C[(long long)(c0 + c) * ldc - kb + q] : 0.f;
            }
            __syncwarp();  // the previous item's reads are done
#pragma unroll
            for (int u = 0; u < PW * kWC / 32; ++u) {
                const int e = lane + 32 * u, c = e / PW, q = e % PW;
                ub[q * kWC + c] = v[u];
            }
            __syncwarp();
            b = ub;
            ldb = kWC;
        }
        const float* a = s.P + kb;
        const int left = end - r0;
        if (left > 64) update_item<4, PW>(a, b, ldb, kb, C, ldc, r0, end, c0, n2, lower);
        else if (left > 32) update_item<2, PW>(a, b, ldb, kb, C, ldc, r0, end, c0, n2, lower);
        else update_item<1, PW>(a, b, ldb, kb, C, ldc, r0, end, c0, n2, lower);
    }
}

// x2 -= L21 x1 for the right-hand side (x1 the panel's kb entries, solved).
template <int T, int PW>
__device__ __forceinline__ void rhs_update(Smem<T, PW>& s, int k, int kb, int m)
{
    for (int r = kb + threadIdx.x; r < m; r += T) {
        float acc = s.x[k + r];
#pragma unroll 8
        for (int q = 0; q < kb; ++q) acc = fmaf(-s.P[q * kLdp + r], s.x[k + q], acc);
        s.x[k + r] = acc;
    }
}

// x / d by d's reciprocal r and one correction (Markstein, IBM J. Res. Dev. 34, 1990:
// the rounded quotient but for rare ties), where the residual is exact; by division
// elsewhere.  The plain product x r rounds twice: 2-3 % more error in a solution.
__device__ __forceinline__ bool plain_quotients(float d) { return d * d > 1e-36f && d * d < 1e36f; }
template <bool PLAIN>
__device__ __forceinline__ float quotient(float x, float d, float r)
{
    const float q = x * r;
    return PLAIN ? fmaf(fmaf(-d, q, x), r, q) : x / d;
}
// One warp's substitution on x (lane i: row i of kB), d its diagonal, row(q) the factor
// of x_q in this lane's row; BACK from the last row up.
template <bool PLAIN, bool BACK, int N, class Row>
__device__ __forceinline__ float warp_substitute(float x, float d, float r, Row row)
{
    const int i = threadIdx.x & 31;
#pragma unroll
    for (int s = 0; s < N; ++s) {
        const int q = BACK ? N - 1 - s : s;
        const float xq = __shfl_sync(0xffffffffu, quotient<PLAIN>(x, d, r), q);
        x = (BACK ? i < q : i > q) ? fmaf(-row(q), xq, x) : x;
    }
    return quotient<PLAIN>(x, d, r);
}
template <bool BACK, int N, class Row>
__device__ __forceinline__ float warp_solve(float x, float d, Row row)
{
    const float r = 1.f / d;
    if (__all_sync(0xffffffffu, plain_quotients(d)))
        return warp_substitute<true, BACK, N>(x, d, r, row);
    return warp_substitute<false, BACK, N>(x, d, r, row);
}

// x1 <- L11^{-1} x1 on one warp (unit: implicit ones on the diagonal).
template <int T, int PW>
__device__ __forceinline__ void rhs_solve(Smem<T, PW>& s, int k, int kb, bool unit)
{
    const int i = threadIdx.x & 31;
    float li[PW];
#pragma unroll
    for (int q = 0; q < PW; ++q) li[q] = (i < kb && q < i) ? s.P[q * kLdp + i] : 0.f;
    float xi = i < kb ? s.x[k + i] : 0.f;
    if (unit) {
#pragma unroll
        for (int q = 0; q < PW; ++q) {
            const float xq = __shfl_sync(0xffffffffu, xi, q);
            xi = i > q ? fmaf(-li[q], xq, xi) : xi;
        }
    } else {
        const float d = i < kb ? s.P[i * kLdp + i] : 1.f;
        xi = warp_solve<false, PW>(xi, d, [&](int q) { return li[q]; });
    }
    if (i < kb) s.x[k + i] = xi;
}

// ------------------------------------------------------------------ LU
template <int T, int PW>
__device__ int lu_factor(Smem<T, PW>& s, float* A, int n, long long lda, int* ipiv)
{
    constexpr int NW = T / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int info = 0;
    for (int k = 0; k < n; k += PW) {
        const int kb = min(PW, n - k), m = n - k;
        float* Ak = A + (long long)k * lda + k;  // panel's top-left corner
        move_panel<T, PW, true>(s, Ak, lda, m, kb, false);
        __syncthreads();
        const int z = lu_panel<T, PW>(s, m, kb);
        if (z && !info) info = k + z;
        move_panel<T, PW, false>(s, Ak, lda, m, kb, false);
        if (tid < kb) ipiv[k + tid] = k + s.piv[tid] + 1;
        // The panel's interchanges as row moves: two per lane, into diagonal
        // position `lane` and into the pivot position of column `lane`; the
        // source is found by undoing the swaps (a position that appears twice
        // gets the same row twice).
        int t0 = lane < kb ? lane : -1, t1 = lane < kb ? s.piv[lane] : -1;
        if (t1 < kb) t1 = -1;
        int s0 = t0, s1 = t1;
        for (int t = kb - 1; t >= 0; --t) {
            const int q = s.piv[t];
            s0 = s0 == t ? q : (s0 == q ? t : s0);
            s1 = s1 == t ? q : (s1 == q ? t : s1);
        }
        const bool m0 = t0 != s0, m1 = t1 != s1;
        // apply them to the columns left and right of the panel: one warp per
        // column, eight columns per pass, every source of a column read before
        // any of its targets is written
        constexpr int kPass = 8;
        for (int c = warp; c < n - kb; c += kPass * NW) {
            float v0[kPass], v1[kPass];
#pragma unroll
            for (int u = 0; u < kPass; ++u) {
                const int cu = c + u * NW;
                v0[u] = v1[u] = 0.f;
                if (cu < n - kb) {
                    const float* Ac = A + (long long)(cu < k ? cu : cu + kb) * lda + k;
                    if (m0) v0[u] = Ac[s0];
                    if (m1) v1[u] = Ac[s1];
                }
            }
            __syncwarp();
#pragma unroll
            for (int u = 0; u < kPass; ++u) {
                const int cu = c + u * NW;
                if (cu < n - kb) {
                    float* Ac = A + (long long)(cu < k ? cu : cu + kb) * lda + k;
                    if (m0) Ac[t0] = v0[u];
                    if (m1) Ac[t1] = v1[u];
                }
            }
        }
        if (warp == NW - 1) {  // and to the right-hand side, then L11^{-1} on it
            const float v0 = m0 ? s.x[k + s0] : 0.f, v1 = m1 ? s.x[k + s1] : 0.f;
            __syncwarp();
            if (m0) s.x[k + t0] = v0;
            if (m1) s.x[k + t1] = v1;
            __syncwarp();
            rhs_solve<T, PW>(s, k, kb, true);
        }
        __syncthreads();
        const int m2 = m - kb;  // trailing rows / columns
        rhs_update<T, PW>(s, k, kb, m);
        // U12 = L11^{-1} A12 (unit lower) for every trailing column at once,
        // one thread per column
        for (int c = tid; c < m2; c += T) {
            float* colp = A + (long long)(k + kb + c) * lda + k;
            float xv[PW];
#pragma unroll
            for (int q = 0; q < PW; ++q) xv[q] = q < kb ? colp[q] : 0.f;
#pragma unroll
            for (int q = 0; q < PW; ++q)
#pragma unroll
                for (int r = q + 1; r < PW; ++r) xv[r] = fmaf(-s.P[q * kLdp + r], xv[q], xv[r]);
#pragma unroll
            for (int q = 0; q < PW; ++q)
                if (q < kb) colp[q] = xv[q];
        }
        __syncthreads();
        trailing_update<T, PW>(s, kb, m2, A + (long long)(k + kb) * lda + k + kb, lda, false);
        __syncthreads();
    }
    return info;
}

// ------------------------------------------------------------ Cholesky
template <int T, int PW>
__device__ int chol_factor(Smem<T, PW>& s, float* A, int n, long long lda)
{
    for (int k = 0; k < n; k += PW) {
        const int kb = min(PW, n - k), m = n - k;
        float* Ak = A + (long long)k * lda + k;
        move_panel<T, PW, true>(s, Ak, lda, m, kb, false);
        __syncthreads();
        const int f = chol_panel<T, PW>(s, m, kb);
        // the strictly upper part of the diagonal block keeps its input values
        move_panel<T, PW, false>(s, Ak, lda, m, kb, true);
        if (f) {
            __syncthreads();
            return k + f;
        }
        if (threadIdx.x >= T - 32) rhs_solve<T, PW>(s, k, kb, false);
        __syncthreads();
        rhs_update<T, PW>(s, k, kb, m);
        trailing_update<T, PW>(s, kb, m - kb, A + (long long)(k + kb) * lda + k + kb, lda, true);
        __syncthreads();
    }
    return 0;
}

// ------------------------------------------------------------------ solves
// Backward substitutions on x (shared memory), 32 rows at a time.  The panel's
// shared memory holds the diagonal blocks D[r * 33 + c] of the current and the
// next step.
constexpr int kBk = 32;

// The diagonal block at k (kb rows) into D by all threads; entries outside the
// triangle are not used.
template <int T>
__device__ __forceinline__ void load_block(float* D, const float* A, long long lda, int k, int kb)
{
    for (int q = threadIdx.x; q < kBk * kBk; q += T) {
        const int c = q >> 5, r = q & 31;
        if (r < kb && c < kb) D[r * 33 + c] = A[(long long)(k + c) * lda + k + r];
    }
}

// x1 <- D^{-1} x1 on one warp, D upper, or lower and transposed.
template <bool TRANS>
__device__ __forceinline__ void block_back(const float* D, float* x, int kb, const float* sub)
{
    const int i = threadIdx.x & 31;
    float d[kBk];
#pragma unroll
    for (int q = 0; q < kBk; ++q)
        d[q] = (i < kb && q > i && q < kb) ? (TRANS ? D[q * 33 + i] : D[i * 33 + q]) : 0.f;
    float xi = i < kb ? x[i] - (sub ? sub[i] : 0.f) : 0.f;
    xi = warp_solve<true, kBk>(xi, i < kb ? D[i * 33 + i] : 1.f, [&](int q) { return d[q]; });
    if (i < kb) x[i] = xi;
}

// x <- U^{-1} x, U the upper triangle of A (non-unit): the block's columns of the
// rows above are loaded while one warp solves the diagonal block.
template <int T>
__device__ void backward_upper(const float* A, int n, long long lda, float* x, float* D)
{
    const int tid = threadIdx.x;
    const int nblk = (n + kBk - 1) / kBk;
    load_block<T>(D + ((nblk - 1) & 1) * kBk * 33, A, lda, (nblk - 1) * kBk,
                  n - (nblk - 1) * kBk);
    __syncthreads();
    for (int bi = nblk - 1; bi >= 0; --bi) {
        const int k = bi * kBk, kb = min(kBk, n - k);
        float a[kBk];
        if (tid < k) {
#pragma unroll
            for (int q = 0; q < kBk; ++q) a[q] = q < kb ? A[(long long)(k + q) * lda + tid] : 0.f;
        }
        if (bi > 0) load_block<T>(D + ((bi - 1) & 1) * kBk * 33, A, lda, k - kBk, kBk);
        if (tid >= T - 32) block_back<false>(D + (bi & 1) * kBk * 33, x + k, kb, nullptr);
        __syncthreads();
        for (int r = tid; r < k; r += T) {
            if (r != tid) {
#pragma unroll
                for (int q = 0; q < kBk; ++q) a[q] = q < kb ? A[(long long)(k + q) * lda + r] : 0.f;
            }
            float acc = x[r];
#pragma unroll
            for (int q = 0; q < kBk; ++q)
                if (q < kb) acc = fmaf(-a[q], x[k + q], acc);
            x[r] = acc;
        }
        __syncthreads();
    }
}

// x <- L^{-T} x, L lower (non-unit): per block, the dot products of its columns
// with the solved rows below (a warp per column), then the block on one warp.
template <int T>
__device__ void backward_lower_t(const float* A, int n, long long lda, float* x, float* dots,
                                 float* D)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nblk = (n + kBk - 1) / kBk;
    for (int bi = nblk - 1; bi >= 0; --bi) {
        const int k = bi * kBk, kb = min(kBk, n - k);
        load_block<T>(D, A, lda, k, kb);
        for (int j = warp; j < kBk; j += T / 32) {
            float sum = 0.f;
            if (j < kb) {
                const float* cj = A + (long long)(k + j) * lda;
                for (int r = k + kb + lane; r < n; r += 128) {  // four loads in flight
                    float v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) v[u] = r + 32 * u < n ? cj[r + 32 * u] : 0.f;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (r + 32 * u < n) sum = fmaf(v[u], x[r + 32 * u], sum);
                }
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
            if (lane == 0) dots[j] = sum;
        }
        __syncthreads();
        if (warp == T / 32 - 1) block_back<true>(D, x + k, kb, dots);
        __syncthreads();
    }
}

// ------------------------------------------------------------------ kernel
// Register budget for two CTAs per SM at 256 threads and three at 128 (the
// 16-column panel's shared footprint allows three): one matrix per CTA spends
// much of its time at barriers, so co-resident CTAs fill the gaps.
template <int T>
constexpr int min_ctas() { return T >= 512 ? 1 : (T >= 256 ? 2 : 3); }

template <int T, int PW>
__global__ void __launch_bounds__(T, min_ctas<T>()) batched_factor_solve_kernel(BatchArgs a)
{
    extern __shared__ __align__(16) unsigned char sm_raw[];
    Smem<T, PW>& s = *reinterpret_cast<Smem<T, PW>*>(sm_raw);
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s.item = (int)atomicAdd(a.queue, 1u);
        __syncthreads();
        const int it = s.item;
        __syncthreads();
        if (it >= a.count) break;
        const int idx = a.order[it];
        const int n = a.n[idx];
        const int op = a.op[idx];
        if (n <= 0 || (op == 0 && n > kMaxChol) || (op != 0 && n > kMaxLu)) continue;
        float* A = a.A[idx];
        const long long lda = a.lda[idx];
        float* b = a.b[idx];
        for (int r = tid; r < n; r += T) s.x[r] = b[r];
        int info;
        if (op == 0) info = chol_factor<T, PW>(s, A, n, lda);
        else info = lu_factor<T, PW>(s, A, n, lda, a.ipiv[idx]);
        if (tid == 0) a.info[idx] = info;
        if (info) continue;  // b keeps its input
        if (op != 0) backward_upper<T>(A, n, lda, s.x, s.P);
        else backward_lower_t<T>(A, n, lda, s.x, s.dots, s.P);
        for (int r = tid; r < n; r += T) b[r] = s.x[r];
        __syncthreads();
    }
}

// Launch shapes: threads per CTA and panel width.
struct Variant {
    int threads, panel;
};
constexpr Variant kVariants[] = {{128, 32}, {256, 32}, {512, 32}, {128, 16}, {256, 16}, {512, 16}};
constexpr int kNumVariants = (int)(sizeof(kVariants) / sizeof(kVariants[0]));

template <int T, int PW>
hdbf_status launch_batched(hdbf_context* ctx, const BatchArgs& a)
{
    const size_t smem = sizeof(Smem<T, PW>);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_factor_solve_kernel<T, PW>,
                                                      T, smem) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    const int ctas = std::max(1, std::min(a.count, ctx->sm_count * per_sm));
    batched_factor_solve_kernel<T, PW><<<ctas, T, smem, ctx->stream>>>(a);
    ctx->launches++;
    return last_cuda(ctx);
}

template <int T, int PW>
void configure_one()
{
    cudaFuncSetAttribute(batched_factor_solve_kernel<T, PW>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(Smem<T, PW>));
}

}  // namespace

void configure_batched_kernels(hdbf_context* ctx)
{
    (void)ctx;
    configure_one<128, 32>();
    configure_one<256, 32>();
    configure_one<512, 32>();
    configure_one<128, 16>();
    configure_one<256, 16>();
    configure_one<512, 16>();
    cudaGetLastError();
}

}  // namespace hdbf

using namespace hdbf;

extern "C" {

int hdbf_batched_num_variants(void) { return kNumVariants; }

hdbf_status hdbf_batched_variant_shape(int variant, int* threads, int* panel)
{
    if (variant < 0 || variant >= kNumVariants || !threads || !panel)
        return HDBF_STATUS_INVALID_VALUE;
    *threads = kVariants[variant].threads;
    *panel = kVariants[variant].panel;
    return HDBF_STATUS_SUCCESS;
}

hdbf_status hdbf_batched_factor_solve(hdbf_handle h, int variant, int count, const int* order,
                                      const int* op, const int* n, const int* lda, float* const* A,
                                      float* const* b, int* const* ipiv, int* info,
                                      unsigned int* queue)
{
    if (!h) return HDBF_STATUS_INVALID_HANDLE;
    if (count < 0 || variant < 0 || variant >= kNumVariants)
        return h->last_status = HDBF_STATUS_INVALID_VALUE;
    if (count == 0) return h->last_status = HDBF_STATUS_SUCCESS;
    if (!order || !op || !n || !lda || !A || !b || !ipiv || !info || !queue)
        return h->last_status = HDBF_STATUS_INVALID_VALUE;
    BatchArgs a{count, order, op, n, lda, A, b, ipiv, info, queue};
    const std::vector<long long> key = {41, variant, count, (long long)order, (long long)op,
                                        (long long)n, (long long)lda, (long long)A, (long long)b,
                                        (long long)ipiv, (long long)info, (long long)queue};
    return h->last_status = run_graph(h, key, [&]() -> hdbf_status {
        cudaMemsetAsync(queue, 0, sizeof(unsigned int), h->stream);
        ProfScope prof(h, kClsBatched, 0.0, 0.0);
        switch (variant) {
        case 0: return launch_batched<128, 32>(h, a);
        case 1: return launch_batched<256, 32>(h, a);
        case 2: return launch_batched<512, 32>(h, a);
        case 3: return launch_batched<128, 16>(h, a);
        case 4: return launch_batched<256, 16>(h, a);
        default: return launch_batched<512, 16>(h, a);
        }
    });
}

}  // extern "C"
