// Cholesky factor and triangular inverse of one 64 x 64 tile in shared memory,
// by a block of 256 threads.  Both sit on the serial chain of every diagonal
// block, so what counts is latency, not rate.
//
// chol64 works in panels whose diagonal block fits in a thread's registers
// (chol_panel_fast), with look-ahead between the panels.
// inv64 inverts the four 16 x 16 diagonal blocks (one warp each, a lane per
// column) and joins them, first 16, then 32: L22 W21 = -L21 W11, the product by all
// threads and the solve by substitution, so that every column is as accurate as one
// long substitution would make it (the product W21 = -W22 (L21 W11) is 0.5 us
// shorter, but its error grows with the condition of L22).
// One tile in one launch (load, factor, inverse, stores): 10.4 us; 62 us before,
// with two barriers, an IEEE square root and a division per column of the
// factor and one thread per column of the inverse, a division per row.
#pragma once

#include <cuda_runtime.h>

#include <cfloat>

namespace hdbf {
namespace tile64 {

constexpr int kN = 64;
constexpr int kLd = 68;        // shared row pitch: float4 / double2 aligned
constexpr int kThreads = 256;
constexpr int kScratch = 32 * 36;

template <class T>
struct alignas(16) Vec4 {
    T x[4];
};

// 1 / sqrt(d) and sqrt(d), each to about an ulp: one Newton step on the hardware
// estimate, and one residual correction of the root.  For d in fast_range, the normal
// numbers up to 2^126: no product here overflows, and the one that may underflow, the
// root's residual below 2^-100, only loses part of the correction.  A matrix may be
// tiny or huge as a whole, and the careful path costs a tile twice its time (n = 64
// times 1e32: 24 us, 49 the careful way).
__device__ __forceinline__ bool fast_range(float d) { return d >= FLT_MIN && d <= 8.5e37f; }
__device__ __forceinline__ bool fast_range(double d) { return d >= DBL_MIN && d <= 4e307; }
__device__ __forceinline__ void rsqrt_pair(float d, float& r, float& s)
{
    r = rsqrtf(d);
    r = fmaf(0.5f * r, fmaf(-d * r, r, 1.f), r);
    s = d * r;
    s = fmaf(fmaf(-s, s, d), 0.5f * r, s);
}
__device__ __forceinline__ void rsqrt_pair(double d, double& r, double& s)
{
    s = sqrt(d);
    r = 1.0 / s;
}
__device__ __forceinline__ float sqrt_t(float d) { return sqrtf(d); }
__device__ __forceinline__ double sqrt_t(double d) { return sqrt(d); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }

// S[c * kLd + r] <- src(r, c) = src[c * ld + r] for r >= c, identity beyond nb,
// zero above the diagonal; every load of the thread in flight before the first
// store.  trans reads src(c, r) instead (a lower tile from an upper matrix).
template <bool CG, class T>
__device__ __forceinline__ void load_lower(T* S, const T* src, long long ld, int nb, bool trans)
{
    constexpr int kPer = kN * kN / kThreads;
    T v[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int q = threadIdx.x + u * kThreads, hi = q >> 6, lo = q & 63;
        const int r = trans ? hi : lo, c = trans ? lo : hi;  // memory (lo, hi) of src
        const T* p = src + (long long)hi * ld + lo;
        v[u] = (r < nb && c <= r) ? (CG ? __ldcg(p) : *p) : (r == c ? T(1) : T(0));
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int q = threadIdx.x + u * kThreads, hi = q >> 6, lo = q & 63;
        S[(trans ? lo : hi) * kLd + (trans ? hi : lo)] = v[u];
    }
}

// Panel width.  Its diagonal block sits in every panel thread's registers; 8
// beats 16 (11.0K against 13.7K cycles a tile), whose panel is bound by the FMA
// issue of its two warps.
constexpr int PW = 8;

// One panel of chol64 on the first two warps: every thread factors its own
// register copy of the PW x PW diagonal block and carries one row below it
// along, so a column costs a reciprocal square root, a multiply and FMAs with
// no exchange between lanes at all (a shuffle per multiplier measured 2.5x
// slower: 180 cycles a column).  Returns false, with nothing written, when a
// pivot is outside the fast range (failed, tiny, huge or NaN).
template <class T>
__device__ bool chol_panel_fast(T* S, int kb)
{
    const int tid = threadIdx.x;
    const int row = kb + PW + tid;
    T D[PW][PW], x[PW];  // D[c][r], r >= c
#pragma unroll
    for (int c = 0; c < PW; ++c) {
#pragma unroll
        for (int g = c / 4; g < PW / 4; ++g) {
            const Vec4<T> v = *reinterpret_cast<const Vec4<T>*>(S + (kb + c) * kLd + kb + 4 * g);
#pragma unroll
            for (int i = 0; i < 4; ++i) D[c][4 * g + i] = v.x[i];
        }
        x[c] = row < kN ? S[(kb + c) * kLd + row] : T(0);
    }
    asm volatile("bar.sync 1, 64;" ::: "memory");  // both warps hold the block: it may be written
    bool ok = true;
#pragma unroll
    for (int j = 0; j < PW; ++j) {
        ok = ok & fast_range(D[j][j]);
        T r;
        rsqrt_pair(D[j][j], r, D[j][j]);
        x[j] *= r;
#pragma unroll
        for (int i = j + 1; i < PW; ++i) D[j][i] *= r;
#pragma unroll
        for (int c = j + 1; c < PW; ++c) {
#pragma unroll
            for (int i = c; i < PW; ++i) D[c][i] = fma_t(-D[j][i], D[j][c], D[c][i]);
            x[c] = fma_t(-x[j], D[j][c], x[c]);
        }
    }
    if (!ok) return false;
    if (row < kN) {
#pragma unroll
        for (int c = 0; c < PW; ++c) S[(kb + c) * kLd + row] = x[c];
    }
    if (tid == 63) {  // the diagonal block; above its diagonal the input stays
#pragma unroll
        for (int c = 0; c < PW; ++c)
#pragma unroll
            for (int i = c; i < PW; ++i) S[(kb + c) * kLd + kb + i] = D[c][i];
    }
    return true;
}

// The same panel for pivots outside the fast range: IEEE operations, the pivot
// tested before each column.  One warp.  Returns the failing column of the
// panel or -1.
template <class T>
__device__ __noinline__ int chol_panel_careful(T* S, int kb)
{
    const int lane = threadIdx.x & 31;
    for (int j = kb; j < kb + PW; ++j) {
        const T d = S[j * kLd + j];
        __syncwarp();
        if (!(d > T(0))) return j - kb;
        const T s = sqrt_t(d), r = T(1) / s;
        for (int i = j + lane; i < kN; i += 32)
            S[j * kLd + i] = i == j ? s : S[j * kLd + i] * r;
        __syncwarp();
        for (int c = j + 1; c < kb + PW; ++c) {
            const T lc = S[j * kLd + c];
            for (int i = c + lane; i < kN; i += 32)
                S[c * kLd + i] = fma_t(-S[j * kLd + i], lc, S[c * kLd + i]);
        }
        __syncwarp();
    }
    return -1;
}

// Columns [c0, c1) of the tile, rows c0 .. 63 on or below the diagonal, minus
// the product of panel columns [kb, kb + kmax): thread t of nthr takes four
// rows of one column at a time.
template <int CW, class T>
__device__ __forceinline__ void chol_update(T* S, int kb, int kmax, int c0, int c1, int t, int nthr)
{
    for (int c = c0 + t % CW; c < c1; c += CW)
    for (int r = c0 + 4 * (t / CW); r < kN; r += 4 * (nthr / CW)) {
        if (r + 3 < c) continue;
        Vec4<T> acc = {};
        const T* p = S + kb * kLd;
#pragma unroll 8
        for (int k = 0; k < kmax; ++k, p += kLd) {
            const Vec4<T> a = *reinterpret_cast<const Vec4<T>*>(p + r);
            const T b = p[c];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc.x[i] = fma_t(a.x[i], b, acc.x[i]);
        }
        Vec4<T>* o = reinterpret_cast<Vec4<T>*>(S + c * kLd + r);
        Vec4<T> v = *o;
#pragma unroll
        for (int i = 0; i < 4; ++i) v.x[i] -= acc.x[i];
        *o = v;
    }
}

// Cholesky of the lower tile in S (identity beyond nb); S is complete on entry
// (barrier before) and on return (barrier inside).  Returns the first column
// whose updated diagonal is not > 0 (or is NaN), or -1, the same in every
// thread.  On failure the columns before it are factored and applied to the
// rest, the failing diagonal holds its updated value.
// Look-ahead: after a panel all warps update only the next panel's columns;
// the rest of that update runs on warps 2..7 beside the next panel.
template <class T>
__device__ int chol64(T* S, int nb, int* s_fail)
{
    const int tid = threadIdx.x;
    for (int kb = 0; kb < nb; kb += PW) {
        if (tid == 0) *s_fail = -1;
        bool ok = true;
        if (tid < 64) ok = chol_panel_fast(S, kb);
        else if (kb > 0) chol_update<16>(S, kb - PW, PW, kb + PW, kN, tid - 64, kThreads - 64);
        if (__syncthreads_or(!ok)) {
            if (tid < 32) {
                const int f = chol_panel_careful(S, kb);
                if (tid == 0) *s_fail = f < 0 ? -1 : kb + f;
            }
            __syncthreads();
            const int fail = *s_fail;
            if (fail >= 0) {
                chol_update<16>(S, kb, fail - kb, kb + PW, kN, tid, kThreads);
                __syncthreads();
                return fail;
            }
        }
        if (kb + PW < kN) {
            chol_update<PW>(S, kb, PW, kb + PW, kb + 2 * PW, tid, kThreads);
            __syncthreads();
        }
    }
    return -1;
}

// The lower part (nb x nb) of S to dst(r, c) = dst[c * ld + r].
template <class T>
__device__ __forceinline__ void store_lower(T* dst, const T* S, long long ld, int nb)
{
#pragma unroll
    for (int u = 0; u < kN * kN / kThreads; ++u) {
        const int q = threadIdx.x + u * kThreads, c = q >> 6, r = q & 63;
        if (r < nb && c <= r) dst[(long long)c * ld + r] = S[c * kLd + r];
    }
}

// All of W, packed: dst[c * 64 + r] (trans: dst[r * 64 + c]) = W(r, c).
template <class T>
__device__ __forceinline__ void store_inv(T* dst, const T* W, bool trans)
{
#pragma unroll
    for (int u = 0; u < kN * kN / kThreads; ++u) {
        const int q = threadIdx.x + u * kThreads, hi = q >> 6, lo = q & 63;
        dst[q] = trans ? W[lo * kLd + hi] : W[hi * kLd + lo];
    }
}

// How a substitution divides by the diagonal: not at all (unit); by a reciprocal; by a
// reciprocal and one correction, q += r (x - d q) (Markstein, IBM J. Res. Dev. 34,
// 1990: the rounded quotient but for rare ties), or, where the diagonal leaves the
// range in which the residual is exact, by division instead.  Against division everywhere, the plain reciprocal gives
// the same errors or less in solves with Cholesky factors (right-side TRSM 3 %,
// POTRS 4 %), but 4-7 % more in U^{-1} and solves with U, which take the correction
// (0.2 us a tile, in a launch of its own and not on a factorization's chain).
enum Divide { kUnit, kReciprocal, kCorrected, kPlain };

// x <- inverse of the 16 x 16 lower block D (pitch kLd, 16-byte aligned) times x, in
// registers; D by broadcast loads of four rows, rd the reciprocals of its diagonal.
template <Divide HOW, class T>
__device__ __forceinline__ void substitute16(T x[16], const T* D, const T* rd)
{
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        T d[16];
#pragma unroll
        for (int g = (HOW == kCorrected || HOW == kPlain ? k : k + 1) / 4; g < 4; ++g) {
            const Vec4<T> v = *reinterpret_cast<const Vec4<T>*>(D + k * kLd + 4 * g);
#pragma unroll
            for (int i = 0; i < 4; ++i) d[4 * g + i] = v.x[i];
        }
        if (HOW == kReciprocal) {
            x[k] *= rd[k];
        } else if (HOW == kCorrected) {
            const T q = x[k] * rd[k];
            x[k] = fma_t(fma_t(-d[k], q, x[k]), rd[k], q);
        } else if (HOW == kPlain) {
            x[k] = x[k] / d[k];
        }
#pragma unroll
        for (int i = k + 1; i < 16; ++i) x[i] = fma_t(-d[i], x[k], x[i]);
    }
}
template <class T>
__device__ __noinline__ void substitute16_plain(T* x, const T* D)
{
    T v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = x[i];
    substitute16<kPlain>(v, D, D);
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = v[i];
}
template <Divide HOW, class T>
__device__ __forceinline__ void solve16(T x[16], const T* D, const T* rd, bool fast)
{
    if (HOW == kCorrected && !fast) substitute16_plain(x, D);
    else substitute16<HOW>(x, D, rd);
}

// W <- inverse of the lower tile in S (upper part of S ignored; HOW kUnit: implicit
// ones on the diagonal), W[c * kLd + r], zero above the diagonal.  X: kScratch
// entries, rd: 64.  S complete on entry; W complete on return.
template <Divide HOW, class T>
__device__ void inv64(const T* __restrict__ S, T* __restrict__ W, T* __restrict__ X,
                      T* __restrict__ rd)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int q = tid; q < kN * kLd; q += kThreads) W[q] = T(0);
    bool fast = true;
    if (tid < kN && HOW != kUnit) {
        const T d = S[tid * kLd + tid];
        rd[tid] = T(1) / d;
        fast = d * d > T(1e-36) && d * d < T(1e36);
    }
    if (HOW == kCorrected) fast = __syncthreads_and(fast);
    else __syncthreads();
    if (warp < 4 && lane < 16) {
        const int b = warp * 16;
        T x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = i == lane ? T(1) : T(0);
        solve16<HOW>(x, S + b * kLd + b, rd + b, fast);
#pragma unroll
        for (int i = 0; i < 16; ++i) W[(b + lane) * kLd + b + i] = x[i];
    }
    __syncthreads();
    {  // two pairs of 16 x 16 blocks: L21 W11, two rows of one column per thread
        const int b = (tid >> 7) * 32, c = (tid & 127) >> 3, r = (tid & 7) * 2;
        T* Xp = X + (tid >> 7) * 272;
        T t0 = T(0), t1 = T(0);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const T w = W[(b + c) * kLd + b + k];
            const T* l = S + (b + k) * kLd + b + 16 + r;
            t0 = fma_t(l[0], w, t0);
            t1 = fma_t(l[1], w, t1);
        }
        Xp[c * 17 + r] = t0;
        Xp[c * 17 + r + 1] = t1;
    }
    __syncthreads();
    if (warp < 2 && lane < 16) {  // a warp per pair, a column per lane
        const int b = warp * 32;
        T x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = -X[warp * 272 + lane * 17 + i];
        solve16<HOW>(x, S + (b + 16) * kLd + b + 16, rd + b + 16, fast);
#pragma unroll
        for (int i = 0; i < 16; ++i) W[(b + lane) * kLd + b + 16 + i] = x[i];
    }
    __syncthreads();
    {  // the pair of 32 x 32 blocks: L21 W11, four rows of one column per thread
        const int c = tid >> 3, r = (tid & 7) * 4;
        Vec4<T> t = {};
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const T w = W[c * kLd + k];
            const Vec4<T> l = *reinterpret_cast<const Vec4<T>*>(S + k * kLd + 32 + r);
#pragma unroll
            for (int i = 0; i < 4; ++i) t.x[i] = fma_t(l.x[i], w, t.x[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) X[c * 33 + r + i] = t.x[i];
    }
    __syncthreads();
    if (warp == 0) {  // its first 16 rows, a column per lane
        T x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = -X[lane * 33 + i];
        solve16<HOW>(x, S + 32 * kLd + 32, rd + 32, fast);
#pragma unroll
        for (int i = 0; i < 16; ++i) W[lane * kLd + 32 + i] = x[i];
    }
    __syncthreads();
    {  // their part in the last 16, two rows of one column per thread: a sum of its own,
       // or (kCorrected) the next links of the column's one chain
        constexpr bool kChain = HOW == kCorrected;
        const int c = tid >> 3, r = (tid & 7) * 2;
        T* x = X + c * 33 + 16 + r;
        T t0 = kChain ? x[0] : T(0), t1 = kChain ? x[1] : T(0);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const T w = W[c * kLd + 32 + k];
            const T* l = S + (32 + k) * kLd + 48 + r;
            t0 = fma_t(l[0], w, t0);
            t1 = fma_t(l[1], w, t1);
        }
        x[0] = kChain ? t0 : x[0] + t0;
        x[1] = kChain ? t1 : x[1] + t1;
    }
    __syncthreads();
    if (warp == 0) {
        T x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = -X[lane * 33 + 16 + i];
        solve16<HOW>(x, S + 48 * kLd + 48, rd + 48, fast);
#pragma unroll
        for (int i = 0; i < 16; ++i) W[lane * kLd + 48 + i] = x[i];
    }
    __syncthreads();
}

}  // namespace tile64
}  // namespace hdbf
