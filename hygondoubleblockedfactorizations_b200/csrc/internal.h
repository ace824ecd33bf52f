// Internal declarations shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <vector>

#include "hdbf/hdbf.h"

namespace hdbf {
// Kernel classes for the per-launch event profiler (hdbf_profile_*).  The names that
// callers see (hdbf_profile_class_name) stay as they were first given.
enum KernelClass {
    kClsGemm = 0,     // sgemm_sub_kernel, gemm_small_kernel and the FP64 GEMMs
    kClsPotf2 = 1,    // potf2_kernel
    kClsTrsmR = 2,    // rlt_block_kernel ("rlt_apply_kernel")
    kClsTrsmL = 3,    // llu_block_kernel, llu_apply_kernel ("llu_apply_kernel")
    kClsPanel = 4,    // getf2_cluster_kernel / getf2_grid_kernel
    kClsCompose = 5,  // compose_swaps_kernel, ipiv_to_perm's kernels
    kClsMoves = 6,    // swap_rows_kernel, apply_moves kernels
    kClsTrsmInv = 7,  // tri_inv64_kernel
    kClsTcGemm = 8,   // tc_gemm_persistent_kernel / tc_gemm_sub_kernel / tc_sgemm_kernel
    kClsConvert = 9,  // FP32 -> 16-bit shadow and word conversions
    kClsIr = 10,      // FP64 residual / update / norm kernels
    kClsOther = 11,
    kClsWave = 12,     // trsv_wave_kernel (wavefront triangular solves)
    kClsSkinny = 13,   // skinny_kernel (updates with N <= 32)
    kClsBatched = 14,  // batched_factor_solve_kernel
    kClsSelector = 15, // selector MLP kernels
    kClsPotrfBlock = 16, // potrf_cluster_kernel, tile_inverse_kernel ("potrf_block_kernel")
    kNumClasses = 17
};
// Algorithm stages of the double-blocked drivers for the per-stage profile
// (hdbf_profile_stages), named as the reference's stage profilers name them
// (src/potrf/profile_double_blocked_potrf.cpp, src/getrf/getrf_batched_pivot_internal.h).
enum Stage {
    kStNone = 0,
    kStPotrf,            // "POTRF": diagonal-block Cholesky
    kStTrsm,             // "TRSM": panel TRSM of the Cholesky
    kStInnerGemm,        // "Inner GEMM"
    kStOuterSyrk,        // "Outer SYRK"
    kStOuterGemm,        // "Outer GEMM"
    kStPanel,            // "Panel GETRF"
    kStPivotProp,        // "Pivot propagation" (immediate pivoting)
    kStInnerPivot,       // "Inner pivot batch"
    kStInnerTrsm,        // "Inner TRSM"
    kStOuterPivot,       // "Outer pivot batch"
    kStOuterTrsmBlock,   // "Outer TRSM block"
    kStOuterTrsmGemm,    // "Outer TRSM GEMM"
    kStOuterTrsmDirect,  // "Outer TRSM direct"
    kNumStages
};
struct ProfRec {
    int cls;
    cudaEvent_t a, b;
    double flops;
    double bytes;
    int m = 0, n = 0, k = 0;  // problem shape (GEMM launches)
    int stage = 0;            // Stage active when the launch was enqueued
    unsigned call = 0;        // which entry into that stage (StageScope instance)
};
struct GraphEntry {
    std::vector<long long> key;
    cudaGraphExec_t exec = nullptr;
    std::vector<ProfRec> prof;  // event pairs baked into the graph (profiling graphs)
    unsigned long long id = 0;
    unsigned long long last_use = 0;
    unsigned long long kernels = 0;  // kernel launches recorded in the graph
};
}  // namespace hdbf

namespace hdbf {
constexpr int kLaEvents = 3;  // two outer-update chunks per block, the join
}

struct hdbf_context {
    cudaStream_t stream = nullptr;
    int device = 0;
    int sm_count = 148;
    size_t max_smem_optin = 0;
    int cluster_max = 0;  // largest cluster the panel kernel can launch (0: none)
    int panel_mode = 0;   // hdbf_set_panel_kernel
    int panel_leaf = 128; // GETRF panel recursion leaf width (32, 64 or 128)
    int panel_rows = 256; // target rows per CTA of the grid-wide panel kernel
    // GETRF look-ahead (hdbf_set_lookahead): the panel chain of an outer block
    // runs on a high-priority internal stream while the caller's stream still
    // applies the outer update in two chunks; la_ev[c] marks chunk c done and
    // la_ev[kLaEvents - 1] joins the panel chain back.
    int lookahead = 1;
    cudaStream_t la_stream = nullptr;
    cudaEvent_t la_ev[hdbf::kLaEvents] = {};
    bool la_used = false;    // the graph being captured forked onto la_stream
    bool no_skinny = false;  // keep GEMMs off the shared split-K scratch
    // K chunk of the FP32 GEMM split (SplitPlan): -1 decides per launch,
    // 0 never splits, > 0 splits K into chunks of this many.  Column chunks of
    // one GEMM take the whole GEMM's plan so their sums match it bit for bit.
    int split_kc = -1;
    // Tensor-core GEMM kernel: 0 persistent 128 x 256 tiles with two TMEM
    // accumulators (default), 1 one 128 x 128 tile per CTA (HDBF_TC_KERNEL).
    int tc_kernel = 0;
    // FP32 updates on the tensor cores (three BF16 words, tc_sgemm.cu): 1 by
    // size, 0 never, 2 at any size (HDBF_TC_SGEMM).  tc_plan fixes the K
    // chunk for the parts of one GEMM, as split_kc does (-1: decide per launch).
    int tc_sgemm = 1;
    int tc_plan = -1;
    int small_plan = -1;  // the same for gemm_small_split (0: the 128 x 128 kernel)
    unsigned spin_limit = 0; // hdbf_set_wait_limit (0: default)
    // Conditional launches (RunIf): while set, the FP32 GEMM and the
    // diagonal-block kernel run only when *run_if != 0 (read on the device).
    const int* run_if = nullptr;
    // Device counter of panels the last mixed Cholesky rebuilt in FP32.
    unsigned* mixed_fallbacks = nullptr;
    // Stage attribution of profiled launches (StageScope) and the per-stage
    // split of the last profiling interval (hdbf_profile_stages).
    int stage = 0;
    unsigned stage_call = 0, stage_seq = 0;
    double stage_ms[32] = {}, stage_flops[32] = {};
    int stage_calls[32] = {};
    // Workspace arena (grown on demand outside stream capture).
    void* ws = nullptr;
    size_t ws_bytes = 0;
    int ws_n = 0;  // largest order whose layout fits in ws_bytes
    // Small always-present device block: [0] error word, [1..] barrier words.
    int* dev_small = nullptr;
    // Operand words of the FP32 updates on the tensor cores, for this handle's stream
    // and for its look-ahead stream; allocated by the calls that run such updates.
    void* words[2] = {nullptr, nullptr};
    size_t words_bytes[2] = {0, 0};
    // Second arena for the mixed-precision path (16-bit shadows, FP64 IR
    // vectors); grown on demand outside stream capture.
    void* mix = nullptr;
    size_t mix_bytes = 0;
    hdbf_status last_status = HDBF_STATUS_SUCCESS;
    unsigned long long launches = 0;
    // Optional per-launch event profiling.
    bool profiling = false;
    std::vector<hdbf::ProfRec> prof;
    // CUDA-graph cache of whole factorizations (key = entry point + arguments).
    bool use_graphs = true;
    bool capturing = false;
    cudaStream_t cap_stream = nullptr;
    std::vector<hdbf::GraphEntry> graphs;
    unsigned long long graph_clock = 0;
    std::vector<unsigned long long> prof_graph_ids;  // graphs replayed while profiling
};

struct hdbf_stream_pool {
    cudaStream_t* streams = nullptr;
    int count = 0;
};

namespace hdbf {

// Layout of hdbf_context::dev_small (ints).
constexpr int kSmallErr = 0;       // device error word (timeouts, invalid pivots)
constexpr int kSmallSpin = 8;        // bounded-wait poll limit of the handle (0: kSpinLimit)
constexpr int kSmallMoveCount = 12;  // move count of the last composed permutation
constexpr int kSmallEpoch = 16;      // panel-kernel exchange epoch
constexpr int kSmallDone = 20;       // panel-kernel finished-CTA counter
constexpr int kSmallScratch = 24;    // host-read reduction results (absmax etc.)
constexpr int kSmallBlockBar = 32;   // diagonal-block kernel: barrier counter, fail, abort
constexpr int kSmallInts = 64;

// Device error codes written into dev_small[kSmallErr]; the first error
// recorded stays (atomicCAS from 0) until hdbf_check_device_errors reads it.
constexpr int kErrTimeout = 1;
constexpr int kErrBadPivot = 2;

// Default bounded-wait poll limit for grid barriers (~0.5 s with back-off).
constexpr unsigned kSpinLimit = 1u << 22;

#ifdef __CUDACC__
// Per-panel power-of-two scale of the 16-bit shadows, from the panel's max |x|
// given as FP32 bits (written by an atomicMax over the panel): s = 2^k with
// max * s in [128, 256); 1 for a zero or non-finite max; k clamped to
// [-60, 60].  Exact (built from the exponent bits), so the converting kernel
// and the GEMM epilogue that undoes it agree bit for bit.
__device__ __forceinline__ int panel_scale_exp(unsigned maxbits)
{
    const int e = (int)((maxbits >> 23) & 0xffu);
    if (maxbits == 0u || e == 0xff) return 0;
    const int k = e == 0 ? 60 : 7 - (e - 127);
    return k < -60 ? -60 : (k > 60 ? 60 : k);
}
__device__ __forceinline__ float pow2f_exact(int k)
{
    return __uint_as_float((unsigned)(127 + k) << 23);
}

// Whether an operand pair is outside the range of the three-word BF16 split
// (tc_sgemm.cu): range[0], range[1] hold the bits of max |x| of A and of B (0: all
// zero, or B is part of A).  With exponents a and b the sum of K products, times 2^32, is
// below 2^(a + b + 2 + 32) K: no overflow for a + b <= 72 and K <= 2^20.  An operand
// wholly below 2^-90 keeps the FP32 kernel too.
__device__ __forceinline__ bool split_range_bad(const unsigned* range)
{
    unsigned ma = __ldcg(range), mb = __ldcg(range + 1);
    if (mb == 0u) mb = ma;
    if (ma == 0u) ma = mb;
    const unsigned a = ma >> 23, b = mb >> 23;  // biased exponents
    const bool tiny = ma != 0u && (a < 127u - 90u || b < 127u - 90u);
    return tiny || a > 127u + 110u || b > 127u + 110u || a + b > 2u * 127u + 72u;
}

// The handle's poll limit, read at kernel start from the small device block
// whose error word `err` points at (hdbf_set_wait_limit).
__device__ __forceinline__ unsigned spin_limit_of(const int* err)
{
    const unsigned v = *reinterpret_cast<const volatile unsigned*>(err + (kSmallSpin - kSmallErr));
    return v ? v : kSpinLimit;
}
#endif

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// RAII: when profiling is on, brackets one launch with a pair of events on
// ctx->stream and records its class and algorithmic work.
class ProfScope {
public:
    ProfScope(hdbf_context* ctx, int cls, double flops, double bytes = 0.0, int m = 0,
              int n = 0, int k = 0);
    ~ProfScope();
private:
    hdbf_context* ctx_;
    int idx_ = -1;
};

// RAII: launches enqueued while it lives are attributed to `stage` (one
// "call" of that stage per scope).
class StageScope {
public:
    StageScope(hdbf_context* ctx, int stage)
        : ctx_(ctx), prev_(ctx->stage), prev_call_(ctx->stage_call)
    {
        ctx->stage = stage;
        ctx->stage_call = ++ctx->stage_seq;
    }
    ~StageScope()
    {
        ctx_->stage = prev_;
        ctx_->stage_call = prev_call_;
    }
private:
    hdbf_context* ctx_;
    int prev_;
    unsigned prev_call_;
};

// RAII: launches of the conditional-capable kernels (FP32 GEMM, diagonal-block
// Cholesky, block-column restore) enqueued while it lives do their work only
// if *flag != 0 when they run; the skinny GEMM path is not taken meanwhile.
class RunIf {
public:
    RunIf(hdbf_context* ctx, const int* flag) : ctx_(ctx), prev_(ctx->run_if) { ctx->run_if = flag; }
    ~RunIf() { ctx_->run_if = prev_; }
private:
    hdbf_context* ctx_;
    const int* prev_;
};

// Make sure the workspace holds at least `bytes`; returns nullptr and sets
// *st on failure.  Growing frees the old buffer (device-synchronising).
void* workspace(hdbf_context* ctx, size_t bytes, hdbf_status* st);

// Mixed-path arena of at least `bytes` (same growth rules as the workspace).
void* mixed_arena(hdbf_context* ctx, size_t bytes, hdbf_status* st);

// Workspace layout for problems of order <= n (byte offsets):
//   panel  panel-kernel exchange slots (fixed size, offset 0)
//   inv   inverted 64x64 diagonal blocks, ceil(n/64)*4096 floats
//   src, tgt, gperm  composed row moves / permutation scratch, n ints each
//   temp  column-tiled swap buffer, 64*n floats
//   skinny  split-K partial sums of the skinny GEMM, 256*n floats
//   wave  wavefront-solve row-major x copy (32 columns) and its flags
struct WsLayout {
    size_t panel, inv, src, tgt, gperm, temp, skinny, wave, split, total;
};
// Split-K partial sums of under-filled FP32 GEMM launches: two halves of
// kSplitFloats each, one for the handle's stream and one for its look-ahead
// stream, so concurrent GEMMs on the two never share scratch.
constexpr size_t kSplitFloats = (size_t)32 << 20;
WsLayout ws_layout(int n);
// Guarantee the layout for order n (grows the arena outside stream capture).
hdbf_status ensure_ws(hdbf_context* ctx, int n);
void* ws_panel(hdbf_context* ctx);
float* ws_inv(hdbf_context* ctx);
int* ws_src(hdbf_context* ctx);
int* ws_tgt(hdbf_context* ctx);
int* ws_gperm(hdbf_context* ctx);
float* ws_temp(hdbf_context* ctx);
float* ws_skinny(hdbf_context* ctx);
// Split-K scratch half for GEMMs enqueued on ctx->stream.
float* ws_split(hdbf_context* ctx);
float* ws_wave(hdbf_context* ctx);
// The operand words (256 bytes of range slots first) of updates on ctx->stream: their
// bytes for a factorization of order n, and their room, grown to `bytes` where no stream
// capture forbids it.  Without room the FP32 kernels do the update.
size_t words_bytes(int n);
bool words_room(hdbf_context* ctx, size_t bytes);
inline void* ws_words(const hdbf_context* ctx)
{
    return ctx->words[ctx->la_stream && ctx->stream == ctx->la_stream ? 1 : 0];
}
// Room for the updates of a factorization of order n (FP32 drivers, outside their
// capture), on the look-ahead stream too, or for one of M x N x K.
void reserve_words(hdbf_context* ctx, int n, bool lookahead);
void reserve_words(hdbf_context* ctx, int M, int N, int K);
template <class T>
inline void reserve_update_words(hdbf_context* ctx, int n, bool lookahead)
{
    if (sizeof(T) == 4) reserve_words(ctx, n, lookahead);
}

hdbf_status last_cuda(hdbf_context* ctx);

// ---------------------------------------------------------------- kernels
// All launchers enqueue on ctx->stream and count launches.

// C(M x N) -= A(M x K) * op(B); op(B) = B^T (B is N x K, nn=false) or B
// (B is K x N, nn=true).  lower_only: tiles wholly above the diagonal are
// skipped and only entries with row >= col (local to C) are written.
hdbf_status sgemm_sub(hdbf_context* ctx, bool nn, bool lower_only, int M, int N, int K,
                      const float* A, long long lda, const float* B, long long ldb,
                      float* C, long long ldc);

// K split of the FP32 GEMM of shape M x N x K (tri: lower-triangle mode):
// the number of chunks (1 = no split) and, in *kc, their length.
int split_count(const hdbf_context* ctx, int M, int N, int K, bool tri, int* kc);
// Updates below one wave of 128 x 128 tiles (gemm_small.cu): the CTAs that share
// a tile's K (0: not taken), the same where an FP32 update takes this kernel
// (sgemm.cu), and the launch (range: only if split_range_bad).
int gemm_small_split(const hdbf_context* ctx, int M, int N, int K);
int sgemm_small(const hdbf_context* ctx, int M, int N, int K, bool tri, bool vec);
// Tiles of b x b of an M x N update (tri: on or below the diagonal), and CTAs of
// one SM, the fullest, when `per` CTAs share each.
inline long long tile_count(int M, int N, int b, bool tri)
{
    const long long tm = (M + b - 1) / b, tn = (N + b - 1) / b;
    if (!tri) return tm * tn;
    const long long d = tm < tn ? tm : tn;
    return d * tm - d * (d - 1) / 2;
}
inline long long small_waves(const hdbf_context* ctx, int M, int N, bool tri, int per)
{
    const long long sm = ctx->sm_count, all = (tile_count(M, N, 64, false) * per + sm - 1) / sm;
    const long long own = (tile_count(M, N, 64, tri) * per + sm - 1) / sm;
    return tri && own < all ? own + 1 : own;  // tiles above the diagonal leave holes
}
hdbf_status gemm_small(hdbf_context* ctx, bool nn, bool lower, int S, int M, int N, int K,
                       const float* A, long long lda, const float* B, long long ldb, float* C,
                       long long ldc, const unsigned* range = nullptr);
hdbf_status gemm_small(hdbf_context* ctx, bool nn, bool lower, int S, int M, int N, int K,
                       const double* A, long long lda, const double* B, long long ldb, double* C,
                       long long ldc);
void configure_gemm_small(hdbf_context* ctx);
void configure_tile_kernels(hdbf_context* ctx);
// FP32 update on the tensor cores (tc_sgemm.cu): the K chunk for this shape, 0
// where the FP32 kernel is taken; one chunk of it (a_kc / b_kc: the operand's K
// is contiguous), whose operand range, in *range, tells the FP32 kernel behind it
// whether it has to do the update (split_range_bad).  NOT_SUPPORTED, with nothing
// launched, where the operands' tensor maps cannot be encoded.
int tc_sgemm_chunk(const hdbf_context* ctx, int M, int N, int K, bool tri);
// The same, or 0 where there is no room for the operands' words.
int tc_sgemm_plan(hdbf_context* ctx, int M, int N, int K, bool tri);
hdbf_status tc_sgemm_chunk_run(hdbf_context* ctx, bool a_kc, bool b_kc, bool lower, int M, int N,
                               int K, const float* A, long long lda, const float* B, long long ldb,
                               float* C, long long ldc, unsigned** range);
void configure_tc_sgemm(hdbf_context* ctx);
// While alive, every FP32 GEMM splits K as the GEMM of the given shape does.
struct SplitPlan {
    hdbf_context* ctx;
    int saved, saved_tc, saved_small;
    SplitPlan(hdbf_context* c, int M, int N, int K)
        : ctx(c), saved(c->split_kc), saved_tc(c->tc_plan), saved_small(c->small_plan)
    {
        int kc = 0;
        c->tc_plan = tc_sgemm_plan(c, M, N, K, false);
        c->small_plan = sgemm_small(c, M, N, K, false, true);
        const int S = split_count(c, M, N, K, false, &kc);
        c->split_kc = S > 1 ? kc : 0;
    }
    ~SplitPlan()
    {
        ctx->small_plan = saved_small;
        ctx->split_kc = saved;
        ctx->tc_plan = saved_tc;
    }
};

// Skinny update (N <= 32): mode 0 C -= A * B^T, 1 C -= A * B, 2 C -= A^T * B,
// with the operand shapes of sgemm_sub / sgemm_sub_tn.  sgemm_launch routes
// narrow non-triangular updates here.
hdbf_status sgemm_skinny(hdbf_context* ctx, int mode, int M, int N, int K, const float* A,
                         long long lda, const float* B, long long ldb, float* C, long long ldc);
size_t skinny_partial_floats(int n);

// C(M x N) -= A^T * B with A stored K x M and B stored K x N (column-major).
hdbf_status sgemm_sub_tn(hdbf_context* ctx, int M, int N, int K, const float* A, long long lda,
                         const float* B, long long ldb, float* C, long long ldc);

// Cholesky of an n x n (n <= 64) diagonal block; with inv also the inverse of
// its factor (one tri_inv64 block).
hdbf_status potf2_small(hdbf_context* ctx, int n, float* A, long long lda, int* info,
                        int info_base, float* inv = nullptr);

// Inverses of the 64x64 diagonal blocks of lower-triangular L (order n) into
// out[b*4096 ...] (column-major blocks); unit selects an implicit unit diagonal.
hdbf_status tri_inv64(hdbf_context* ctx, int n, const float* L, long long ldl, bool unit,
                      float* out);
// Inverse modes: 0 lower non-unit, 1 lower unit, 2 upper non-unit.
hdbf_status tri_inv64_mode(hdbf_context* ctx, int n, const float* L, long long ldl, int mode,
                           float* out);
// B(rows <= 256 x cols) <- L^{-1} B for unit lower L in one launch (block
// forward substitution with the 64x64 inverses in inv, trsm_block.cu).
hdbf_status llu_block(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                      const float* inv, float* B, long long ldb);
hdbf_status llu_block(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                      const double* inv, double* B, long long ldb);
int llu_block_max_rows();
// B(rows x cols <= 256) <- B L^{-T}, L lower non-unit, same scheme.
hdbf_status rlt_block(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                      const float* inv, float* B, long long ldb);
hdbf_status rlt_block(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                      const double* inv, double* B, long long ldb);
void configure_trsm_block_kernels(hdbf_context* ctx);
// B <- inv * B (trans=false) or inv^T * B (trans=true), rows <= 64.
hdbf_status llu_apply_t(hdbf_context* ctx, int rows, int cols, const float* inv, float* B,
                        long long ldb, bool trans);

// Solves on FP32 factors (solves.cu).
hdbf_status ipiv_to_perm(hdbf_context* ctx, const int* ipiv, int n, int* perm);
hdbf_status gather_rows_perm(hdbf_context* ctx, const float* src, long long lds, float* dst,
                             long long ldd, const int* perm, int n, int cols);
hdbf_status potrs_f32(hdbf_context* ctx, const float* L, long long ldl, int n, int nrhs, float* B,
                      long long ldb);
hdbf_status getrs_f32_permuted(hdbf_context* ctx, const float* LU, long long ldlu, int n, int nrhs,
                               float* B, long long ldb);
void configure_solve_kernels(hdbf_context* ctx);

// Wavefront block triangular solve (trsm_wave.cu): B <- op(M)^{-1} B, M = T
// (trans false) or T^T (trans true); forward for a lower M, backward for an
// upper one.  inv holds the 64x64 diagonal-block inverses of T from
// tri_inv64_mode (applied transposed when trans is set).  One launch per 32
// right-hand-side columns.
hdbf_status trsv_wave(hdbf_context* ctx, int n, int nrhs, const float* T, long long ldt, bool trans,
                      const float* inv, bool backward, float* B, long long ldb);
size_t wave_scratch_bytes(int n);
void configure_wave_kernels(hdbf_context* ctx);
void configure_batched_kernels(hdbf_context* ctx);

// Partially pivoted LU of an m x w panel leaf, FP32 and FP64.  Pivots are written
// 1-based as (local row + 1 + ipiv_add).  On one thread-block cluster with the
// block in distributed shared memory (getf2_cluster.cu), or grid-wide with rows in
// registers (getf2_grid.cu); NOT_SUPPORTED when w is above getf2_*_leaf(m).
hdbf_status getf2_cluster(hdbf_context* ctx, int m, int w, float* A, long long lda, int* ipiv,
                          int ipiv_add, int* info, int info_base, bool pivot);
hdbf_status getf2_cluster(hdbf_context* ctx, int m, int w, double* A, long long lda, int* ipiv,
                          int ipiv_add, int* info, int info_base, bool pivot);
hdbf_status getf2_grid(hdbf_context* ctx, int m, int w, float* A, long long lda, int* ipiv,
                       int ipiv_add, int* info, int info_base, bool pivot);
hdbf_status getf2_grid(hdbf_context* ctx, int m, int w, double* A, long long lda, int* ipiv,
                       int ipiv_add, int* info, int info_base, bool pivot);
// Widest leaf that one cluster, or the grid, holds at height m for elements of
// `elem` bytes (0: none).
int getf2_cluster_leaf(hdbf_context* ctx, int m, int elem);
int getf2_grid_leaf(hdbf_context* ctx, int m, int elem);
size_t getf2_grid_scratch_bytes();
// The leaf the panel recursion takes on the cluster kernel (0: the grid-wide one).
int panel_cluster_leaf(hdbf_context* ctx, int m, int elem);
void configure_getrf_kernels(hdbf_context* ctx);
void configure_grid_panel(hdbf_context* ctx);
int configure_cluster_panel(hdbf_context* ctx);

// Compose LAPACK swaps  row (i) <-> row (ipiv[i]-1-ipiv_minus), i in [0,k),
// over local rows [0, m) into (src, tgt, *count) moves (at most 2k): rows
// [0, k) in order, then the distinct pivot rows >= k in increasing order.
// k <= 4096 runs without replaying the swaps (sorted-group composition, O(k)
// rows touched); longer sequences are replayed by one thread over perm[m]
// (gperm when m ints do not fit in shared memory).
hdbf_status compose_swaps(hdbf_context* ctx, const int* ipiv, int k, int ipiv_minus, int m,
                          int* src, int* tgt, int* count, int* gperm, int* info);
// The same swaps, composed and applied in one launch (NOT_SUPPORTED above 512
// swaps and where the two launches are faster), to columns [c0, c0 + n0) and
// [c1, c1 + n1) of A, whose row 0 is the swaps' row 0.  A pivot outside [its row, m) moves nothing, sets info = -1 and the
// device error.
hdbf_status swap_rows(hdbf_context* ctx, float* A, long long lda, const int* ipiv, int k, int minus,
                      int m, int c0, int n0, int c1, int n1, int* info);
hdbf_status swap_rows(hdbf_context* ctx, double* A, long long lda, const int* ipiv, int k, int minus,
                      int m, int c0, int n0, int c1, int n1, int* info);
// A[tgt[i], c] = old A[src[i], c] for c < ncols, i < *count (<= max_moves).
hdbf_status apply_moves(hdbf_context* ctx, float* A, long long lda, int ncols,
                        const int* src, const int* tgt, const int* count, int max_moves,
                        float* temp, long long temp_cols);

// ------------------------------------------------ tensor-core (tcgen05) path
// A K-major 16-bit operand: row r, element k at base[(row0 + r) * ld + k0 + k].
struct TcOperand {
    const void* base = nullptr;
    long long ld = 0;  // elements; multiple of 8
    int row0 = 0;
    int k0 = 0;        // multiple of 8
};
constexpr int kFmtF16 = 0;   // IEEE binary16
constexpr int kFmtBF16 = 1;  // bfloat16
// C(M x N, FP32 column-major) -= scale * A * B^T on the tensor cores.
// Optional device scales (sa_max / sb_max: panel max bits, see
// panel_scale_exp): the epilogue then uses scale / (s_a s_b).
hdbf_status tc_gemm_sub(hdbf_context* ctx, int fmt, int M, int N, int K, const TcOperand& A,
                        const TcOperand& B, float* C, long long ldc, float scale, bool lower_only,
                        const unsigned* sa_max = nullptr, const unsigned* sb_max = nullptr);
// C -= scale * (A B^T + A Blo^T + Alo B^T): the split-precision product in one
// launch (hi/lo operands share row/K origins), one FP32 accumulator in TMEM.
hdbf_status tc_gemm_sub_split(hdbf_context* ctx, int fmt, int M, int N, int K, const TcOperand& A,
                              const TcOperand& Alo, const TcOperand& B, const TcOperand& Blo,
                              float* C, long long ldc, float scale, bool lower_only,
                              const unsigned* sa_max = nullptr, const unsigned* sb_max = nullptr);
void configure_tc_kernels(hdbf_context* ctx);
// dst(r, k) = round16(s * src(r, k)) for an rows x cols FP32 column-major block
// into a K-major (row-major, ldd elements) 16-bit block; `hi_lo` additionally
// writes the rounding residual round16(s*src - hi) into lo (may be null).
// smax (optional): device max bits of the panel; the scale is then
// 2^panel_scale_exp(*smax) instead of s.
hdbf_status convert_transpose16(hdbf_context* ctx, int fmt, int rows, int cols, const float* src,
                                long long lds, void* hi, void* lo, long long ldd, float s,
                                const unsigned* smax = nullptr);
// dst[c * ldd + r] = round16(s * src[c * lds + r]): same layout (column-major
// FP32 -> "column = K-major row" 16-bit), with optional residual.
hdbf_status convert_direct16(hdbf_context* ctx, int fmt, int rows, int cols, const float* src,
                             long long lds, void* hi, void* lo, long long ldd, float s,
                             const unsigned* smax = nullptr);
// *slot = FP32 bits of max |A(r, c)| over rows x cols (slot cleared first).
hdbf_status panel_absmax(hdbf_context* ctx, const float* A, long long lda, int rows, int cols,
                         unsigned* slot);

// Auxiliary kernels.
hdbf_status fill_uniform(hdbf_context* ctx, float* x, size_t count, uint64_t seed,
                         uint64_t offset);
hdbf_status add_damping(cudaStream_t s, float* A, int n, long long lda, float lambda);

// ---------------------------------------------------------------- drivers
// Cholesky of an n x n (n <= potrf_block_max_n()) diagonal block on one cluster;
// with W non-null also W = L^{-1} (lower, upper zeroed), in a second launch.
hdbf_status potrf_block(hdbf_context* ctx, int n, float* A, long long lda, int* info,
                        int info_base, float* W, long long ldw, bool last = false);
int potrf_block_max_n();
void configure_potrf_block(hdbf_context* ctx);
// Orders up to potrf_block_max_n() also leave the 64x64 diagonal-block
// inverses of the factor in ws_inv, for a trsm_rlt_ready with the same block;
// not the last one with `last` (nothing below the block).
hdbf_status potrf_diag(hdbf_context* ctx, int n, float* A, long long lda, int* info,
                       int info_base, bool last);
hdbf_status trsm_rlt(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                     float* B, long long ldb);
// trsm_rlt against the block that potrf_diag has just factored on this stream.
hdbf_status trsm_rlt_ready(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                           float* B, long long ldb);
hdbf_status trsm_llu(hdbf_context* ctx, int rows, int cols, const float* L, long long ldl,
                     float* B, long long ldb);
// Create the look-ahead stream and events (outside stream capture).
hdbf_status ensure_lookahead(hdbf_context* ctx);
hdbf_status syrk_lower(hdbf_context* ctx, int n, int k, const float* A, long long lda,
                       float* C, long long ldc);
struct GetrfWs {
    int* src = nullptr;    // composed move sources (n ints)
    int* tgt = nullptr;    // composed move targets (n ints)
    int* count = nullptr;  // device move count
    int* gperm = nullptr;  // global permutation scratch (n ints) for very tall panels
    float* temp = nullptr;  // column-tiled swap buffer
    long long temp_cols = 0;
};
// A part's interchanges on columns [c0, c0 + nc) of its rows (drivers.cu).
hdbf_status panel_swaps(hdbf_context* ctx, float* A, long long lda, const int* ipiv, int k,
                        int ipiv_add, int m, int c0, int nc, int* info, const GetrfWs& ws);
hdbf_status panel_swaps(hdbf_context* ctx, double* A, long long lda, const int* ipiv, int k,
                        int ipiv_add, int m, int c0, int nc, int* info, const GetrfWs& ws);
// Carve the factorization workspace for order n (reserves it first).
hdbf_status getrf_workspace(hdbf_context* ctx, int n, GetrfWs* ws);
hdbf_status getrf_panel(hdbf_context* ctx, int m, int w, float* A, long long lda, int* ipiv,
                        int ipiv_add, int* info, int info_base, bool pivot, const GetrfWs& ws);

// ---------------------------------------------------------------- FP64
// Overloads of the primitives above for the `_double` entry points
// (fp64.cu).  The FP64 workspace is the FP32 layout of order 2n.
inline hdbf_status gemm_sub(hdbf_context* ctx, bool nn, bool lower_only, int M, int N, int K,
                            const float* A, long long lda, const float* B, long long ldb,
                            float* C, long long ldc)
{
    return sgemm_sub(ctx, nn, lower_only, M, N, K, A, lda, B, ldb, C, ldc);
}
hdbf_status gemm_sub(hdbf_context* ctx, bool nn, bool lower_only, int M, int N, int K,
                     const double* A, long long lda, const double* B, long long ldb, double* C,
                     long long ldc);
hdbf_status gemm_sub_tn(hdbf_context* ctx, int M, int N, int K, const double* A, long long lda,
                        const double* B, long long ldb, double* C, long long ldc);
hdbf_status potf2_small(hdbf_context* ctx, int n, double* A, long long lda, int* info,
                        int info_base, double* inv = nullptr);
hdbf_status tri_inv64(hdbf_context* ctx, int n, const double* L, long long ldl, bool unit,
                      double* out);
hdbf_status trsm_rlt(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                     double* B, long long ldb);
// After potrf_diag of order <= 64 the inverse is ready; above, it is formed here.
hdbf_status trsm_rlt_ready(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                           double* B, long long ldb);
hdbf_status trsm_llu(hdbf_context* ctx, int rows, int cols, const double* L, long long ldl,
                     double* B, long long ldb);
hdbf_status syrk_lower(hdbf_context* ctx, int n, int k, const double* A, long long lda,
                       double* C, long long ldc);
hdbf_status potrf_diag(hdbf_context* ctx, int n, double* A, long long lda, int* info,
                       int info_base, bool last);
hdbf_status apply_moves(hdbf_context* ctx, double* A, long long lda, int ncols, const int* src,
                        const int* tgt, const int* count, int max_moves, double* temp,
                        long long temp_cols);
hdbf_status getrf_panel(hdbf_context* ctx, int m, int w, double* A, long long lda, int* ipiv,
                        int ipiv_add, int* info, int info_base, bool pivot, const GetrfWs& ws);
// Workspace order for a problem of order n in scalar type T: FP64 needs the
// FP32 layout of twice as many whole 64-row blocks (the inverse-block table
// holds 4096 doubles per block).
template <class T>
inline int ws_order(int n) { return sizeof(T) == 8 ? 2 * ((n + 63) / 64 * 64) : n; }
// Graph-cache key tag separating the FP32 and FP64 drivers.
template <class T>
inline long long type_tag() { return sizeof(T) == 8 ? 1000 : 0; }

// ---------------------------------------------------------------- graphs
// A whole factorization is a long chain of dependent launches; replaying it
// as one CUDA graph removes the per-launch host cost.  The first call with a
// given key records the work on a private capture stream; later calls with
// the same key replay the instantiated graph on the caller's stream.  The
// workspace must already be reserved (no allocation may happen inside).
GraphEntry* graph_find(hdbf_context* ctx, const std::vector<long long>& key);
bool graph_can_capture(hdbf_context* ctx);
hdbf_status graph_capture_begin(hdbf_context* ctx, cudaStream_t* saved);
hdbf_status graph_capture_end(hdbf_context* ctx, cudaStream_t saved, hdbf_status body_status,
                              const std::vector<long long>& key, size_t prof_mark,
                              unsigned long long launches_before);
hdbf_status graph_launch(hdbf_context* ctx, GraphEntry* e);
void graph_cache_clear(hdbf_context* ctx);

template <class Body>
hdbf_status run_graph(hdbf_context* ctx, std::vector<long long> key, Body&& body)
{
    if (!graph_can_capture(ctx)) return body();
    key.push_back(ctx->profiling ? 1 : 0);
    key.push_back(ctx->tc_sgemm);
    if (GraphEntry* e = graph_find(ctx, key)) return graph_launch(ctx, e);
    cudaStream_t saved = nullptr;
    const size_t mark = ctx->prof.size();
    const unsigned long long l0 = ctx->launches;
    if (graph_capture_begin(ctx, &saved) != HDBF_STATUS_SUCCESS) return body();
    const hdbf_status st = body();
    const hdbf_status ge = graph_capture_end(ctx, saved, st, key, mark, l0);
    if (ge == HDBF_STATUS_NOT_SUPPORTED) return body();  // capture refused: run eagerly
    return ge;
}

}  // namespace hdbf

#define HDBF_TRY(expr)                                   \
    do {                                                 \
        hdbf_status _st = (expr);                        \
        if (_st != HDBF_STATUS_SUCCESS) return _st;      \
    } while (0)
