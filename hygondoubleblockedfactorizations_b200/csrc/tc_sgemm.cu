// FP32 trailing updates on the tensor cores:  C -= op(A) * op(B)  with FP32
// operands carried as three BF16 words each.
//
// An FP32 value is the exact sum of three BF16 values, x = x0 + x1 + x2 (8
// significant bits each, rounded to nearest with signed remainders).  Of the
// nine products the six largest are formed, x0 y0, x0 y1, x1 y0, x1 y1, x0 y2
// and x2 y0; the three left out are below 2^-23 |x y| in the worst case and
// 2^-26 typically, under the rounding that an FP32 sum of the products makes.
// The tensor cores add into FP32 accumulators but truncate, so no sum stays
// there for long: an accumulator takes 64 values of K (the small products
// first, x0 y0 last), then the epilogue warps add it to FP32 registers with
// round-to-nearest adds, and those are subtracted from C at the end.  Error
// against FP64 over U[-1,1) operands, rms, relative to the rms of the product:
// K = 256 8.7e-8 (FP32 FMA chain 2.9e-7), K = 4096 1.5e-7 (1.2e-6); over [0,1)
// operands, whose sums only grow, K = 4096 1.2e-7 (8.5e-7).
//
// Bound: tensor pipe (6 x 2 M N K BF16 operations) and, through it, power.
// Kernel: as the 16-bit GEMM (tc_gemm.cu), one persistent CTA per SM over 128 x
// 256 tiles, a TMA producer warp, an MMA warp and here eight epilogue warps
// (128 accumulators per thread).  A ring slot holds one word of A (128 x 64)
// and of B (256 x 64), 48 KB, four slots; words arrive in the order 1, 0, 2 and
// are used as x1 y1 | x0 y1, x1 y0 | x0 y2, x2 y0 | x0 y0, so that every slot is
// free at least half a step before the word that reuses it is needed.  Two
// TMEM accumulators alternate per 64 of K; draining one takes a quarter of the
// time the other takes to fill.
//
// Range: an FP32 value is a multiple of 2^-149, a BF16 word of 2^-133, so values are
// split times 2^16 and the sums taken off C times 2^-32: the split is then exact for
// every value below 2^111, subnormal ones included, row by row and entry by entry, and
// no result that FP32 can hold comes from a sum below the normal range.  The conversion
// records max |x| of each operand; where one is not finite, above 2^110 or below
// 2^-90, or their product so large that a scaled sum might overflow (2^74), these
// kernels leave C alone and the FP32 kernel, launched behind them, does the update (it
// returns at once otherwise).
#include "tc_common.cuh"

#include <cuda_bf16.h>

#include <algorithm>

namespace hdbf {
namespace {

constexpr int kTM = 128, kTN = 256, kTK = 64;
constexpr int kABytes = kTM * kTK * 2;
constexpr int kSlot = kABytes + kTN * kTK * 2;  // 48 KB
constexpr int kSlots = 4;
constexpr int kTmemCols = 2 * kTN;
constexpr int kEpiWarps = 8;
constexpr int kThr = 64 + 32 * kEpiWarps;
constexpr size_t kSmemBytes = (size_t)kSlots * kSlot + 1024;
constexpr float kSplitScale = 65536.f, kUnscale = 1.f / (65536.f * 65536.f);

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x,
                                            int y, int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

struct X6Args {
    int M, N, K;
    int b_row0;  // first row of B in its shadow
    float* C;
    long long ldc;
    int tiles_m, tiles_n;
    long long total;
    int lower;
    const unsigned* range;  // max bits of A and B
    int* err;
};

__global__ void __launch_bounds__(kThr, 1)
tc_sgemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                const X6Args args)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kSlots];
    __shared__ __align__(8) uint64_t empty_bar[kSlots];
    __shared__ __align__(8) uint64_t tfull_bar[2];
    __shared__ __align__(8) uint64_t tempty_bar[2];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_fail;

    if (split_range_bad(args.range)) return;
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    auto sA = [&](int st) { return smem + st * kSlot; };
    auto sB = [&](int st) { return smem + st * kSlot + kABytes; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* fail = &s_fail;

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_slot)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull_bar[b], 1);
            mbar_init(&tempty_bar[b], kEpiWarps);
        }
        mbar_init(&done_bar, 1);
        s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t taddr = tmem_slot;
    const int ktiles = (args.K + kTK - 1) / kTK;
    const long long G = gridDim.x;

    if (warp == 0) {
        if (lane == 0) {  // TMA producer
            TileWalk walk;
            uint32_t it = 0;
            bool ok = true;
            for (long long t = blockIdx.x; t < args.total && ok; t += G) {
                int tm, tn;
                walk.locate(args, t, tm, tn);
                const int m0 = tm * kTM, n0 = args.b_row0 + tn * kTN;
                for (int kt = 0; kt < ktiles && ok; ++kt) {
#pragma unroll
                    for (int q = 0; q < 3; ++q, ++it) {
                        const int word = q == 0 ? 1 : (q == 1 ? 0 : 2);
                        const int s = (int)(it % kSlots);
                        if (it >= (uint32_t)kSlots &&
                            !mbar_wait_or_fail(&empty_bar[s], ((it / kSlots) - 1) & 1, args.err,
                                               fail)) {
                            ok = false;
                            break;
                        }
                        mbar_expect_tx(&full_bar[s], kSlot);
                        tma_load_3d(sA(s), &mapA, &full_bar[s], kt * kTK, m0, word);
                        tma_load_3d(sB(s), &mapB, &full_bar[s], kt * kTK, n0, word);
                    }
                }
            }
            if (!ok) {  // let the copies already issued land before the CTA exits
                const uint32_t first = it > (uint32_t)kSlots ? it - kSlots : 0u;
                for (uint32_t q = first; q < it; ++q) {
                    const long long t0 = clock64();
                    while (!mbar_try_wait(&full_bar[q % kSlots], (q / kSlots) & 1) &&
                           clock64() - t0 < kWaitCycles) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {  // MMA issuer
            const uint32_t idesc = make_idesc_n(kFmtBF16, kTN);
            uint32_t it = 0, chunk = 0;
            bool ok = true;
            for (long long t = blockIdx.x; t < args.total && ok; t += G) {
                for (int kt = 0; kt < ktiles && ok; ++kt, ++chunk) {
                    const int buf = (int)(chunk & 1);
                    if (chunk >= 2 && !mbar_wait_or_fail(&tempty_bar[buf], ((chunk >> 1) - 1) & 1,
                                                         args.err, fail)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t d = taddr + (uint32_t)(buf * kTN);
                    auto mma = [&](uint32_t a0, uint32_t b0, bool first) {
#pragma unroll
                        for (int kk = 0; kk < kTK / 16; ++kk) {
                            const uint32_t acc = (first && kk == 0) ? 0u : 1u;
                            asm volatile(
                                "{\n\t.reg .pred p;\n\t"
                                "setp.ne.b32 p, %4, 0;\n\t"
                                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(
                                    d),
                                "l"(sw128_desc(a0 + kk * 32)), "l"(sw128_desc(b0 + kk * 32)),
                                "r"(idesc), "r"(acc));
                        }
                    };
                    auto commit = [&](uint64_t* bar) {
                        asm volatile(
                            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 "
                            "[%0];" ::"r"(smem_u32(bar))
                            : "memory");
                    };
                    auto wait_full = [&](uint32_t q) {
                        const bool got = mbar_wait_or_fail(&full_bar[q % kSlots], (q / kSlots) & 1,
                                                           args.err, fail);
                        asm volatile("tcgen05.fence::after_thread_sync;");
                        return got;
                    };
                    const int s1 = (int)(it % kSlots), s0 = (int)((it + 1) % kSlots),
                              s2 = (int)((it + 2) % kSlots);
                    const uint32_t a1 = smem_u32(sA(s1)), b1 = smem_u32(sB(s1));
                    const uint32_t a0 = smem_u32(sA(s0)), b0 = smem_u32(sB(s0));
                    const uint32_t a2 = smem_u32(sA(s2)), b2 = smem_u32(sB(s2));
                    if (!(ok = wait_full(it))) break;
                    mma(a1, b1, true);
                    if (!(ok = wait_full(it + 1))) break;
                    mma(a0, b1, false);
                    mma(a1, b0, false);
                    commit(&empty_bar[s1]);
                    if (!(ok = wait_full(it + 2))) break;
                    mma(a0, b2, false);
                    mma(a2, b0, false);
                    commit(&empty_bar[s2]);
                    mma(a0, b0, false);
                    commit(&empty_bar[s0]);
                    commit(&tfull_bar[buf]);
                    it += 3;
                }
            }
            // done_bar fires once every MMA issued above has completed.
            asm volatile(
                "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                    smem_u32(&done_bar))
                : "memory");
            const long long t0 = clock64();
            while (!mbar_try_wait(&done_bar, 0) && clock64() - t0 < kWaitCycles) {
            }
        }
    } else {  // epilogue: TMEM sub-partition warp % 4, columns 0..127 or 128..255 of the tile
        const int sub = warp & 3, half = (warp - 2) >> 2;
        TileWalk walk;
        uint32_t chunk = 0;
        bool ok = true;
        for (long long t = blockIdx.x; t < args.total && ok; t += G) {
            int tm, tn;
            walk.locate(args, t, tm, tn);
            const int row = tm * kTM + sub * 32 + lane, n0 = tn * kTN + half * 128;
            float acc[128];
#pragma unroll
            for (int j = 0; j < 128; ++j) acc[j] = 0.f;
#pragma unroll 1
            for (int kt = 0; kt < ktiles; ++kt, ++chunk) {
                const int buf = (int)(chunk & 1);
                // warp-uniform outcome: tcgen05.ld needs the whole warp
                const bool ready =
                    mbar_wait_or_fail(&tfull_bar[buf], (chunk >> 1) & 1, args.err, fail);
                if (!__all_sync(0xffffffffu, ready)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
                const uint32_t src =
                    taddr + ((uint32_t)(sub * 32) << 16) + (uint32_t)(buf * kTN + half * 128);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    uint32_t v[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                          "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                        : "r"(src + (uint32_t)(q * 16)));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (q == 7) {  // accumulator read out: hand it back to the MMA warp
                        asm volatile("tcgen05.fence::before_thread_sync;");
                        __syncwarp();
                        if (lane == 0)
                            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                                             smem_u32(&tempty_bar[buf]))
                                         : "memory");
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[q * 16 + j] += __uint_as_float(v[j]);
                }
            }
            if (!ok) break;
            if (row < args.M) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    float cv[16];  // 16 loads in flight
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int col = n0 + q * 16 + j;
                        cv[j] = (col < args.N && (!args.lower || row >= col))
                                    ? __ldcg(args.C + (long long)col * args.ldc + row)
                                    : 0.f;
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int col = n0 + q * 16 + j;
                        if (col < args.N && (!args.lower || row >= col))
                            args.C[(long long)col * args.ldc + row] =
                                fmaf(acc[q * 16 + j], -kUnscale, cv[j]);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr),
                     "r"(kTmemCols));
}

// ---------------------------------------------------------------- conversion
struct Words {
    unsigned short w[3];
};
__device__ __forceinline__ Words split3(float x)
{
    Words o;
    x *= kSplitScale;
    const __nv_bfloat16 h0 = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(h0);
    const __nv_bfloat16 h1 = __float2bfloat16_rn(r1);
    const float r2 = r1 - __bfloat162float(h1);
    const __nv_bfloat16 h2 = __float2bfloat16_rn(r2);
    o.w[0] = __bfloat16_as_ushort(h0);
    o.w[1] = __bfloat16_as_ushort(h1);
    o.w[2] = __bfloat16_as_ushort(h2);
    return o;
}

// Eight values to 16 bytes of each word.
__device__ __forceinline__ void store_words(unsigned short* dst, size_t word_stride, const float* x)
{
    uint4 o[3];
    unsigned* p[3] = {&o[0].x, &o[1].x, &o[2].x};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const Words a = split3(x[2 * i]), b = split3(x[2 * i + 1]);
#pragma unroll
        for (int w = 0; w < 3; ++w) p[w][i] = (unsigned)a.w[w] | ((unsigned)b.w[w] << 16);
    }
#pragma unroll
    for (int w = 0; w < 3; ++w) *reinterpret_cast<uint4*>(dst + w * word_stride) = o[w];
}

__device__ __forceinline__ void record_max(unsigned m, unsigned* slot)
{
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m != 0u && m > *reinterpret_cast<volatile unsigned*>(slot))
        atomicMax(slot, m);
}

// src is rows x k column-major (rows contiguous): dst(r, k), K-major.  64 x 64
// tile per CTA through shared memory.
__global__ void __launch_bounds__(256) split_rows_kernel(int rows, int k, const float* __restrict__ src,
                                                         long long lds, unsigned short* dst,
                                                         int ldk, size_t word_stride,
                                                         unsigned* max_slot)
{
    __shared__ float T[64][65];  // T[k][r]
    const int r0 = blockIdx.x * 64, k0 = blockIdx.y * 64, tid = threadIdx.x;
    float v[16];
    unsigned m = 0;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int r = r0 + (tid & 63), kk = k0 + (tid >> 6) + 4 * u;
        v[u] = (r < rows && kk < k) ? src[(long long)kk * lds + r] : 0.f;
        m = max(m, __float_as_uint(v[u]) & 0x7fffffffu);
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) T[(tid >> 6) + 4 * u][tid & 63] = v[u];
    record_max(m, max_slot);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int q = tid + 256 * u, r = q >> 3, kk = (q & 7) * 8;
        if (r0 + r < rows && k0 + kk < ldk) {
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = T[kk + i][r];
            store_words(dst + (size_t)(r0 + r) * ldk + k0 + kk, word_stride, x);
        }
    }
}

// src is k x rows column-major (k contiguous): dst(r, k) = src[r * lds + k].
__global__ void __launch_bounds__(256) split_cols_kernel(int rows, int k, const float* __restrict__ src,
                                                         long long lds, unsigned short* dst,
                                                         int ldk, size_t word_stride,
                                                         unsigned* max_slot)
{
    const int groups = ldk / 8;
    const long long total = (long long)rows * groups;
    unsigned m = 0;
    for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < total;
         e += (long long)gridDim.x * 256) {
        const int r = (int)(e / groups), kk = (int)(e - (long long)r * groups) * 8;
        const float* p = src + (long long)r * lds + kk;
        float x[8];
        if (kk + 8 <= k && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(p));
            const float4 b = __ldg(reinterpret_cast<const float4*>(p + 4));
            x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
            x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = kk + i < k ? __ldg(p + i) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) m = max(m, __float_as_uint(x[i]) & 0x7fffffffu);
        store_words(dst + (size_t)r * ldk + kk, word_stride, x);
    }
    record_max(m, max_slot);
}

// 3-D map over the three K-major words: dims (k, rows, word).
bool word_map(CUtensorMap* map, const void* base, int ldk, int rows, int k, int box_rows)
{
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)rows, 3};
    cuuint64_t strides[2] = {(cuuint64_t)ldk * 2, (cuuint64_t)ldk * 2 * (cuuint64_t)rows};
    cuuint32_t box[3] = {(cuuint32_t)kTK, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box,
              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

hdbf_status split_operand(hdbf_context* ctx, bool k_contiguous, int rows, int k, const float* src,
                          long long lds, unsigned short* dst, int ldk, unsigned* slot)
{
    const size_t ws = (size_t)rows * ldk;
    ProfScope prof(ctx, kClsConvert, 0.0, 10.0 * rows * k);
    if (k_contiguous) {
        const long long total = (long long)rows * (ldk / 8);
        const int g = (int)std::min<long long>((total + 255) / 256, 8LL * ctx->sm_count);
        split_cols_kernel<<<g, 256, 0, ctx->stream>>>(rows, k, src, lds, dst, ldk, ws, slot);
    } else {
        const dim3 g((rows + 63) / 64, (k + 63) / 64);
        split_rows_kernel<<<g, 256, 0, ctx->stream>>>(rows, k, src, lds, dst, ldk, ws, slot);
    }
    ctx->launches++;
    return last_cuda(ctx);
}

}  // namespace

void configure_tc_sgemm(hdbf_context*)
{
    cudaFuncSetAttribute(tc_sgemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kSmemBytes);
    cudaGetLastError();
}

// Longest K chunk of an update of this shape: its operands' words are at most those of
// an update of order max(M, N) + K, the order of the factorization it belongs to
// (words_bytes, runtime.cu), so the chunk follows from the shape alone.
static long long shape_chunk(int M, int N, int K)
{
    const long long order = (long long)std::max(M, N) + K;
    return std::max<long long>(
        64, 2 * order * std::min<long long>(order, 2048) / ((long long)M + N) / 64 * 64);
}

// K chunk of the split path for an update of this shape: 0 = not taken.  The
// line is where both take the same time: 2 M N K = 2e9 at tile-sized N, where
// the conversions, three more launches and a partly filled wave cost what the
// faster products save (2048 x 512 x 512: 51 us against 45; 4096 x 512 x 512: 55
// against 76; 16384 x 512 x 512: 115 against 204; 16384 x 4096 x 4096: 2.85 ms
// against 10.5, 193 TFLOP/s).  Below 128 columns half of a tile or more is idle.
// Accuracy draws a second line, in every mode: where few tiles make an FP32
// kernel cut K into five or more partial sums, its rounding errors average out
// and, on operands of one sign, come out below the truncation here (777 x 640 x
// 2100 over [0,1): 9.9e-8 against 1.16e-7), so it keeps those shapes.
int tc_sgemm_chunk(const hdbf_context* ctx, int M, int N, int K, bool tri)
{
    if (!ctx->ws || ctx->run_if || ctx->tc_sgemm == 0) return 0;
    if (ctx->tc_sgemm != 2 &&
        (M < 256 || N < 128 || K < 128 || (double)M * N * K < 1.0e9))
        return 0;
    int kc_fp32 = 0;
    if (split_count(ctx, M, N, K, tri, &kc_fp32) > 4 || gemm_small_split(ctx, M, N, K) > 4) return 0;
    return (int)std::min<long long>((K + 63) / 64 * 64, shape_chunk(M, N, K));
}

int tc_sgemm_plan(hdbf_context* ctx, int M, int N, int K, bool tri)
{
    const int kc = tc_sgemm_chunk(ctx, M, N, K, tri);
    return kc > 0 && words_room(ctx, 256 + 6 * ((size_t)M + N) * kc) ? kc : 0;
}

void reserve_words(hdbf_context* ctx, int M, int N, int K)
{
    if (ctx->tc_sgemm == 0 || (ctx->tc_sgemm == 1 && (double)M * N * K < 1.0e9)) return;
    const long long kc = std::min<long long>((K + 63) / 64 * 64, shape_chunk(M, N, K));
    words_room(ctx, 256 + 6 * ((size_t)M + N) * kc);
}

hdbf_status tc_sgemm_chunk_run(hdbf_context* ctx, bool a_kc, bool b_kc, bool lower, int M, int N,
                               int K, const float* A, long long lda, const float* B, long long ldb,
                               float* C, long long ldc, unsigned** range)
{
    char* base = static_cast<char*>(ws_words(ctx));
    unsigned* slots = reinterpret_cast<unsigned*>(base);
    unsigned short* wa = reinterpret_cast<unsigned short*>(base + 256);
    const int ldk = (K + 7) / 8 * 8;
    // C -= A A^T: B is the head of A
    const bool same = !a_kc && !b_kc && A == B && lda == ldb && N <= M;
    unsigned short* wb = same ? wa : wa + 3 * (size_t)M * ldk;
    const int b_rows = same ? M : N;
    CUtensorMap ma, mb;  // before the first launch: without them nothing has happened
    if (!word_map(&ma, wa, ldk, M, K, kTM) || !word_map(&mb, wb, ldk, b_rows, K, kTN))
        return HDBF_STATUS_NOT_SUPPORTED;
    *range = slots;
    if (cudaMemsetAsync(slots, 0, 2 * sizeof(unsigned), ctx->stream) != cudaSuccess)
        return last_cuda(ctx);
    HDBF_TRY(split_operand(ctx, a_kc, M, K, A, lda, wa, ldk, slots));
    if (!same) HDBF_TRY(split_operand(ctx, b_kc, N, K, B, ldb, wb, ldk, slots + 1));
    X6Args a;
    a.M = M;
    a.N = N;
    a.K = K;
    a.b_row0 = 0;
    a.C = C;
    a.ldc = ldc;
    a.tiles_m = (M + kTM - 1) / kTM;
    a.tiles_n = (N + kTN - 1) / kTN;
    a.lower = lower ? 1 : 0;
    a.range = slots;
    a.err = ctx->dev_small + kSmallErr;
    a.total = 0;
    for (int tn = 0; tn < a.tiles_n; ++tn)
        a.total += lower ? std::max(0, a.tiles_m - 2 * tn) : a.tiles_m;
    double entries = (double)M * N;
    if (lower) {
        const double d = (double)std::min(M, N);
        entries = d * (double)M - d * (d - 1.0) / 2.0;
    }
    ProfScope prof(ctx, kClsTcGemm, 2.0 * entries * K, 6.0 * ((double)M + N) * K + 8.0 * entries, M,
                   N, K);
    const unsigned g = (unsigned)std::min<long long>(a.total, ctx->sm_count);
    tc_sgemm_kernel<<<g, kThr, kSmemBytes, ctx->stream>>>(ma, mb, a);
    ctx->launches++;
    return last_cuda(ctx);
}

}  // namespace hdbf
