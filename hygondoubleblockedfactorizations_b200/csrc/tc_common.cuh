// tcgen05 / TMA building blocks shared by the tensor-core GEMMs.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <mutex>

#include "internal.h"

namespace hdbf {
namespace {

constexpr long long kWaitCycles = 4000000000LL;  // ~2 s at 2 GHz

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait on an mbarrier phase; false (and *err set) on expiry.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err)
{
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > kWaitCycles) {
            atomicCAS(err, 0, kErrTimeout);
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int x, int y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (SBO), LBO unused for swizzled K-major, version 1.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor, kind::f16: FP32 accumulate, A/B = BF16 (fmt 1) or FP16
// (fmt 0), both K-major, M = 128.
__host__ __device__ constexpr uint32_t make_idesc_n(int fmt, int n)
{
    return (1u << 4) | ((uint32_t)fmt << 7) | ((uint32_t)fmt << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(128 >> 4) << 24);
}

// Bounded wait that also gives up once another role of the CTA has failed.
__device__ __forceinline__ bool mbar_wait_or_fail(uint64_t* bar, uint32_t parity, int* err,
                                                  volatile int* fail)
{
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (*fail) return false;
        if (clock64() - t0 > kWaitCycles) {
            atomicCAS(err, 0, kErrTimeout);
            *fail = 1;
            return false;
        }
    }
    return true;
}

// Linear tile index -> (tm, tn), band by band (tn outer); the cursor only
// moves forward, as every role visits its tiles in increasing order.
struct TileWalk {
    int tn = 0;
    long long base = 0;
    template <class Args>
    __device__ __forceinline__ void locate(const Args& a, long long t, int& tm, int& tnn)
    {
        for (;;) {
            const long long cnt = a.lower ? (long long)max(0, a.tiles_m - 2 * tn) : a.tiles_m;
            if (t < base + cnt || tn >= a.tiles_n - 1) {
                tm = (a.lower ? 2 * tn : 0) + (int)(t - base);
                tnn = tn;
                return;
            }
            base += cnt;
            ++tn;
        }
    }
};

PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        cudaGetLastError();
    });
    return fn;
}

}  // namespace
}  // namespace hdbf
