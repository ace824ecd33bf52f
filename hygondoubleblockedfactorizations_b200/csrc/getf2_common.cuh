// Pivot search and scalar helpers shared by the LU panel kernels.
#pragma once

#include <cfloat>
#include <climits>

namespace hdbf {

template <class T>
struct Bits;
template <>
struct Bits<float> {
    using Mag = unsigned;
    static __device__ __forceinline__ Mag of(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float val(Mag m) { return __uint_as_float(m); }
    static __device__ __forceinline__ float rcp(float v) { return __frcp_rn(v); }
};
template <>
struct Bits<double> {
    using Mag = unsigned long long;
    static __device__ __forceinline__ Mag of(double v)
    {
        return (unsigned long long)__double_as_longlong(v);
    }
    static __device__ __forceinline__ double val(Mag m) { return __longlong_as_double((long long)m); }
    static __device__ __forceinline__ double rcp(double v) { return 1.0 / v; }
};
template <class T>
using Mag = typename Bits<T>::Mag;

// |v| as bits that order like the values; a NaN loses to everything else.
template <class T>
__device__ __forceinline__ Mag<T> mag_bits(T v)
{
    return v == v ? Bits<T>::of(v < T(0) ? -v : v) & (~(Mag<T>)0 >> 1) : (Mag<T>)0;
}
// Largest magnitude over the warp and the lowest row that has it (INT_MAX: no
// candidate).
__device__ __forceinline__ void warp_argmax(unsigned vb, int row, unsigned& mv, int& mrow)
{
    mv = __reduce_max_sync(0xffffffffu, vb);
    mrow = __reduce_min_sync(0xffffffffu, vb == mv ? row : INT_MAX);
}
__device__ __forceinline__ void warp_argmax(unsigned long long vb, int row, unsigned long long& mv,
                                            int& mrow)
{
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(vb >> 32));
    const unsigned lo = __reduce_max_sync(
        0xffffffffu, (unsigned)(vb >> 32) == hi ? (unsigned)(vb & 0xffffffffu) : 0u);
    mv = ((unsigned long long)hi << 32) | lo;
    mrow = __reduce_min_sync(0xffffffffu, vb == mv ? row : INT_MAX);
}

__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float min_normal(float) { return FLT_MIN; }
__device__ __forceinline__ double min_normal(double) { return DBL_MIN; }
__device__ __forceinline__ float abs_t(float v) { return fabsf(v); }
__device__ __forceinline__ double abs_t(double v) { return fabs(v); }

}  // namespace hdbf
