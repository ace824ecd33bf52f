// Two FP32 values that go through one packed FMA (fma.rn.f32x2, each half rounded
// as a scalar FMA), and the same interface over two FP64 values.
#pragma once

#include <cuda_runtime.h>

namespace hdbf {

template <class T>
struct Two;

template <>
struct Two<float> {
    unsigned long long v;
    static __device__ __forceinline__ Two make(float x, float y)
    {
        Two t;
        asm("mov.b64 %0, {%1, %2};" : "=l"(t.v) : "f"(x), "f"(y));
        return t;
    }
    static __device__ __forceinline__ Two zero() { return Two{0ull}; }
    __device__ __forceinline__ void fma(Two a, Two b)
    {
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(a.v), "l"(b.v));
    }
    __device__ __forceinline__ void get(float& x, float& y) const
    {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    }
};

template <>
struct Two<double> {
    double x, y;
    static __device__ __forceinline__ Two make(double a, double b) { return Two{a, b}; }
    static __device__ __forceinline__ Two zero() { return Two{0.0, 0.0}; }
    __device__ __forceinline__ void fma(Two a, Two b)
    {
        x = ::fma(a.x, b.x, x);
        y = ::fma(a.y, b.y, y);
    }
    __device__ __forceinline__ void get(double& a, double& b) const
    {
        a = x;
        b = y;
    }
};

// Four consecutive values (16-byte aligned) as two pairs, and back.
__device__ __forceinline__ void load_pairs(const float* p, Two<float>& a, Two<float>& b)
{
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    a.v = v.x;
    b.v = v.y;
}
__device__ __forceinline__ void load_pairs(const double* p, Two<double>& a, Two<double>& b)
{
    const double2 u = *reinterpret_cast<const double2*>(p);
    const double2 v = *reinterpret_cast<const double2*>(p + 2);
    a = Two<double>{u.x, u.y};
    b = Two<double>{v.x, v.y};
}
__device__ __forceinline__ void store_pairs(float* p, Two<float> a, Two<float> b)
{
    ulonglong2 v;
    v.x = a.v;
    v.y = b.v;
    *reinterpret_cast<ulonglong2*>(p) = v;
}
__device__ __forceinline__ void store_pairs(double* p, Two<double> a, Two<double> b)
{
    *reinterpret_cast<double2*>(p) = make_double2(a.x, a.y);
    *reinterpret_cast<double2*>(p + 2) = make_double2(b.x, b.y);
}

}  // namespace hdbf
