// vel.cuh -- the velocities that one lane of a gather holds.
#pragma once

#include <cuda_runtime.h>

namespace alebgk {

// The velocities of one lane: two of FP32 (packed FMAs), or one.
template <typename T, int VPL> struct Vel;
template <> struct Vel<float, 2>
{
    typedef float2 V;
    static __device__ __forceinline__ V zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return __ffma2_rn(a, b, c); }
    static __device__ __forceinline__ V mul(V a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
};
template <typename T> struct Vel<T, 1>
{
    typedef T V;
    static __device__ __forceinline__ V zero() { return T(0); }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return ::fma(a, b, c); }
    static __device__ __forceinline__ V mul(V a, T s) { return a * s; }
};

}  // namespace alebgk
