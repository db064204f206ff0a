// Two values per thread side by side.  In FP32 the arithmetic on a pair is the packed instructions of
// sm_100 and later (each half rounded as the scalar instruction rounds it, in one issue slot); in FP64
// it is two scalar operations.
#pragma once
#include <cuda_runtime.h>

namespace tcsem {

template <typename T> struct Pair {
    T a, b;
};
template <typename T> __device__ __forceinline__ Pair<T> pair(T a, T b) { return {a, b}; }
template <typename T> __device__ __forceinline__ Pair<T> dup(T a) { return {a, a}; }

__device__ __forceinline__ float2 f2(Pair<float> x) { return make_float2(x.a, x.b); }
__device__ __forceinline__ Pair<float> pf(float2 x) { return {x.x, x.y}; }
__device__ __forceinline__ Pair<float> operator-(Pair<float> x) { return {-x.a, -x.b}; }
__device__ __forceinline__ Pair<float> operator+(Pair<float> x, Pair<float> y) { return pf(__fadd2_rn(f2(x), f2(y))); }
__device__ __forceinline__ Pair<float> operator-(Pair<float> x, Pair<float> y) { return pf(__fadd2_rn(f2(x), f2(-y))); }
__device__ __forceinline__ Pair<float> operator*(Pair<float> x, Pair<float> y) { return pf(__fmul2_rn(f2(x), f2(y))); }
// x y + z
__device__ __forceinline__ Pair<float> fma(Pair<float> x, Pair<float> y, Pair<float> z) {
    return pf(__ffma2_rn(f2(x), f2(y), f2(z)));
}
__device__ __forceinline__ Pair<double> operator-(Pair<double> x) { return {-x.a, -x.b}; }
__device__ __forceinline__ Pair<double> operator+(Pair<double> x, Pair<double> y) { return {x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ Pair<double> operator-(Pair<double> x, Pair<double> y) { return {x.a - y.a, x.b - y.b}; }
__device__ __forceinline__ Pair<double> operator*(Pair<double> x, Pair<double> y) { return {x.a * y.a, x.b * y.b}; }
__device__ __forceinline__ Pair<double> fma(Pair<double> x, Pair<double> y, Pair<double> z) {
    return {::fma(x.a, y.a, z.a), ::fma(x.b, y.b, z.b)};
}

}  // namespace tcsem
