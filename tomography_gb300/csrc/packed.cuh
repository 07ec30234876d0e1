// Pairs of values for the packed FP32 instructions (f32x2) of sm_103a.
#pragma once
#include <cuda_runtime.h>

namespace tomo {

// Two values of one operation: a packed f32x2 instruction in FP32 (the same
// rounding per half as the scalar form), two scalar ones in FP64.
template <typename Real>
struct alignas(2 * sizeof(Real)) Two {
    Real x, y;
};
__device__ __forceinline__ unsigned long long two_bits(Two<float> a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ Two<float> two_of(unsigned long long v) {
    Two<float> r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ Two<float> add2(Two<float> a, Two<float> b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(two_bits(a)), "l"(two_bits(b)));
    return two_of(r);
}
__device__ __forceinline__ Two<float> sub2(Two<float> a, Two<float> b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(two_bits(a)), "l"(two_bits(b)));
    return two_of(r);
}
__device__ __forceinline__ Two<float> fma2(Two<float> a, Two<float> b, Two<float> c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(two_bits(a)), "l"(two_bits(b)), "l"(two_bits(c)));
    return two_of(r);
}
// A packed product must not feed a packed sum or difference: the compiler may
// fuse the two.  Such products are written as scalar ones (times2).
__device__ __forceinline__ Two<float> mul2(Two<float> a, Two<float> b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(two_bits(a)), "l"(two_bits(b)));
    return two_of(r);
}
__device__ __forceinline__ Two<double> add2(Two<double> a, Two<double> b) {
    return {__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)};
}
__device__ __forceinline__ Two<double> sub2(Two<double> a, Two<double> b) {
    return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)};
}
__device__ __forceinline__ Two<double> mul2(Two<double> a, Two<double> b) {
    return {__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)};
}
__device__ __forceinline__ Two<double> fma2(Two<double> a, Two<double> b, Two<double> c) {
    return {__fma_rn(a.x, b.x, c.x), __fma_rn(a.y, b.y, c.y)};
}
template <typename Real>
__device__ __forceinline__ Two<Real> times2(Two<Real> a, Two<Real> b) {
    if constexpr (sizeof(Real) == 4) return {__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)};
    else return {__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)};
}
template <typename Real>
__device__ __forceinline__ Two<Real> dup2(Real v) {
    return {v, v};
}

}  // namespace tomo
