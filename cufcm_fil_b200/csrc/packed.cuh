// packed.cuh -- two FP32 values in one register pair.
//
// The packed instructions (add, mul, fma .f32x2, sm_100) do the arithmetic of
// two scalar ones, rounded the same, in one issue slot and with one read of
// each operand pair.  The FP32 pipe is no faster for them (70.6 TFLOP/s either
// way on independent fma chains), but a kernel that is held up by issue or by
// register reads gains: the pair product of rpy_pairs.cuh 3.59 -> 2.81 ms per
// 10^9 pairs.  Code for both is written once, over a real type T = float, F1 or F2.
#pragma once

#include <cuda_runtime.h>

namespace cufil {

struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ F2 vadd(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vsub(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vmul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }
__device__ __forceinline__ float vmul(float a, float b) { return a * b; }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
// One value, rounded after every operation as each half of F2 is (a plain float may be contracted).  Products that are
// added are written as vfma: the compiler contracts packed ones that are not.
struct F1 {
    float v;
};
__device__ __forceinline__ F1 vadd(F1 a, F1 b) { return {__fadd_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 vsub(F1 a, F1 b) { return {__fsub_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 vmul(F1 a, F1 b) { return {__fmul_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 vfma(F1 a, F1 b, F1 c) { return {__fmaf_rn(a.v, b.v, c.v)}; }
template <class T>
__device__ __forceinline__ T splat(float c);
template <>
__device__ __forceinline__ F1 splat<F1>(float c) {
    return {c};
}
template <>
__device__ __forceinline__ float splat<float>(float c) {
    return c;
}
template <>
__device__ __forceinline__ F2 splat<F2>(float c) {
    return pack2(c, c);
}
__device__ __forceinline__ float rsqrt_approx(float a) { return rsqrtf(a); }
__device__ __forceinline__ F1 rsqrt_approx(F1 a) { return {rsqrtf(a.v)}; }
__device__ __forceinline__ F2 rsqrt_approx(F2 a) {
    const float2 v = unpack2(a);
    return pack2(rsqrtf(v.x), rsqrtf(v.y));
}

}  // namespace cufil
