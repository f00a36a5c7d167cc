// Two FP32 values in one 64-bit register pair (the f32x2 instructions of sm_100a): each
// half is rounded as the scalar operation rounds it, so packing never changes a result.
// Measured on B200: one packed operation takes one issue slot and two cycles of the FP32
// pipe, so it halves the issue slots of an issue-bound kernel and leaves the pipe's own
// limit (32 lanes per cycle and scheduler) where it was.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace ctsim {

using f32x2 = float2;

__device__ __forceinline__ f32x2 pack2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ void unpack2(f32x2 x, float &a, float &b) {
    a = x.x;
    b = x.y;
}

// The same operations on one value (float) and on two (f32x2), so that a kernel body can
// be written once for both widths.  All of them are round-to-nearest and never contracted,
// except padd_rd (toward -inf) -- but see padd_product.
__device__ __forceinline__ float padd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float psub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float pmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float pfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float padd_rd(float a, float b) { return __fadd_rd(a, b); }

__device__ __forceinline__ f32x2 padd(f32x2 a, f32x2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ f32x2 psub(f32x2 a, f32x2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ f32x2 pmul(f32x2 a, f32x2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f32x2 padd_rd(f32x2 a, f32x2 b) { return __fadd2_rd(a, b); }
__device__ __forceinline__ f32x2 pfma(f32x2 a, f32x2 b, f32x2 c) { return __ffma2_rn(a, b, c); }
// a * b + c rounded toward -inf
__device__ __forceinline__ f32x2 pfma_rd(f32x2 a, f32x2 b, f32x2 c) { return __ffma2_rd(a, b, c); }

// x + y where x or y is a product that the reference rounds before it adds.  ptxas
// contracts a packed product and a packed sum into one fma although both are marked .rn
// (observed with nvcc 12.9: different bits), so the sum is written as fma(x, one, y) with
// `one` = 1.0f passed to the kernel at run time.
__device__ __forceinline__ float padd_product(float x, float, float y) { return __fadd_rn(x, y); }
__device__ __forceinline__ f32x2 padd_product(f32x2 x, f32x2 one, f32x2 y) { return pfma(x, one, y); }

// Broadcast of one value, halves, and a map over the halves.
template <class V>
struct Packed;
template <>
struct Packed<float> {
    static constexpr int kWidth = 1;
    static __device__ __forceinline__ float all(float a) { return a; }
    static __device__ __forceinline__ float get(float x, int) { return x; }
    template <class F>
    static __device__ __forceinline__ float make(F f) {
        return f(0);
    }
};
template <>
struct Packed<f32x2> {
    static constexpr int kWidth = 2;
    static __device__ __forceinline__ f32x2 all(float a) { return pack2(a, a); }
    static __device__ __forceinline__ float get(f32x2 x, int i) { return i ? x.y : x.x; }
    template <class F>
    static __device__ __forceinline__ f32x2 make(F f) {
        const float a = f(0), b = f(1);
        return pack2(a, b);
    }
};

}  // namespace ctsim
