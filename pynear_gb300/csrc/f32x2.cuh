// f32x2.cuh — packed FP32: two IEEE round-to-nearest results per instruction.
//
// Measured on GB300: add and fma on pairs give the FP32 pipe's full 128
// results per SM and clock from half the issue slots of the scalar forms
// (scalar FFMA alone reaches 117), so loops bound by issue gain, and each
// result is bit for bit the scalar _rn one.  There is no packed product here:
// followed by a packed sum it is fused into one rounding.
#pragma once

#include <stdint.h>

namespace gn {

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 dup2(float v) { return pack2(v, v); }
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

}  // namespace gn
