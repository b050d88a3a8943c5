// Packed fp32 arithmetic of the gradient kernels and the conversion of their 16-bit slab entries.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace lutgemm {

// two fp32 values in one 64-bit register (the operand form of the packed fp32 instructions)
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 t;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(t.x), "=f"(t.y) : "l"(v));
    return t;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// the two signed table entries of a slab word: 0x4B000000 | u is the float 2^23 + u, u = entry + 2^15
__device__ __forceinline__ f32x2 entries2(uint32_t word, f32x2 bias) {
    const float lo = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7610));
    const float hi = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7632));
    return add2(pack2(lo, hi), bias);
}

}  // namespace lutgemm
