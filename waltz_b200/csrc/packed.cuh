// Pairs of floats and the packed operations on them: two independent correctly
// rounded operations per instruction (no flush to zero), so the bits are those
// of the scalar operations; see f2_mul for its one exception.
#pragma once
#include "common.cuh"

namespace wb {

// Two floats in one 64-bit register pair.
using f2 = unsigned long long;
__device__ __forceinline__ f2 f2_pack(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// The assembler contracts a packed product whose only use is a packed sum into
// one rounding, --fmad=false notwithstanding (seen on quantised codes; the same
// product as a multiply-add of -0 is contracted too). A product that feeds only
// a sum therefore has to be formed with the scalar __fmul_rn; in the lifting
// every scaled sample is also the addend of a multiply-add and stays a product.
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

} // namespace wb
