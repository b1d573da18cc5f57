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
// Another assembler may contract otherwise: the parity tests against the oracle
// hold every form that uses this file to the exact bits.
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// lift_inverse<float, P, true> (common.cuh) on two lines at once.
template <int P> __device__ __forceinline__ void lift_inverse2(f2 (&e)[P], f2 (&o)[P]) {
    const f2 ca = f2_pack(-K97<float>::a, -K97<float>::a), cb = f2_pack(-K97<float>::b, -K97<float>::b),
             cg = f2_pack(-K97<float>::g, -K97<float>::g), cd = f2_pack(-K97<float>::d, -K97<float>::d),
             ck = f2_pack(-K97<float>::k, -K97<float>::k), ci = f2_pack(K97<float>::ik, K97<float>::ik);
    const f2 raw_first = o[0], raw_last = o[P - 1];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        e[j] = f2_mul(e[j], ci);
        o[j] = f2_mul(o[j], ck);
    }
#pragma unroll
    for (int j = 1; j < P; ++j) {
        f2 s;
        if (j == 1) s = f2_fma(raw_first, ck, o[1]);
        else if (j == P - 1) s = f2_fma(raw_last, ck, o[P - 2]);
        else s = f2_add(o[j - 1], o[j]);
        e[j] = f2_fma(cd, s, e[j]);
    }
#pragma unroll
    for (int j = 1; j < P - 1; ++j) o[j] = f2_fma(cg, f2_add(e[j], e[j + 1]), o[j]);
#pragma unroll
    for (int j = 2; j < P - 1; ++j) e[j] = f2_fma(cb, f2_add(o[j - 1], o[j]), e[j]);
#pragma unroll
    for (int j = 2; j < P - 2; ++j) o[j] = f2_fma(ca, f2_add(e[j], e[j + 1]), o[j]);
}

} // namespace wb
