// Sources and outputs of the CDF 9/7 lifting levels.
//
// A level reads a box of samples (forward) or of split-band coefficients
// (inverse) and hands every finished sample to an emitter functor. Lifted
// lines are processed in windows of W outputs that read W+8 samples, like the
// reference's halo windows (cpu/src/transform.cpp:149-179,
// include/transformers/halo3d.cuh:66-169):
//  * forward windows are independent of their origin (any even one gives the
//    same bits), so W is chosen for speed;
//  * inverse Y and Z windows fold their endpoint normalisations, so their
//    results depend on the window: W_Y = 8 and W_Z = 16 (f32) / 8 (f64)
//    with origins at multiples of W, the reference's canonical windows;
//  * inverse X does not fold and is window independent.
#pragma once
#include "common.cuh"

namespace wb {

enum Axes : int { AX = 1, AY = 2, AZ = 4 };

// Forward source: a compact or strided box, reflected at its edges. With
// `status` set, every staged sample is also checked for finiteness (the
// finest level stages every input sample at least once). Samples are staged
// row by row: `row(y, z)` resolves a row once, `get(row, x)` reads one sample.
template <class T> struct FwdSrc {
    const T* p;
    size_t sy, sz; // element strides
    uint32_t* status = nullptr;
    struct Row {
        const T* p;
    };
    __device__ __forceinline__ Row row(uint32_t y, uint32_t z) const { return {p + size_t(z) * sz + size_t(y) * sy}; }
    __device__ __forceinline__ T get(const Row& r, uint32_t x) const { return r.p[x]; }
};

// Inverse source: coefficient box whose low corner (lo dims) may come from a
// separately reconstructed compact array, the rest from `base`.
template <class T> struct InvSrc {
    const T* base;
    size_t sy, sz;
    const T* low; // nullable
    Dims lo;
};

// Forward output: high bands to `dst` at split positions; the all-even low
// corner to `low` (compact, dims lo) when given, else to dst as well.
template <class T> struct FwdOut {
    T* dst;
    size_t sy, sz;
    T* low;
    Dims lo;
};

// Inverse output into a compact or strided array.
template <class T> struct StoreOut {
    static constexpr bool kPrefetch = false;
    T* dst;
    size_t sy, sz;
    __device__ __forceinline__ void operator()(uint32_t x, uint32_t y, uint32_t z, T v) const {
        dst[size_t(z) * sz + size_t(y) * sy + x] = v;
    }
};

// Emitters whose samples sit at dst + z * sz + y * sy + x take pointers
// computed once per row or column; the others take each sample through
// their own operator().
template <class Out> struct RowStore {
    static constexpr bool value = false;
};
template <class T> struct RowStore<StoreOut<T>> {
    static constexpr bool value = true;
};

// Outputs of a canonical inverse Z window.
template <class T> constexpr int inverse_zwin() { return sizeof(T) == 4 ? 16 : 8; }

} // namespace wb
