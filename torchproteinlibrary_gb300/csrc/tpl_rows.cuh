// Rows of atoms (xyz interleaved) read and written in 16-byte vectors whatever the
// row's alignment; shared by the CoordsTransform and Coords2RMSD kernels.
//
// A group of N = 16 / sizeof(T) consecutive atoms is three whole vectors, and starts
// on a 16-byte boundary when its first atom i has W + 3 i = 0 (mod N), W being the
// row's first element counted from such a boundary.  3 is its own inverse modulo 4 and
// modulo 2, so that is i = W (mod N): after row_head() atoms every group is aligned.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace tpl {

template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    using type = float4;
    static constexpr int n = 4;
};
template <>
struct Vec16<double> {
    using type = double2;
    static constexpr int n = 2;
};

// Atoms before the first aligned group of the row p (0 .. N - 1).
template <typename T>
__device__ __forceinline__ int row_head(const T *p) {
    return (int)((reinterpret_cast<uintptr_t>(p) / sizeof(T)) & (Vec16<T>::n - 1));
}

// The 3 N values of an aligned group at p.
template <typename T>
__device__ __forceinline__ void load_group(const T *p, T (&v)[3 * Vec16<T>::n]) {
    using V = typename Vec16<T>::type;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const V x = reinterpret_cast<const V *>(p)[i];
        memcpy(v + i * Vec16<T>::n, &x, sizeof(V));
    }
}
template <typename T>
__device__ __forceinline__ void store_group(T *p, const T (&v)[3 * Vec16<T>::n]) {
    using V = typename Vec16<T>::type;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        V x;
        memcpy(&x, v + i * Vec16<T>::n, sizeof(V));
        reinterpret_cast<V *>(p)[i] = x;
    }
}

}  // namespace tpl
