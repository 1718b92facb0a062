// Sizes and slots of an expansion of degree p: (p+1)^2 real coefficients, the complex one of
// degree n and order m in slots n^2 + n + m (real part) and n^2 + n - m (imaginary part).
#pragma once

#include <cuda_runtime.h>

namespace fmmb {

__host__ __device__ constexpr int nc_of(int p) { return (p + 1) * (p + 1); }
// row stride of the translation products (Y, Yo): (p+1)^2 rounded up to whole 16-byte
// groups of f32, as the expansions' rows, so that the rows of a tile are one contiguous
// run with no padding to write and read back (measured: 32-slot rows cost 12 % more of
// the product traffic at p = 8)
__host__ __device__ constexpr int ys_of(int p) { return ((nc_of(p) + 3) / 4) * 4; }
// row stride of one expansion (one box, one vector) in the multipole and local arrays:
// (p+1)^2 rounded up to whole 16-byte groups in f32, so that every row starts on a
// 16-byte boundary (the tensor-memory-access gathers of the tensor-core M2L need it)
__host__ __device__ constexpr int ms_of(int p) { return ((nc_of(p) + 3) / 4) * 4; }
__host__ __device__ constexpr int slot(int n, int m) { return n * n + n + m; }

template <typename T>
struct Cx {
    T re, im;
};

// coefficient of degree n, stored order m >= 0, from real storage (zero beyond degree)
template <typename T>
__device__ __forceinline__ Cx<T> coef_at(const T* c, int n, int m) {
    Cx<T> z;
    if (m < 0 || m > n || n < 0) {
        z.re = T(0);
        z.im = T(0);
        return z;
    }
    z.re = c[slot(n, m)];
    z.im = m ? c[slot(n, -m)] : T(0);
    return z;
}

}  // namespace fmmb
