// Device-side helpers shared by the kernels of libfftgal_gb300.so.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fg {

template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };
template <typename T> using vec2_t = typename Vec2<T>::type;

template <typename T2>
__device__ __forceinline__ T2 mk2(decltype(T2::x) a, decltype(T2::x) b) {
    T2 r;
    r.x = a;
    r.y = b;
    return r;
}

template <typename T2>
__device__ __forceinline__ T2 cadd(T2 a, T2 b) { return mk2<T2>(a.x + b.x, a.y + b.y); }
template <typename T2>
__device__ __forceinline__ T2 csub(T2 a, T2 b) { return mk2<T2>(a.x - b.x, a.y - b.y); }
template <typename T2>
__device__ __forceinline__ T2 cmul(T2 a, T2 b) {
    return mk2<T2>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <typename T2>
__device__ __forceinline__ T2 cconj(T2 a) { return mk2<T2>(a.x, -a.y); }
// multiply by (sign * i)
template <typename T2>
__device__ __forceinline__ T2 cmul_si(T2 a, int sign) {
    return sign < 0 ? mk2<T2>(a.y, -a.x) : mk2<T2>(-a.y, a.x);
}

__host__ __device__ __forceinline__ long ceil_div(long a, long b) { return (a + b - 1) / b; }

// Column passes of the FFT in tiles of C = 2^logC columns, element n at g + n es.
// Tiles per batch: where all rows of a column share their alignment (es a multiple of
// C: the i pass) a tile starts on a C-value boundary of memory, `off` columns early.  A
// row of 16 columns is then one 128-byte line instead of five sectors of two lines
// (i pass at Ng = 512: 583 us -> 364 with the loads below, j, which has no common
// alignment, 571 -> 420; both grids), and the grids' Ng/2 + 1 = 1 mod 16 columns take
// no more tiles than before.
__host__ __device__ __forceinline__ int cols_tiles(int ncols, long es, int logC) {
    const int C = 1 << logC;
    return (ncols + C - 1 + ((es & (C - 1)) == 0 ? C - 1 : 0)) >> logC;
}
// columns of a tile that lie before the batch at g
__device__ __forceinline__ int cols_offset(const void *g, long es, int logC) {
    const int C = 1 << logC;
    return (es & (C - 1)) == 0 ? (int)((uintptr_t)g / 8) & (C - 1) : 0;
}

}  // namespace fg
