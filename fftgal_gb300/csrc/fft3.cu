// Mixed-radix FFT passes of FP32 grids (sm_103a): lengths N = N1 N2 with N1, N2
// <= 32 and prime factors up to 13, e.g. 96, 225, 384, 500 -- the sizes that the
// power-of-two passes of fft2.cu do not take.
//
// As in fft2.cu a transform is two in-register FFTs around one trip through
// shared memory,
//   X[k1 + N1 k2] = sum_n2 W_N2^{n2 k2} W_N^{n2 k1} sum_n1 x[N2 n1 + n2] W_N1^{n1 k1},
// with the lengths chosen at run time: step functions are instantiated for every
// length up to 32 and selected by a switch.  A backward transform is the forward
// one between two conjugations.
//   strided axes: 16 adjacent columns per CTA, so every row access is a 128-byte run;
//   k axis: two real rows are one complex row a + i b, for odd and even lengths
//   alike: A[k] = (Z[k] + conj Z[N-k]) / 2, B[k] = (Z[k] - conj Z[N-k]) / 2i.
// The general kernels of fft.cu (radix passes through shared memory with
// run-time strides) remain for other lengths and FP64 grids.
// Measured (GB300, both interlacing grids, us): Ng = 384 k 1402 -> 266, j + i 3655 -> 404
// and Ng = 225 1083 -> 57, 1493 -> 94 (in the general kernels: run-time divisions per
// element, one memory round trip per radix and O(R^2) odd butterflies from constant
// memory).  128 registers for the longest lengths hold the kernels to two CTAs of 256
// threads per SM, whose load and store phases bound them (Ng = 384: 3.4 and 4.5 TB/s
// of the 6.8 a copy does); 16 columns per CTA, on a 128-byte boundary where the rows
// share one (cols_tiles), keep global rows at 128 bytes and shared accesses free of
// conflicts without padding.
#include "internal.h"
#include "common.cuh"
#include "regfft.cuh"

#include <math.h>

namespace fg {

constexpr int kF3Threads = 256;
constexpr int kF3LogCols = 4, kF3Cols = 1 << kF3LogCols;  // columns per CTA

#define FG_F3_LENGTHS(X)                                                                                       \
    X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(18) X(20) X(21) \
        X(22) X(24) X(25) X(26) X(27) X(28) X(30) X(32)

// ---- strided axis ---------------------------------------------------------------------
// columns first .. left - 1 of a tile are there (at least one); the others load it too
// step 1: x[N2 n1 + n2] of column c -> S[n2 P + k1 C + c]
template <int M>
__device__ __noinline__ void cols_step1(const float2 *__restrict__ base, float2 *S, int first, int left, long es,
                                        int N2, int P, const float2 *__restrict__ W, float sgn) {
    for (int s = threadIdx.x; s < kF3Cols * N2; s += kF3Threads) {
        const int c = s & (kF3Cols - 1), n2 = s / kF3Cols;
        const float2 *src = base + (long)n2 * es + (c >= first && c < left ? c : max(first, 0));
        const long st = (long)N2 * es;
        float2 v[M];
#pragma unroll
        for (int n = 0; n < M; ++n, src += st) v[n] = *src;
#pragma unroll
        for (int n = 0; n < M; ++n) v[n].y *= sgn;
        fft_reg<M>(v);
        float2 *dst = S + n2 * P + c;
#pragma unroll
        for (int k = 0; k < M; ++k) dst[k * kF3Cols] = k ? cmul(v[k], __ldg(&W[n2 * k])) : v[k];
    }
}

// step 2: S -> X[k1 + N1 k2] scale
template <int M>
__device__ __noinline__ void cols_step2(float2 *__restrict__ base, const float2 *S, int first, int left, long es,
                                        int N1, int P, float sgn, float scale) {
    for (int s = threadIdx.x; s < kF3Cols * N1; s += kF3Threads) {
        const int c = s & (kF3Cols - 1), k1 = s / kF3Cols;
        const float2 *src = S + s;
        float2 u[M];
#pragma unroll
        for (int n = 0; n < M; ++n) u[n] = src[n * P];
        fft_reg<M>(u);
        if (c < first || c >= left) continue;
        float2 *dst = base + (long)k1 * es + c;
        const long st = (long)N1 * es;
        const float sy = scale * sgn;
#pragma unroll
        for (int k = 0; k < M; ++k) {
            *dst = make_float2(u[k].x * scale, u[k].y * sy);
            dst += st;
        }
    }
}

__global__ void __launch_bounds__(kF3Threads, 2)
fft3_cols_kernel(float2 *g0, float2 *g1, int ncols, long es, long bs, int N1, int N2, int P,
                 const float2 *__restrict__ W, float sgn, float scale) {
    extern __shared__ __align__(16) float2 f3_smem[];
    const int ncb = cols_tiles(ncols, es, kF3LogCols);
    const int cb = blockIdx.x % ncb;
    const long batch = blockIdx.x / ncb;
    float2 *base = (blockIdx.y == 0 ? g0 : g1) + batch * bs;
    const int c0 = cb * kF3Cols - cols_offset(base, es, kF3LogCols);
    if (c0 >= ncols) return;
    base += c0;
    switch (N1) {
#define FG_CASE(M) \
    case M: cols_step1<M>(base, f3_smem, -c0, ncols - c0, es, N2, P, W, sgn); break;
        FG_F3_LENGTHS(FG_CASE)
#undef FG_CASE
    }
    __syncthreads();
    switch (N2) {
#define FG_CASE(M) \
    case M: cols_step2<M>(base, f3_smem, -c0, ncols - c0, es, N1, P, sgn, scale); break;
        FG_F3_LENGTHS(FG_CASE)
#undef FG_CASE
    }
}

// ---- k axis -----------------------------------------------------------------------------
// the layout of a CTA's R row pairs: S[(r N2 + n2) Q + k1], D[r PZ + n]
struct Rows {
    int N, N1, N2, Q, PZ, R;
    uint32_t inv_n, inv_nh;  // e / N and e / (N/2 + 1) as the high word of a product
};

// step 1 of the forward pass: rows 2r and 2r + 1 of g (from row0; nrows in all)
template <int M>
__device__ __noinline__ void rows_step1(const float *__restrict__ g, float2 *S, long row0, long nrows, int Ng_pad,
                                        const Rows &d, const float2 *__restrict__ W) {
    const int N2 = d.N2;
    for (int s = threadIdx.x; s < d.R * N2; s += kF3Threads) {
        const int r = s / N2, n2 = s - r * N2;
        const long row = row0 + 2 * r;
        const float *a = g + row * Ng_pad + n2;
        const bool oka = row < nrows, okb = row + 1 < nrows;
        float2 v[M];
#pragma unroll
        for (int n = 0; n < M; ++n) {
            v[n].x = oka ? a[n * N2] : 0.f;
            v[n].y = okb ? a[Ng_pad + n * N2] : 0.f;
        }
        fft_reg<M>(v);
        float2 *dst = S + s * d.Q;
#pragma unroll
        for (int k = 0; k < M; ++k) dst[k] = k ? cmul(v[k], __ldg(&W[n2 * k])) : v[k];
    }
}

// step 1 from D (backward pass)
template <int M>
__device__ __noinline__ void rows_step1d(const float2 *D, float2 *S, const Rows &d, const float2 *__restrict__ W) {
    const int N2 = d.N2;
    for (int s = threadIdx.x; s < d.R * N2; s += kF3Threads) {
        const int r = s / N2, n2 = s - r * N2;
        float2 v[M];
#pragma unroll
        for (int n = 0; n < M; ++n) v[n] = D[r * d.PZ + n * N2 + n2];
        fft_reg<M>(v);
        float2 *dst = S + s * d.Q;
#pragma unroll
        for (int k = 0; k < M; ++k) dst[k] = k ? cmul(v[k], __ldg(&W[n2 * k])) : v[k];
    }
}

// step 2: S -> D in natural order
template <int M>
__device__ __noinline__ void rows_step2(const float2 *S, float2 *D, const Rows &d) {
    const int N1 = d.N1;
    for (int s = threadIdx.x; s < d.R * N1; s += kF3Threads) {
        const int r = s / N1, k1 = s - r * N1;
        const float2 *src = S + r * d.N2 * d.Q + k1;
        float2 u[M];
#pragma unroll
        for (int n = 0; n < M; ++n) u[n] = src[n * d.Q];
        fft_reg<M>(u);
        float2 *dst = D + r * d.PZ + k1;
#pragma unroll
        for (int k = 0; k < M; ++k) dst[k * N1] = u[k];
    }
}

__device__ __forceinline__ void rows_fft2(const float2 *S, float2 *D, const Rows &d) {
    switch (d.N2) {
#define FG_CASE(M) \
    case M: rows_step2<M>(S, D, d); break;
        FG_F3_LENGTHS(FG_CASE)
#undef FG_CASE
    }
}

__global__ void __launch_bounds__(kF3Threads, 2)
fft3_k_r2c_kernel(float *g0, float *g1, long nrows, int Ng_pad, Rows d, const float2 *__restrict__ W) {
    extern __shared__ __align__(16) float2 f3_smem[];
    float2 *S = f3_smem, *D = f3_smem + d.R * d.N2 * d.Q;
    float *g = blockIdx.y == 0 ? g0 : g1;
    const long row0 = (long)blockIdx.x * 2 * d.R;
    switch (d.N1) {
#define FG_CASE(M) \
    case M: rows_step1<M>(g, S, row0, nrows, Ng_pad, d, W); break;
        FG_F3_LENGTHS(FG_CASE)
#undef FG_CASE
    }
    __syncthreads();
    rows_fft2(S, D, d);
    __syncthreads();
    const int nh = d.N / 2 + 1;
    for (int e = threadIdx.x; e < d.R * nh; e += kF3Threads) {
        const int r = (int)__umulhi(e, d.inv_nh), k = e - r * nh;
        const long row = row0 + 2 * r;
        if (row >= nrows) break;
        const float2 z = D[r * d.PZ + k], y = D[r * d.PZ + (k ? d.N - k : 0)];
        float2 *out = reinterpret_cast<float2 *>(g + row * Ng_pad) + k;
        *out = make_float2(0.5f * (z.x + y.x), 0.5f * (z.y - y.y));
        if (row + 1 < nrows) out[Ng_pad / 2] = make_float2(0.5f * (z.y + y.y), 0.5f * (y.x - z.x));
    }
}

__global__ void __launch_bounds__(kF3Threads, 2)
fft3_k_c2r_kernel(float *g0, float *g1, long nrows, int Ng_pad, Rows d, const float2 *__restrict__ W, float scale) {
    extern __shared__ __align__(16) float2 f3_smem[];
    float2 *S = f3_smem, *D = f3_smem + d.R * d.N2 * d.Q;
    float *g = blockIdx.y == 0 ? g0 : g1;
    const long row0 = (long)blockIdx.x * 2 * d.R;
    const int N = d.N, nh = N / 2 + 1;
    // conj Z, Z = A + i B of a row pair over all N wavenumbers; the imaginary parts
    // of k = 0 and the Nyquist column are ignored
    for (int e = threadIdx.x; e < d.R * nh; e += kF3Threads) {
        const int r = (int)__umulhi(e, d.inv_nh), k = e - r * nh;
        const long row = row0 + 2 * r;
        const float2 *in = reinterpret_cast<const float2 *>(g + row * Ng_pad) + k;
        float2 a = row < nrows ? *in : make_float2(0.f, 0.f);
        float2 b = row + 1 < nrows ? in[Ng_pad / 2] : make_float2(0.f, 0.f);
        if (k == 0 || 2 * k == N) a.y = b.y = 0.f;
        D[r * d.PZ + k] = make_float2(a.x - b.y, -(a.y + b.x));
        if (k && 2 * k != N) D[r * d.PZ + N - k] = make_float2(a.x + b.y, a.y - b.x);
    }
    __syncthreads();
    switch (d.N1) {
#define FG_CASE(M) \
    case M: rows_step1d<M>(D, S, d, W); break;
        FG_F3_LENGTHS(FG_CASE)
#undef FG_CASE
    }
    __syncthreads();
    rows_fft2(S, D, d);
    __syncthreads();
    for (int e = threadIdx.x; e < d.R * N; e += kF3Threads) {
        const int r = (int)__umulhi(e, d.inv_n), n = e - r * N;
        const long row = row0 + 2 * r;
        if (row >= nrows) break;
        const float2 z = D[r * d.PZ + n];
        float *out = g + row * Ng_pad + n;
        *out = z.x * scale;
        if (row + 1 < nrows) out[Ng_pad] = -z.y * scale;
        if (n < Ng_pad - N) {  // the row padding keeps its values, scaled like the rest of the grid
            out[N] *= scale;
            if (row + 1 < nrows) out[Ng_pad + N] *= scale;
        }
    }
}

// ---- host side ----------------------------------------------------------------------------
static bool length_ok(int m) {
    switch (m) {
#define FG_CASE(M) \
    case M: return true;
        FG_F3_LENGTHS(FG_CASE)
#undef FG_CASE
    }
    return false;
}

// N = N1 N2, N1 >= N2, as close to each other as the factors allow
static bool split3(int N, int *N1, int *N2) {
    for (int b = 32; b >= 1; --b)
        if (N % b == 0 && N / b >= b && length_ok(b) && length_ok(N / b)) {
            *N1 = N / b;
            *N2 = b;
            return true;
        }
    return false;
}

static size_t cols3_smem(int N1, int N2, int *P) {
    *P = N1 * kF3Cols;
    return (size_t)N2 * *P * sizeof(float2);
}

// row pairs per CTA: about one step-1 and step-2 task per thread, two CTAs per SM
static Rows rows_shape(int N, int N1, int N2) {
    Rows d;
    d.N = N;
    d.N1 = N1;
    d.N2 = N2;
    d.Q = N1 | 1;
    d.PZ = N | 1;
    d.R = kF3Threads / N1;
    const size_t one = (size_t)(N2 * d.Q + d.PZ) * sizeof(float2);
    while (d.R > 1 && d.R * one > 64 * 1024) --d.R;
    if (d.R > 16) d.R = 16;
    // ceil(2^32 / v): exact for e < 2^32 / v, and e < R v <= 2^14
    d.inv_n = (uint32_t)((0x100000000ull + N - 1) / N);
    d.inv_nh = (uint32_t)((0x100000000ull + N / 2) / (N / 2 + 1));
    return d;
}

bool fft3_supported(int Ng, int prec) {
    int a, b, P;
    return prec == 4 && Ng >= 4 && split3(Ng, &a, &b) && cols3_smem(a, b, &P) <= 200 * 1024;
}

int fft3_cols(int N, const void *W, void *g0, void *g1, int ngrids, int ncols, long es, long bs, long nbatch, int sign,
              double scale, cudaStream_t s) {
    int N1, N2, P;
    if (!split3(N, &N1, &N2)) return set_error(ERR_UNSUPPORTED, "fft3_cols: N=%d", N);
    const size_t smem = cols3_smem(N1, N2, &P);
    FG_CUDA(cudaFuncSetAttribute(fft3_cols_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    const dim3 grid((unsigned)(cols_tiles(ncols, es, kF3LogCols) * nbatch), ngrids);
    fft3_cols_kernel<<<grid, kF3Threads, smem, s>>>((float2 *)g0, (float2 *)g1, ncols, es, bs, N1, N2, P,
                                                    (const float2 *)W, sign > 0 ? -1.f : 1.f, (float)scale);
    FG_LAUNCHED(1);
    return OK;
}

int fft3_k(int Ng, const void *W, void *g0, void *g1, int ngrids, bool forward, double scale, cudaStream_t s) {
    int N1, N2;
    if (!split3(Ng, &N1, &N2)) return set_error(ERR_UNSUPPORTED, "fft3_k: Ng=%d", Ng);
    const Rows d = rows_shape(Ng, N1, N2);
    const size_t smem = (size_t)d.R * (d.N2 * d.Q + d.PZ) * sizeof(float2);
    const long nrows = (long)Ng * Ng;
    const int Ng_pad = 2 * (Ng / 2 + 1);
    const dim3 grid((unsigned)ceil_div(nrows, 2L * d.R), ngrids);
    FG_CUDA(cudaFuncSetAttribute(fft3_k_r2c_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
    FG_CUDA(cudaFuncSetAttribute(fft3_k_c2r_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
    if (forward)
        fft3_k_r2c_kernel<<<grid, kF3Threads, smem, s>>>((float *)g0, (float *)g1, nrows, Ng_pad, d, (const float2 *)W);
    else
        fft3_k_c2r_kernel<<<grid, kF3Threads, smem, s>>>((float *)g0, (float *)g1, nrows, Ng_pad, d, (const float2 *)W,
                                                         (float)scale);
    FG_LAUNCHED(1);
    return OK;
}

}  // namespace fg
