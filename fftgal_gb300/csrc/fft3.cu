// FP32 FFT passes for sizes that are no power of two (sm_103a): the radix passes of
// fft.cu's general kernels, fused.
//
// A self-sorting (Stockham) pass of radix R at block length Ns takes butterfly j
// from x[j + r N/R], twiddles W^(r (j mod Ns) N/(Ns R)), to (j / Ns) Ns R + j mod Ns +
// r Ns.  Up to three consecutive passes R1, R2, R3 (product M <= 32) need no memory in
// between: a thread that holds the M values a + r3 N/M + r2 N/(R1 R2) + r1 N/R1
// (a < N/M) has every butterfly of the three passes that its values meet.  So a
// length is cut into two groups of passes or more, the fewest and then those with the
// smallest largest one, e.g. 384 = (8)(8)(2 3), 225 = (3 3)(5 5): a thread loads a
// group's values (the first group from global memory, the others from shared),
// transforms them in registers and stores them (the last group to global memory).
// The arithmetic, twiddle tables and order of operations are the general kernels'.
// So are the results, bit for bit, with nvcc 13.0 (compared at 92 lengths): the
// butterflies leave the fusing of products to the compiler in both files, so another
// compiler may round them differently, which nothing relies on.  (A two-step form with
// its own factors, N = N1 N2 in registers around one trip through shared memory, is
// faster -- 384: 266 and 404 us for the passes below -- and its L2 error is no larger,
// but the power of a small grid is dominated by a few modes at the cube's corner,
// whose error then goes either way by up to 2.)
// Measured (GB300, both interlacing grids, us): Ng = 384 k pass 1402 -> 430, j + i 3655
// -> 893; Ng = 225 1083 -> 231, 1493 -> 217.  The general kernels spent it on a
// shared-memory round trip per radix, run-time divisions per element and constants
// converted from FP64; what is left is latency (128 registers for the longest groups
// hold the kernels to 16 warps per SM, long-scoreboard stalls lead; 80 registers and
// three CTAs or 384 threads were slower, 64 and 512 threads more so).
// The groups are instantiated once per kind of memory they go from and to, as
// functions selected by a switch.
#include "internal.h"
#include "common.cuh"

namespace fg {

// cos and sin of 2 pi m / R at compile time, FP64: the angle is reduced to [0, pi/4]
// by symmetry and the Taylor series summed until its terms vanish
struct CosSin {
    double c, s;
};
constexpr CosSin cos_sin_turn(long m, long R) {
    const long q = 4 * m / R, r4 = 4 * m - q * R;  // quadrant; the rest is (r4 / R) pi/2
    const bool swap = 2 * r4 > R;                  // beyond pi/4: the complement
    const long u = swap ? R - r4 : r4;
    const double x = 1.57079632679489661923 * (double)u / (double)R;
    double c = 1, s = x, tc = 1, ts = x;
    for (int n = 1; n < 14; ++n) {
        tc *= -x * x / ((2 * n - 1) * (2 * n));
        ts *= -x * x / ((2 * n) * (2 * n + 1));
        c += tc;
        s += ts;
    }
    const double cc = swap ? s : c, ss = swap ? c : s;
    return q == 0 ? CosSin{cc, ss} : q == 1 ? CosSin{-ss, cc} : q == 2 ? CosSin{-cc, -ss} : CosSin{ss, -cc};
}

// cos(2 pi m / R) and sign sin(2 pi m / R), m < R, of the odd radices
constexpr int dft_off(int R) { return R == 3 ? 0 : R == 5 ? 3 : R == 7 ? 8 : R == 11 ? 15 : 26; }
struct DftTable {
    float c[39], s[2][39];
    constexpr DftTable() : c(), s() {
        for (int R : {3, 5, 7, 11, 13})
            for (int m = 0; m < R; ++m) {
                const CosSin v = cos_sin_turn(m, R);
                c[dft_off(R) + m] = (float)v.c;
                s[0][dft_off(R) + m] = -(float)v.s;
                s[1][dft_off(R) + m] = (float)v.s;
            }
    }
};
__constant__ DftTable c_dft3 = DftTable();

// The butterflies of fft.cu's general kernels, for FP32.  The sign stays a run-time
// value as there, so that the compiler fuses the same products.
__device__ __forceinline__ void dft4(float2 &v0, float2 &v1, float2 &v2, float2 &v3, int sign) {
    const float2 a = cadd(v0, v2), b = csub(v0, v2);
    const float2 c = cadd(v1, v3), d = cmul_si(csub(v1, v3), sign);
    v0 = cadd(a, c);
    v2 = csub(a, c);
    v1 = cadd(b, d);
    v3 = csub(b, d);
}

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R], int sign) {
    if constexpr (R == 2) {
        const float2 t = v[0];
        v[0] = cadd(t, v[1]);
        v[1] = csub(t, v[1]);
    } else if constexpr (R == 4) {
        dft4(v[0], v[1], v[2], v[3], sign);
    } else if constexpr (R == 8) {
        const float h = 0.70710678118654752440f;
        float2 a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            a[r] = cadd(v[r], v[r + 4]);
            b[r] = csub(v[r], v[r + 4]);
        }
        b[1] = make_float2(h * (b[1].x - sign * b[1].y), h * (b[1].y + sign * b[1].x));
        b[2] = cmul_si(b[2], sign);
        b[3] = make_float2(h * (-b[3].x - sign * b[3].y), h * (-b[3].y + sign * b[3].x));
        dft4(a[0], a[1], a[2], a[3], sign);
        dft4(b[0], b[1], b[2], b[3], sign);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[2 * q] = a[q];
            v[2 * q + 1] = b[q];
        }
    } else if constexpr (R > 1) {
        constexpr int off = dft_off(R);
        const float *sn = c_dft3.s[sign > 0];
        float2 out[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            float sr = 0, si = 0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float c = c_dft3.c[off + (r * q) % R], s = sn[off + (r * q) % R];
                sr += v[r].x * c - v[r].y * s;
                si += v[r].x * s + v[r].y * c;
            }
            out[q] = make_float2(sr, si);
        }
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = out[q];
    }
}

// v w, contracted as the general kernels' twiddle product is
__device__ __forceinline__ float2 twiddle(float2 v, float2 w, int sign) {
    if (sign > 0) w.y = -w.y;
    return make_float2(__fmaf_rn(v.x, w.x, -__fmul_rn(v.y, w.y)),
                       __fmaf_rn(v.y, w.x, __fmul_rn(v.x, w.y)));
}

constexpr int kF3Threads = 256;

// the groups of consecutive radices (8s first, then 4 or 2, then odd primes in
// ascending order) with product <= 32
#define FG_F3_GROUPS(X)                                                                                          \
    X(8, 1, 1) X(4, 1, 1) X(2, 1, 1) X(3, 1, 1) X(5, 1, 1) X(7, 1, 1) X(11, 1, 1) X(13, 1, 1) X(8, 4, 1) X(8, 2, 1) \
        X(8, 3, 1) X(4, 3, 1) X(4, 5, 1) X(4, 7, 1) X(2, 3, 1) X(2, 5, 1) X(2, 7, 1) X(2, 11, 1) X(2, 13, 1)     \
            X(3, 3, 1) X(3, 5, 1) X(3, 7, 1) X(5, 5, 1) X(2, 3, 3) X(2, 3, 5) X(3, 3, 3)

constexpr int group_code(int r1, int r2, int r3) { return (r1 * 16 + r2) * 16 + r3; }

constexpr int kF3MaxGroups = 6;
struct Groups {
    int n, count;             // length, number of groups
    int code[kF3MaxGroups], len[kF3MaxGroups];
    const float2 *W;          // exp(-2 pi i t / n)
};

// Where a group's data lie.  Value e of column (or row) c: in global memory at
// p[c cs + e es] for first <= c < left (the others load one that is there and are not
// stored), in shared memory at off + e ncol + c (columns) or off + c cs + e + e / 16
// (rows: the padding spreads strided accesses over the banks) for all c.
struct Side {
    float2 *p;
    int off;
    long es, cs;
    int first, left;
};
struct GroupArgs {
    Side src, dst;
    const float2 *W;
    int n, ns;       // length, product of the radices before this group
    int ncol, logc;  // columns; logc >= 0: lanes along 2^logc = ncol columns, else along the values
    int sign;
    float scale;     // the stored values are multiplied with it
};

extern __shared__ __align__(16) float2 f3_smem[];

// KIND bit 0: from shared memory, bit 1: to shared memory.  From global memory is the
// first group (Ns = 1), to global memory the last (Ns M = N).  COLS: columns, the
// lanes along them and no padding; else rows, the lanes along their values.
template <int R1, int R2, int R3, int KIND, bool COLS>
__device__ __noinline__ void fft_group(const GroupArgs &g) {
    constexpr int M = R1 * R2 * R3;
    const int N = g.n, m = N / M, Ns = KIND == 2 ? 1 : (KIND == 1 ? m : g.ns), sign = g.sign, ncol = g.ncol;
    const float2 *__restrict__ W = g.W;
    const int t1 = N / (Ns * R1), t2 = N / (Ns * R1 * R2), t3 = N / (Ns * M);
    const float scale = g.scale;
    for (int first = 0; first < m * ncol; first += kF3Threads) {
        const int task = first + threadIdx.x, t = min(task, m * ncol - 1);
        int a, c;
        if constexpr (COLS) {
            c = t & (ncol - 1);
            a = t >> g.logc;
        } else {
            c = t / m;
            a = t - c * m;
        }
        const int blk = KIND == 2 ? a : (KIND == 1 ? 0 : a / Ns), jm = KIND == 2 ? 0 : a - blk * Ns;
        float2 v[R3][R2][R1];
        if constexpr (KIND & 1) {
            const float2 *s = f3_smem + g.src.off + (COLS ? a * ncol + c : c * (int)g.src.cs);
#pragma unroll
            for (int q = 0; q < M; ++q) {
                const int e = COLS ? m * ncol * q : a + m * q;
                v[q % R3][q / R3 % R2][q / (R3 * R2)] = s[COLS ? e : e + (e >> 4)];
            }
        } else {
            const int cc = c < g.src.first ? g.src.first : (c < g.src.left ? c : max(g.src.first, 0));
            const float2 *s = g.src.p + cc * g.src.cs + a * g.src.es;
            const long step = m * g.src.es;
#pragma unroll
            for (int q = 0; q < M; ++q, s += step) v[q % R3][q / R3 % R2][q / (R3 * R2)] = *s;
        }
        // pass 1
        if (Ns > 1) {
#pragma unroll
            for (int r1 = 1; r1 < R1; ++r1) {
                const float2 w = __ldg(&W[r1 * jm * t1]);
#pragma unroll
                for (int r2 = 0; r2 < R2; ++r2)
#pragma unroll
                    for (int r3 = 0; r3 < R3; ++r3) v[r3][r2][r1] = twiddle(v[r3][r2][r1], w, sign);
            }
        }
        float2 u[R3][R1][R2];  // after pass 1, by the inputs r2 of pass 2
#pragma unroll
        for (int r3 = 0; r3 < R3; ++r3)
#pragma unroll
            for (int r2 = 0; r2 < R2; ++r2) {
                dft<R1>(v[r3][r2], sign);
#pragma unroll
                for (int q = 0; q < R1; ++q) u[r3][q][r2] = v[r3][r2][q];
            }
        // pass 2
        float2 x[R1][R2][R3];  // by the inputs r3 of pass 3
#pragma unroll
        for (int q1 = 0; q1 < R1; ++q1) {
            if (R2 > 1 && (Ns > 1 || q1 > 0)) {
#pragma unroll
                for (int r2 = 1; r2 < R2; ++r2) {
                    const float2 w = __ldg(&W[r2 * (jm + q1 * Ns) * t2]);
#pragma unroll
                    for (int r3 = 0; r3 < R3; ++r3) u[r3][q1][r2] = twiddle(u[r3][q1][r2], w, sign);
                }
            }
#pragma unroll
            for (int r3 = 0; r3 < R3; ++r3) {
                dft<R2>(u[r3][q1], sign);
#pragma unroll
                for (int q2 = 0; q2 < R2; ++q2) x[q1][q2][r3] = u[r3][q1][q2];
            }
        }
        // pass 3
        if constexpr (R3 > 1) {
#pragma unroll
            for (int q1 = 0; q1 < R1; ++q1)
#pragma unroll
                for (int q2 = 0; q2 < R2; ++q2) {
                    if (Ns > 1 || q1 + q2 > 0) {
#pragma unroll
                        for (int r3 = 1; r3 < R3; ++r3)
                            x[q1][q2][r3] =
                                twiddle(x[q1][q2][r3], __ldg(&W[r3 * (jm + (q1 + q2 * R1) * Ns) * t3]), sign);
                    }
                    dft<R3>(x[q1][q2], sign);
                }
        }
        const int e0 = blk * Ns * M + jm;
        // in place, with no more tasks than threads: all have read before one writes
        if (KIND == 3 && g.src.off == g.dst.off) __syncthreads();
        if (task != t) continue;
        if constexpr (KIND & 2) {
            float2 *d = f3_smem + g.dst.off + (COLS ? e0 * ncol + c : c * (int)g.dst.cs);
#pragma unroll
            for (int q = 0; q < M; ++q) {
                const int e = COLS ? Ns * ncol * q : e0 + Ns * q;
                d[COLS ? e : e + (e >> 4)] = x[q % R1][q / R1 % R2][q / (R1 * R2)];
            }
        } else {
            if (c < g.dst.first || c >= g.dst.left) continue;
            float2 *d = g.dst.p + c * g.dst.cs + e0 * g.dst.es;
            const long step = Ns * g.dst.es;
#pragma unroll
            for (int q = 0; q < M; ++q, d += step) {
                const float2 y = x[q % R1][q / R1 % R2][q / (R1 * R2)];
                *d = make_float2(y.x * scale, y.y * scale);
            }
        }
    }
}

template <int KIND, bool COLS>
__device__ __forceinline__ void run_group(int code, const GroupArgs &g) {
    switch (code) {
#define FG_CASE(A, B, C) \
    case group_code(A, B, C): fft_group<A, B, C, KIND, COLS>(g); break;
        FG_F3_GROUPS(FG_CASE)
#undef FG_CASE
    }
}

// The whole transform: groups from src (global memory, or the shared buffer at src.off with
// p null) through the shared buffers at 0 and `other` (laid out as buf) to dst, in
// global memory or, with p null, a buffer; the offset of the last one used is
// returned, and the caller synchronises before reading it.
template <bool COLS>
__device__ __forceinline__ int fft_groups(const Groups &f, const Side &src, const Side &dst, const Side &buf,
                                          int other, int ncol, int logc, int sign, float scale) {
    GroupArgs g;
    g.W = f.W;
    g.n = f.n;
    g.ns = 1;
    g.ncol = ncol;
    g.logc = logc;
    g.sign = sign;
    g.src = src;
    for (int q = 0; q < f.count; ++q) {
        const bool last = q == f.count - 1;
        const bool from = g.src.p == nullptr, to = !last || dst.p == nullptr;
        g.dst = last ? dst : buf;
        if (to) g.dst.off = !from ? 0 : (f.n / f.len[q] * ncol <= kF3Threads ? g.src.off : other - g.src.off);
        g.scale = last ? scale : 1.f;
        if (!from) run_group<2, COLS>(f.code[q], g);
        else if (to) run_group<3, COLS>(f.code[q], g);
        else run_group<1, COLS>(f.code[q], g);
        if (!last) __syncthreads();
        g.ns *= f.len[q];
        g.src = g.dst;
    }
    return g.dst.off;
}

// ---- strided axes -----------------------------------------------------------------------
__global__ void __launch_bounds__(kF3Threads, 2)
fft3_cols_kernel(float2 *g0, float2 *g1, int ncols, long es, long bs, Groups f, int logc, int sign, float scale) {
    const int C = 1 << logc, ncb = cols_tiles(ncols, es, logc);
    const int cb = blockIdx.x % ncb;
    const long batch = blockIdx.x / ncb;
    float2 *base = (blockIdx.y == 0 ? g0 : g1) + batch * bs;
    const int c0 = cb * C - cols_offset(base, es, logc);
    if (c0 >= ncols) return;
    const Side gl = {base + c0, 0, es, 1, -c0, ncols - c0}, buf = {nullptr, 0, 0, 0, 0, C};
    fft_groups<true>(f, gl, gl, buf, f.n * C, C, logc, sign, scale);
}

// ---- k axis -------------------------------------------------------------------------------
// R rows per CTA; a row's n values (n = Ng/2 packed pairs for even Ng, else Ng) at
// pitch P in shared memory, value m at m + m / 16
struct Rows {
    int R, P;
    uint32_t inv_nh, inv_n, inv_np;  // e / (Ng/2 + 1), e / n and e / (n/2 + 1) as high words of products
};
__device__ __forceinline__ int row_pos(int m) { return m + (m >> 4); }

__global__ void __launch_bounds__(kF3Threads, 2)
fft3_k_r2c_kernel(float *g0, float *g1, long nrows, int Ng, Rows d, Groups f, const float2 *__restrict__ rtw) {
    const int R = d.R, P = d.P;
    const int Ng_pad = 2 * (Ng / 2 + 1), nh = Ng / 2 + 1, Nc = f.n;
    const bool even = (Ng & 1) == 0;
    const long row0 = (long)blockIdx.x * R;
    float *g = (blockIdx.y == 0 ? g0 : g1) + row0 * Ng_pad;
    const int left = nrows - row0 < R ? (int)(nrows - row0) : R;
    const Side buf = {nullptr, 0, 1, P, 0, R};
    Side src = {reinterpret_cast<float2 *>(g), 0, 1, Ng_pad / 2, 0, left}, dst = buf;
    if (!even) {  // real rows as complex ones
        for (int e = threadIdx.x; e < R * Nc; e += kF3Threads) {
            const int r = (int)__umulhi(e, d.inv_n), m = e - r * Nc;
            f3_smem[r * P + row_pos(m)] = make_float2(r < left ? g[(long)r * Ng_pad + m] : 0.f, 0.f);
        }
        __syncthreads();
        src = buf;
    }
    const int fin = fft_groups<false>(f, src, dst, buf, R * P, R, -1, -1, 1.f);
    __syncthreads();
    for (int e = threadIdx.x; e < left * nh; e += kF3Threads) {
        const int r = (int)__umulhi(e, d.inv_nh), k = e - r * nh;
        const float2 *s = f3_smem + fin + r * P;
        float2 X;
        if (even) {
            const int k1 = k == Nc ? 0 : k, k2 = k == 0 || k == Nc ? 0 : Nc - k;
            const float2 z1 = s[row_pos(k1)];
            const float2 z2 = cconj(s[row_pos(k2)]);
            const float2 E = make_float2(0.5f * (z1.x + z2.x), 0.5f * (z1.y + z2.y));
            const float2 D = csub(z1, z2);
            const float2 O = make_float2(0.5f * D.y, -0.5f * D.x);
            X = cadd(E, cmul(rtw[k], O));
        } else {
            X = s[row_pos(k)];
        }
        reinterpret_cast<float2 *>(g + (long)r * Ng_pad)[k] = X;
    }
}

__global__ void __launch_bounds__(kF3Threads, 2)
fft3_k_c2r_kernel(float *g0, float *g1, long nrows, int Ng, Rows d, Groups f, const float2 *__restrict__ rtw,
                  float scale) {
    const int R = d.R, P = d.P;
    const int Ng_pad = 2 * (Ng / 2 + 1), nh = Ng / 2 + 1, Nc = f.n;
    const bool even = (Ng & 1) == 0;
    const long row0 = (long)blockIdx.x * R;
    float *g = (blockIdx.y == 0 ? g0 : g1) + row0 * Ng_pad;
    const int left = nrows - row0 < R ? (int)(nrows - row0) : R;
    if (even) {
        // Z[k] = A[k] + i B[k], A = X[k] + X[k+h], B = (X[k] - X[k+h]) e^{+2 pi i k/Ng},
        // X[k+h] = conj X[h-k]; pairs (k, Nc-k) by one thread
        const int npair = Nc / 2 + 1;
        for (int e = threadIdx.x; e < left * npair; e += kF3Threads) {
            const int r = (int)__umulhi(e, d.inv_np), k = e - r * npair, k2 = Nc - k;
            const float2 *row = reinterpret_cast<const float2 *>(g + (long)r * Ng_pad);
            float2 xa = row[k], xb = row[k2];
            if (k == 0) xa.y = xb.y = 0.f;
            float2 *o = f3_smem + r * P;
            {
                const float2 y = cconj(xb);
                const float2 A = cadd(xa, y);
                const float2 B = cmul(csub(xa, y), cconj(rtw[k]));
                o[row_pos(k)] = make_float2(A.x - B.y, A.y + B.x);
            }
            if (k2 != k && k2 < Nc) {
                const float2 y = cconj(xa);
                const float2 A = cadd(xb, y);
                const float2 B = cmul(csub(xb, y), cconj(rtw[k2]));
                o[row_pos(k2)] = make_float2(A.x - B.y, A.y + B.x);
            }
        }
    } else {
        for (int e = threadIdx.x; e < left * nh; e += kF3Threads) {
            const int r = (int)__umulhi(e, d.inv_nh), k = e - r * nh;
            float2 v = reinterpret_cast<const float2 *>(g + (long)r * Ng_pad)[k];
            if (k == 0) v.y = 0.f;
            f3_smem[r * P + row_pos(k)] = v;
            if (k > 0) f3_smem[r * P + row_pos(Ng - k)] = cconj(v);
        }
    }
    __syncthreads();
    const Side buf = {nullptr, 0, 1, P, 0, R};
    Side dst = buf;
    if (even) {  // packed pairs straight to the rows
        dst = {reinterpret_cast<float2 *>(g), 0, 1, Ng_pad / 2, 0, left};
        fft_groups<false>(f, buf, dst, buf, R * P, R, -1, 1, scale);
    } else {
        const int fin = fft_groups<false>(f, buf, dst, buf, R * P, R, -1, 1, 1.f);
        __syncthreads();
        for (int e = threadIdx.x; e < left * Nc; e += kF3Threads) {
            const int r = (int)__umulhi(e, d.inv_n), m = e - r * Nc;
            g[(long)r * Ng_pad + m] = f3_smem[fin + r * P + row_pos(m)].x * scale;
        }
    }
    // the row padding keeps its values, scaled like the rest of the grid
    const int pad = Ng_pad - Ng;
    for (int e = threadIdx.x; e < left * pad; e += kF3Threads) g[(long)(e / pad) * Ng_pad + Ng + e % pad] *= scale;
}

// ---- host side ----------------------------------------------------------------------------
static bool group_ok(int r1, int r2, int r3) {
    switch (group_code(r1, r2, r3)) {
#define FG_CASE(A, B, C) \
    case group_code(A, B, C): return true;
        FG_F3_GROUPS(FG_CASE)
#undef FG_CASE
    }
    return false;
}

// rounds of kF3Threads tasks times the work of one: its values, and about as much as
// six more for indices, a stretch of shared memory and the barrier
static long group_cost(int n, int len, int ncol) {
    return ceil_div((long)n / len * ncol, kF3Threads) * (len + 6);
}

// cut the radices into the fewest groups, and among those the one with the smallest largest
static bool make_groups(const Fft1dPlan &p, Groups *out) {
    const int n = p.nrad;
    struct Best {
        int count = 1 << 20, worst = 0, cut = 0;
    };
    Best best[kMaxRadixPasses + 1];
    if (n < 1) return false;
    best[0].count = 0;
    for (int e = 1; e <= n; ++e)
        for (int l = 1; l <= 3 && l <= e; ++l) {
            const int *r = p.rad + e - l;
            if (!group_ok(r[0], l > 1 ? r[1] : 1, l > 2 ? r[2] : 1)) continue;
            int len = 1;
            for (int q = 0; q < l; ++q) len *= r[q];
            const int count = best[e - l].count + 1, worst = len > best[e - l].worst ? len : best[e - l].worst;
            if (count < best[e].count || (count == best[e].count && worst < best[e].worst)) best[e] = {count, worst, l};
        }
    if (best[n].count > kF3MaxGroups) return false;
    out->n = p.n;
    out->count = best[n].count;
    out->W = static_cast<const float2 *>(p.tw);
    for (int e = n, q = out->count - 1; e > 0; --q) {
        const int l = best[e].cut;
        const int *r = p.rad + e - l;
        out->code[q] = group_code(r[0], l > 1 ? r[1] : 1, l > 2 ? r[2] : 1);
        out->len[q] = r[0] * (l > 1 ? r[1] : 1) * (l > 2 ? r[2] : 1);
        e -= l;
    }
    return true;
}

// shared buffers that groups q0 .. q1 - 1, which go from shared memory to shared, need
static int buffers(const Groups &f, int q0, int q1, int ncol) {
    for (int q = q0; q < q1; ++q)
        if (f.n / f.len[q] * ncol > kF3Threads) return 2;
    return 1;
}

constexpr size_t kF3Smem = 100 * 1024;  // two CTAs per SM

// columns per CTA: 8, 16 or 32 (64- to 256-byte rows), whatever costs least per column
// with room for two CTAs; where not even 8 columns fit (some lengths from 810 on, all
// above 864) 4 or 2, whose rows of 32 or 16 bytes waste a part of each line
static bool cols_shape(const Groups &f, int *logc, size_t *smem) {
    long best = 0;
    *logc = -1;
    for (int l = 5; l >= 1; --l) {
        const size_t need = (size_t)buffers(f, 1, f.count - 1, 1 << l) * f.n * (1 << l) * sizeof(float2);
        if (need > kF3Smem) continue;
        if (l < 3 && *logc >= 0) break;
        long cost = 0;
        for (int q = 0; q < f.count; ++q) cost += group_cost(f.n, f.len[q], 1 << l);
        cost <<= 5 - l;
        if (*logc < 0 || cost < best) {
            best = cost;
            *logc = l;
            *smem = need;
        }
    }
    return *logc >= 0;
}

static uint32_t inverse(int v) { return (uint32_t)((0x100000000ull + v - 1) / v); }  // exact for e < 2^32 / v

// rows per CTA: the number that costs least per row
static bool rows_shape(const Groups &f, int Ng, Rows *d, size_t *smem) {
    const int nh = Ng / 2 + 1;
    d->P = (f.n + (f.n >> 4)) | 1;
    d->R = 0;
    double best = 0;
    for (int R = 1; R <= 64; ++R) {
        const size_t need = (size_t)buffers(f, 0, f.count, R) * R * d->P * sizeof(float2);
        if (need > kF3Smem) continue;
        long cost = 40 + 8 * ceil_div((long)R * nh, kF3Threads);
        for (int q = 0; q < f.count; ++q) cost += group_cost(f.n, f.len[q], R);
        if (d->R == 0 || (double)cost / R < best) {
            best = (double)cost / R;
            d->R = R;
            *smem = need;
        }
    }
    d->inv_nh = inverse(nh);
    d->inv_n = inverse(f.n);
    d->inv_np = inverse(f.n / 2 + 1);
    return d->R > 0 && Ng <= 8192;
}

bool fft3_supported(const FftPlan *p) {
    Groups f, h;
    int a;
    Rows d;
    size_t s;
    return p->prec == 4 && p->Ng >= 4 && make_groups(p->axis, &f) && f.count > 1 && cols_shape(f, &a, &s) &&
           make_groups(p->even ? p->half : p->axis, &h) && rows_shape(h, p->Ng, &d, &s);
}

int fft3_cols(const FftPlan *p, void *g0, void *g1, int ngrids, long es, long bs, int sign, double scale,
              cudaStream_t s) {
    Groups f;
    int logc;
    size_t smem;
    if (!make_groups(p->axis, &f) || !cols_shape(f, &logc, &smem))
        return set_error(ERR_UNSUPPORTED, "fft3_cols: N=%d", p->Ng);
    FG_CUDA(cudaFuncSetAttribute(fft3_cols_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kF3Smem));
    const dim3 grid((unsigned)(cols_tiles(p->nh, es, logc) * p->Ng), ngrids);
    fft3_cols_kernel<<<grid, kF3Threads, smem, s>>>((float2 *)g0, (float2 *)g1, p->nh, es, bs, f, logc, sign,
                                                    (float)scale);
    FG_LAUNCHED(1);
    return OK;
}

int fft3_k(const FftPlan *p, void *g0, void *g1, int ngrids, bool forward, double scale, cudaStream_t s) {
    Groups f;
    Rows d;
    size_t smem;
    if (!make_groups(p->even ? p->half : p->axis, &f) || !rows_shape(f, p->Ng, &d, &smem))
        return set_error(ERR_UNSUPPORTED, "fft3_k: Ng=%d", p->Ng);
    const long nrows = (long)p->Ng * p->Ng;
    const dim3 grid((unsigned)ceil_div(nrows, d.R), ngrids);
    FG_CUDA(cudaFuncSetAttribute(fft3_k_r2c_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kF3Smem));
    FG_CUDA(cudaFuncSetAttribute(fft3_k_c2r_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kF3Smem));
    const float2 *rtw = (const float2 *)p->rtw;
    if (forward)
        fft3_k_r2c_kernel<<<grid, kF3Threads, smem, s>>>((float *)g0, (float *)g1, nrows, p->Ng, d, f, rtw);
    else
        fft3_k_c2r_kernel<<<grid, kF3Threads, smem, s>>>((float *)g0, (float *)g1, nrows, p->Ng, d, f, rtw,
                                                         (float)scale);
    FG_LAUNCHED(1);
    return OK;
}

}  // namespace fg
