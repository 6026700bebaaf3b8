// In-register FFTs of any length whose prime factors are 2, 3, 5, 7, 11 and 13,
// fully unrolled, with twiddles as compile-time constants.
#pragma once

#include "common.cuh"

namespace fg {

// cos and sin of 2 pi t / m in FP64 at compile time: the angle is reduced to
// [0, pi/4] by symmetry and the Taylor series summed until its terms vanish
struct CosSin {
    double c, s;
};
constexpr CosSin cos_sin_turn(long t, long m) {
    t %= m;
    if (t < 0) t += m;
    // 8 t / m octants: quadrant and remainder, exact in integers
    const long q = 4 * t / m;  // quadrant 0..3
    const long r4 = 4 * t - q * m;  // remaining angle = (r4 / m) * pi/2
    const bool swap = 2 * r4 > m;   // beyond pi/4: use the complement
    const long u = swap ? m - r4 : r4;
    const double x = 1.57079632679489661923 * (double)u / (double)m;
    double c = 1, s = x, tc = 1, ts = x;
    for (int n = 1; n < 14; ++n) {
        tc *= -x * x / ((2 * n - 1) * (2 * n));
        ts *= -x * x / ((2 * n) * (2 * n + 1));
        c += tc;
        s += ts;
    }
    const double cc = swap ? s : c, ss = swap ? c : s;  // cos, sin of the remainder
    return q == 0 ? CosSin{cc, ss} : q == 1 ? CosSin{-ss, cc} : q == 2 ? CosSin{-cc, -ss} : CosSin{ss, -cc};
}

template <typename T, int M>
struct TwTable {
    T c[M], s[M];
    constexpr TwTable() : c(), s() {
        for (int t = 0; t < M; ++t) {
            const CosSin v = cos_sin_turn(t, M);
            c[t] = (T)v.c;
            s[t] = (T)v.s;
        }
    }
};

// the radix taken off a length: 4 and 2 first, then the odd primes
constexpr int fft_radix(int m) {
    return m % 4 == 0 ? 4 : m % 2 == 0 ? 2 : m % 3 == 0 ? 3 : m % 5 == 0 ? 5 : m % 7 == 0 ? 7 : m % 11 == 0 ? 11 : 13;
}

// forward DFT (exp(-2 pi i nk / R)) of R values, natural order, in place
template <int R, typename T2>
__device__ __forceinline__ void dft_reg(T2 (&v)[R]) {
    using T = decltype(T2::x);
    if constexpr (R == 2) {
        const T2 a = v[0];
        v[0] = cadd(a, v[1]);
        v[1] = csub(a, v[1]);
    } else if constexpr (R == 4) {
        const T2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), e = csub(v[1], v[3]);
        const T2 d = mk2<T2>(e.y, -e.x);  // -i (v1 - v3)
        v[0] = cadd(a, c);
        v[2] = csub(a, c);
        v[1] = cadd(b, d);
        v[3] = csub(b, d);
    } else if constexpr (R > 2) {
        // odd R: sums and differences of v_r and v_(R-r)
        constexpr int H = (R - 1) / 2;
        constexpr TwTable<T, R> tw;
        T2 a[H], b[H];
        T2 x0 = v[0];
#pragma unroll
        for (int r = 0; r < H; ++r) {
            a[r] = cadd(v[r + 1], v[R - 1 - r]);
            b[r] = csub(v[r + 1], v[R - 1 - r]);
            x0 = cadd(x0, a[r]);
        }
        const T2 v0 = v[0];
        v[0] = x0;
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            T2 p = v0;
            T sx = 0, sy = 0;
#pragma unroll
            for (int r = 1; r <= H; ++r) {
                const T c = tw.c[(r * q) % R], s = tw.s[(r * q) % R];
                p.x += a[r - 1].x * c;
                p.y += a[r - 1].y * c;
                sx += b[r - 1].x * s;
                sy += b[r - 1].y * s;
            }
            // X_q = p - i s, X_(R-q) = p + i s
            v[q] = mk2<T2>(p.x + sy, p.y - sx);
            v[R - q] = mk2<T2>(p.x - sy, p.y + sx);
        }
    }
}

// forward FFT of M values in natural order, in place
template <int M, typename T2>
__device__ __forceinline__ void fft_reg(T2 (&v)[M]) {
    using T = decltype(T2::x);
    if constexpr (M > 1) {
        constexpr int R = fft_radix(M), K = M / R;
        if constexpr (K == 1) {
            dft_reg<R>(v);
        } else {
            constexpr TwTable<T, M> tw;
            T2 u[R][K];
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int k = 0; k < K; ++k) u[r][k] = v[r + R * k];
                fft_reg<K>(u[r]);
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
                T2 w[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int t = (r * k) % M;
                    if (t == 0) w[r] = u[r][k];
                    else if (4 * t == M) w[r] = mk2<T2>(u[r][k].y, -u[r][k].x);
                    else if (2 * t == M) w[r] = mk2<T2>(-u[r][k].x, -u[r][k].y);
                    else w[r] = cmul(u[r][k], mk2<T2>(tw.c[t], -tw.s[t]));
                }
                dft_reg<R>(w);
#pragma unroll
                for (int q = 0; q < R; ++q) v[k + K * q] = w[q];
            }
        }
    }
}

}  // namespace fg
