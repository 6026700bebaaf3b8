// Learned aliasing correction: a 5 -> 64 -> 64 -> 64 -> 3 perceptron (tanh
// hidden units, linear output, FP32) that maps the single-paint multipoles of
// a k bin to the interlaced ones, and its training kernels (mean squared
// error, batch gradients, Adam).  No counterpart in the reference: the
// interlaced estimator (fft_p2k, src/fft.c:257-276) is the training target and the measure of its error.
//
// Features of bin b (fftgal_alias_features), den = |P0| + Pshot:
//   k / k_Nyq, Pshot / den, P2 / den, P4 / den, d ln den / d ln k (neighbours);
// outputs y_l with P_l^interlaced - P_l^single = den e(k / k_Nyq) y_l for
// l = 0, 2, 4, e(u) = u^6 / (1 + u^6) (fftgal_alias_envelope).  The envelope
// takes out the steep rise of the aliased power towards k_Nyq (the measured
// differences grow about as u^6 below u = 1), so one squared error weighs
// every k range alike.
//
// Parameter layout (floats): W1[5][64] b1[64] W2[64][64] b2[64] W3[64][64]
// b3[64] W4[64][3] b4[3].
#include "internal.h"
#include "common.cuh"
#include "fftgal_gb300.h"

#include <cmath>
#include <math.h>
#include <vector>

namespace fg {

constexpr int kIn = 5, kHid = 64, kOut = 3;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kIn * kHid, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid,
              kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kHid, kOffW4 = kOffB3 + kHid,
              kOffB4 = kOffW4 + kHid * kOut, kNParams = kOffB4 + kOut;
constexpr int kMlpThreads = 256, kMlpS = 32;  // samples per CTA round

// Gradient kernel.  Activations and deltas are kept as [unit][sample] with a pitch of
// kPitch floats, W2 and W3 as [in][out] with a pitch of kWPitch (odd: a warp reads
// a row or a column of either without bank conflicts).  Warp w takes samples 4w ..
// 4w + 3, lane l the units l and l + 32 of a layer: 8 sums per thread and step from
// one broadcast of 4 samples and two weights.  Every sum runs over its inputs (a
// weight's gradient over the samples) in ascending order.  A training step at n =
// 4096 (128 CTAs): 104 us with one output per thread at a time (two shared loads
// per multiply-add, one scalar atomic per gradient and CTA; 68 us the kernel), 57 us
// so.
constexpr int kPitch = 36, kWPitch = 65;

// out[l], out[l + 32] of the warp's 4 samples: z = b + sum_i x[i] W[i][.], i < nin
template <int NIN>
__device__ __forceinline__ void mlp_dense(const float *x, const float *W, int wp, const float *b, float (&z)[2][4],
                                          int lane, int warp) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        z[0][q] = b[lane];
        z[1][q] = b[lane + 32];
    }
#pragma unroll 8
    for (int i = 0; i < NIN; ++i) {
        const float4 v = *reinterpret_cast<const float4 *>(x + i * kPitch + 4 * warp);
        const float w0 = W[i * wp + lane], w1 = W[i * wp + lane + 32];
        z[0][0] = fmaf(v.x, w0, z[0][0]);
        z[0][1] = fmaf(v.y, w0, z[0][1]);
        z[0][2] = fmaf(v.z, w0, z[0][2]);
        z[0][3] = fmaf(v.w, w0, z[0][3]);
        z[1][0] = fmaf(v.x, w1, z[1][0]);
        z[1][1] = fmaf(v.y, w1, z[1][1]);
        z[1][2] = fmaf(v.z, w1, z[1][2]);
        z[1][3] = fmaf(v.w, w1, z[1][3]);
    }
}

__device__ __forceinline__ void mlp_put(float *a, const float (&z)[2][4], int lane, int warp) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float4 *>(a + (lane + 32 * h) * kPitch + 4 * warp) =
            make_float4(z[h][0], z[h][1], z[h][2], z[h][3]);
}

// d[i] = (sum_j dn[j] W[i][j]) (1 - a[i]^2) for hidden units i = l, l + 32
template <int NN>
__device__ __forceinline__ void mlp_back(const float *dn, const float *W, int wp, const float *a, float *d, int lane,
                                         int warp) {
    float g[2][4] = {};
#pragma unroll 8
    for (int j = 0; j < NN; ++j) {
        const float4 v = *reinterpret_cast<const float4 *>(dn + j * kPitch + 4 * warp);
        const float w0 = W[lane * wp + j], w1 = W[(lane + 32) * wp + j];
        g[0][0] = fmaf(v.x, w0, g[0][0]);
        g[0][1] = fmaf(v.y, w0, g[0][1]);
        g[0][2] = fmaf(v.z, w0, g[0][2]);
        g[0][3] = fmaf(v.w, w0, g[0][3]);
        g[1][0] = fmaf(v.x, w1, g[1][0]);
        g[1][1] = fmaf(v.y, w1, g[1][1]);
        g[1][2] = fmaf(v.z, w1, g[1][2]);
        g[1][3] = fmaf(v.w, w1, g[1][3]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float4 v = *reinterpret_cast<const float4 *>(a + (lane + 32 * h) * kPitch + 4 * warp);
        g[h][0] *= 1.f - v.x * v.x;
        g[h][1] *= 1.f - v.y * v.y;
        g[h][2] *= 1.f - v.z * v.z;
        g[h][3] *= 1.f - v.w * v.w;
    }
    mlp_put(d, g, lane, warp);
}

// four neighbouring gradients; one vector atomic where the caller's array is 16-byte aligned
__device__ __forceinline__ void grad_add4(float *g, float a, float b, float c, float d, bool vec) {
    if (vec) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
    } else {
        atomicAdd(g, a);
        atomicAdd(g + 1, b);
        atomicAdd(g + 2, c);
        atomicAdd(g + 3, d);
    }
}

// gW[i][j] += sum_s x[i][s] d[j][s] (64 outputs), gb[j] += sum_s d[j][s]: 4 x 4 weights per thread
template <int NIN>
__device__ __forceinline__ void mlp_accum64(const float *x, const float *d, float *gW, float *gb, bool vec) {
    for (int t = threadIdx.x; t < (NIN + 3) / 4 * 16; t += kMlpThreads) {
        const int j0 = 4 * (t & 15), i0 = 4 * (t >> 4);
        float g[4][4] = {};
#pragma unroll 2
        for (int q = 0; q < kMlpS; q += 4) {
            float4 u[4], v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                u[e] = i0 + e < NIN ? *reinterpret_cast<const float4 *>(x + (i0 + e) * kPitch + q)
                                    : make_float4(0.f, 0.f, 0.f, 0.f);
                v[e] = *reinterpret_cast<const float4 *>(d + (j0 + e) * kPitch + q);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    g[i][j] = fmaf(u[i].w, v[j].w,
                                   fmaf(u[i].z, v[j].z, fmaf(u[i].y, v[j].y, fmaf(u[i].x, v[j].x, g[i][j]))));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i0 + i < NIN) grad_add4(gW + (i0 + i) * kHid + j0, g[i][0], g[i][1], g[i][2], g[i][3], vec);
    }
    for (int j = threadIdx.x; j < kHid; j += kMlpThreads) {
        float g = 0.f;
        for (int q = 0; q < kMlpS; ++q) g += d[j * kPitch + q];
        atomicAdd(&gb[j], g);
    }
}

// grad += d/dparams of sum_s scale * |y_s - t_s|^2 (scale = 1/n for the mean), loss += that sum
__global__ void __launch_bounds__(kMlpThreads)
mlp_grad_kernel(const float *__restrict__ params, const float *__restrict__ X, const float *__restrict__ T, long n,
                float scale, float *__restrict__ grad, float *__restrict__ loss, int vec) {
    extern __shared__ __align__(16) float sm[];
    float *W2 = sm, *W3 = W2 + kHid * kWPitch;     // [64][kWPitch]
    float *W1 = W3 + kHid * kWPitch;               // [5][64]
    float *W4 = W1 + kIn * kHid;                   // [64][3]
    float *b1 = W4 + kHid * kOut, *b2 = b1 + kHid, *b3 = b2 + kHid, *b4 = b3 + kHid;
    float *x0 = b4 + 4;                            // [5][kPitch] (rows are 16-byte aligned)
    float *a1 = x0 + kIn * kPitch;                 // [64][kPitch]
    float *a2 = a1 + kHid * kPitch, *a3 = a2 + kHid * kPitch;
    float *dy = a3 + kHid * kPitch;                // [3][kPitch] output deltas
    float *d3 = dy + kOut * kPitch, *d2 = d3 + kHid * kPitch, *d1 = d2 + kHid * kPitch;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int e = tid; e < kHid * kHid; e += kMlpThreads) {
        W2[e / kHid * kWPitch + e % kHid] = params[kOffW2 + e];
        W3[e / kHid * kWPitch + e % kHid] = params[kOffW3 + e];
    }
    for (int e = tid; e < kIn * kHid; e += kMlpThreads) W1[e] = params[kOffW1 + e];
    for (int e = tid; e < kHid * kOut; e += kMlpThreads) W4[e] = params[kOffW4 + e];
    if (tid < kHid) {
        b1[tid] = params[kOffB1 + tid];
        b2[tid] = params[kOffB2 + tid];
        b3[tid] = params[kOffB3 + tid];
        if (tid < kOut) b4[tid] = params[kOffB4 + tid];
    }
    float part = 0.f;  // this lane's share of the loss
    for (long s0 = (long)blockIdx.x * kMlpS; s0 < n; s0 += (long)gridDim.x * kMlpS) {
        const int S = n - s0 < kMlpS ? (int)(n - s0) : kMlpS;
        __syncthreads();  // the parameters, or the previous round's reads
        for (int e = tid; e < kMlpS * kIn; e += kMlpThreads) {
            const int q = e / kIn, i = e - q * kIn;
            // beyond the last sample its copies, whose output deltas are 0: values of their
            // own could make 0 x inf = NaN of a weight that is infinite
            x0[i * kPitch + q] = X[q < S ? s0 * kIn + e : (n - 1) * kIn + i];
        }
        __syncthreads();
        float z[2][4];
        // a warp's layers use its own 4 samples only: no barrier between them
        mlp_dense<kIn>(x0, W1, kHid, b1, z, lane, warp);
#pragma unroll
        for (int e = 0; e < 8; ++e) z[e >> 2][e & 3] = tanhf(z[e >> 2][e & 3]);
        mlp_put(a1, z, lane, warp);
        __syncwarp();
        mlp_dense<kHid>(a1, W2, kWPitch, b2, z, lane, warp);
#pragma unroll
        for (int e = 0; e < 8; ++e) z[e >> 2][e & 3] = tanhf(z[e >> 2][e & 3]);
        mlp_put(a2, z, lane, warp);
        __syncwarp();
        mlp_dense<kHid>(a2, W3, kWPitch, b3, z, lane, warp);
#pragma unroll
        for (int e = 0; e < 8; ++e) z[e >> 2][e & 3] = tanhf(z[e >> 2][e & 3]);
        mlp_put(a3, z, lane, warp);
        __syncwarp();
        // outputs and their deltas: lane = (sample, output) of the warp's 12
        if (lane < 4 * kOut) {
            const int q = 4 * warp + lane / kOut, o = lane % kOut;
            float y = b4[o];
#pragma unroll 8
            for (int i = 0; i < kHid; ++i) y = fmaf(a3[i * kPitch + q], W4[i * kOut + o], y);
            float r = 0.f;
            if (q < S) r = y - T[(s0 + q) * kOut + o];
            part += scale * r * r;
            dy[o * kPitch + q] = 2.f * scale * r;
        }
        __syncwarp();
        mlp_back<kOut>(dy, W4, kOut, a3, d3, lane, warp);
        __syncwarp();
        mlp_back<kHid>(d3, W3, kWPitch, a2, d2, lane, warp);
        __syncwarp();
        mlp_back<kHid>(d2, W2, kWPitch, a1, d1, lane, warp);
        __syncthreads();
        mlp_accum64<kHid>(a2, d3, grad + kOffW3, grad + kOffB3, vec);
        mlp_accum64<kHid>(a1, d2, grad + kOffW2, grad + kOffB2, vec);
        mlp_accum64<kIn>(x0, d1, grad + kOffW1, grad + kOffB1, vec);
        for (int e = tid; e < kHid * kOut + kOut; e += kMlpThreads) {
            // W4 and b4: one of the 195 sums per thread
            const int o = e % kOut, i = e / kOut;
            float g = 0.f;
            for (int q = 0; q < kMlpS; ++q)
                g = i < kHid ? fmaf(a3[i * kPitch + q], dy[o * kPitch + q], g) : g + dy[o * kPitch + q];
            atomicAdd(i < kHid ? &grad[kOffW4 + e] : &grad[kOffB4 + o], g);
        }
    }
    // the loss: one addition to the caller's sum per CTA, as few roundings as there are CTAs
    __shared__ float wsum[kMlpThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) wsum[warp] = part;
    __syncthreads();
    if (tid == 0) {
        float sum = 0.f;
        for (int w = 0; w < kMlpThreads / 32; ++w) sum += wsum[w];
        atomicAdd(loss, sum);
    }
}

__global__ void mlp_adam_kernel(float *__restrict__ params, const float *__restrict__ grad, float *__restrict__ m,
                                float *__restrict__ v, float lr, float beta1, float beta2, float eps, float c1,
                                float c2) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= kNParams) return;
    const float g = grad[e];
    const float mm = beta1 * m[e] + (1.f - beta1) * g;
    const float vv = beta2 * v[e] + (1.f - beta2) * g * g;
    m[e] = mm;
    v[e] = vv;
    params[e] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
}

// y = f(x): a warp takes NS samples at a time, lane l the hidden units l and l + 32, the
// sums over the inputs in ascending order.  NS = 1 where there are few samples: the
// learned call at Ng = 256 (222 bins, 56 CTAs) 536 -> 467 us against one thread per
// sample (two CTAs, the activations in local memory: 67 us the kernel).  NS = 4 shares
// the two weights that a lane reads per input among four samples, from as many samples
// as give every warp four: 2e4 samples 54 -> 31 us, 7e5 1311 -> 450 (a thread per sample:
// 74 and 691).
constexpr int kFwdWarps = 4;
template <int NS> struct __align__(4 * NS) Samples {
    float v[NS];
};
template <int NS>
__global__ void __launch_bounds__(32 * kFwdWarps)
mlp_forward_kernel(const float *__restrict__ params, const float *__restrict__ X, long n, float *__restrict__ Y) {
    __shared__ __align__(16) float P[kNParams];
    __shared__ Samples<NS> act[kFwdWarps][2][kHid];
    for (int e = threadIdx.x; e < kNParams; e += blockDim.x) P[e] = params[e];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Samples<NS> *a = act[warp][0], *b = act[warp][1];
    const long step = (long)gridDim.x * kFwdWarps * NS;
    for (long s = (blockIdx.x * (long)kFwdWarps + warp) * NS; s < n; s += step) {
        auto dense = [&](const Samples<NS> *x, int nin, int oW, int ob, Samples<NS> *out) {
            Samples<NS> z0, z1;
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                z0.v[q] = P[ob + lane];
                z1.v[q] = P[ob + lane + 32];
            }
#pragma unroll 8
            for (int i = 0; i < nin; ++i) {
                const float w0 = P[oW + i * kHid + lane], w1 = P[oW + i * kHid + lane + 32];
                const Samples<NS> u = x[i];
#pragma unroll
                for (int q = 0; q < NS; ++q) {
                    z0.v[q] = fmaf(u.v[q], w0, z0.v[q]);
                    z1.v[q] = fmaf(u.v[q], w1, z1.v[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                z0.v[q] = tanhf(z0.v[q]);
                z1.v[q] = tanhf(z1.v[q]);
            }
            out[lane] = z0;
            out[lane + 32] = z1;
            __syncwarp();
        };
        const int S = n - s < NS ? (int)(n - s) : NS;
        if (lane < kIn * NS) {
            const int q = lane / kIn, i = lane - q * kIn;
            b[i].v[q] = X[(s + (q < S ? q : S - 1)) * kIn + i];
        }
        __syncwarp();
        dense(b, kIn, kOffW1, kOffB1, a);
        dense(a, kHid, kOffW2, kOffB2, b);
        dense(b, kHid, kOffW3, kOffB3, a);
        if (lane < kOut * S) {
            const int q = lane / kOut, o = lane - q * kOut;
            float z = P[kOffB4 + o];
#pragma unroll 8
            for (int i = 0; i < kHid; ++i) z = fmaf(a[i].v[q], P[kOffW4 + i * kOut + o], z);
            Y[(s + q) * kOut + o] = z;
        }
        __syncwarp();
    }
}

static size_t grad_smem() {
    return sizeof(float) * ((size_t)2 * kHid * kWPitch + kIn * kHid + kHid * kOut + 3 * kHid + 4 +
                            (kIn + kOut + 6 * kHid) * kPitch);
}

}  // namespace fg

using namespace fg;

extern "C" int fftgal_mlp_nparams(void) { return kNParams; }

extern "C" int fftgal_mlp_grad(const float *params, const float *X, const float *T, long n, float *grad,
                               float *loss, void *stream) {
    if (!params || !X || !T || !grad || !loss || n < 1) return set_error(ERR_ARG, "fftgal_mlp_grad: bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t smem = grad_smem();
    FG_CUDA(cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    long nb = ceil_div(n, kMlpS);
    if (nb > 2L * num_sms()) nb = 2L * num_sms();
    mlp_grad_kernel<<<(unsigned)nb, kMlpThreads, smem, st>>>(params, X, T, n, 1.0f / (float)n, grad, loss,
                                                             reinterpret_cast<uintptr_t>(grad) % 16 == 0);
    FG_LAUNCHED(1);
    return OK;
}

extern "C" int fftgal_mlp_adam(float *params, const float *grad, float *m, float *v, int step, float lr,
                               void *stream) {
    if (!params || !grad || !m || !v || step < 1) return set_error(ERR_ARG, "fftgal_mlp_adam: bad arguments");
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    mlp_adam_kernel<<<(unsigned)ceil_div(kNParams, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        params, grad, m, v, lr, b1, b2, 1e-8f, c1, c2);
    FG_LAUNCHED(1);
    return OK;
}

extern "C" int fftgal_mlp_forward(const float *params, const float *X, long n, float *Y, void *stream) {
    if (!params || !X || !Y || n < 1) return set_error(ERR_ARG, "fftgal_mlp_forward: bad arguments");
    const long full = 4L * num_sms() * kFwdWarps;  // warps of a full grid
    const int ns = n >= 4 * full ? 4 : 1;
    long nb = ceil_div(n, kFwdWarps * ns);
    if (nb > 4L * num_sms()) nb = 4L * num_sms();
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (ns == 4)
        mlp_forward_kernel<4><<<(unsigned)nb, 32 * kFwdWarps, 0, st>>>(params, X, n, Y);
    else
        mlp_forward_kernel<1><<<(unsigned)nb, 32 * kFwdWarps, 0, st>>>(params, X, n, Y);
    FG_LAUNCHED(1);
    return OK;
}

extern "C" double fftgal_alias_envelope(double u) {
    const double u2 = u * u, u6 = u2 * u2 * u2;
    return u6 / (1.0 + u6);
}

extern "C" int fftgal_alias_features(int NK, const double *K, const double *P, double Pshot, double kNyq,
                                     float *X) {
    if (NK < 1 || !K || !P || !X || !(kNyq > 0)) return set_error(ERR_ARG, "fftgal_alias_features: bad arguments");
    std::vector<double> lden(NK), lk(NK);
    std::vector<char> ok(NK);
    for (int b = 0; b < NK; ++b) {
        const double den = fabs(P[4 * b]) + Pshot;
        ok[b] = std::isfinite(P[4 * b]) && std::isfinite(K[b]) && K[b] > 0 && den > 0;
        lden[b] = ok[b] ? log(den) : 0;
        lk[b] = ok[b] ? log(K[b]) : 0;
    }
    for (int b = 0; b < NK; ++b) {
        float *x = X + (size_t)kIn * b;
        if (!ok[b]) {
            for (int i = 0; i < kIn; ++i) x[i] = 0.f;
            continue;
        }
        const double den = fabs(P[4 * b]) + Pshot;
        int lo = b - 1, hi = b + 1;
        while (lo >= 0 && !ok[lo]) --lo;
        while (hi < NK && !ok[hi]) ++hi;
        if (lo < 0) lo = b;
        if (hi >= NK) hi = b;
        double slope = 0;
        if (hi != lo && lk[hi] != lk[lo]) slope = (lden[hi] - lden[lo]) / (lk[hi] - lk[lo]);
        slope = slope < -5 ? -5 : (slope > 5 ? 5 : slope);
        x[0] = (float)(K[b] / kNyq);
        x[1] = (float)(Pshot / den);
        x[2] = (float)(P[4 * b + 1] / den);
        x[3] = (float)(P[4 * b + 2] / den);
        x[4] = (float)slope;
    }
    return OK;
}
