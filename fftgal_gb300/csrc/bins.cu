// k-shell binning of the half spectrum for sm_103a: multipoles l = 0,2,4,6
// (src/power.c:30-101) and mu wedges (src/power.c:104-178) in one pass.
//
// Mode classification is exact with respect to the reference's FP64 code:
//  * the k bin iK = floor(sqrt(n2) * dKinv) depends only on the integer
//    n2 = kx^2 + ky^2 + kz^2, so the host evaluates the reference expression
//    once per n2 and ships the bin thresholds; the kernel finds iK from an FP32
//    estimate corrected against those exact thresholds;
//  * the wedge imu = floor(|mu * Nmu|) is estimated in FP32 and, only when the
//    estimate lies within its error bound of a wedge edge, re-evaluated in FP64
//    with the reference's operation order (explicitly rounded, no FMA).
// Mode counts N and the mean |k| per bin do not depend on the data: they are
// built once per (Ng, L, dK, los, Nmu) from an exact (n2, imu) multiplicity
// histogram and cached; every catalog then only accumulates power sums.
// Power sums: per-warp segmented reductions over runs of equal bins, FP32
// shared-memory accumulators flushed every chunk of rows into FP64 shared
// accumulators, FP64 global atomics once per CTA.
#include "internal.h"
#include "common.cuh"
#include "binmath.cuh"

#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <vector>

namespace fg {

constexpr double kSqrt3 = 1.73205080756887729352744634151;

int bin_spec_init(BinSpec *b, int Ng, double L, double dK, const double los_hat[3], int Nmu) {
    if (!(dK > 0) || !(L > 0)) return set_error(ERR_ARG, "dK and L must be > 0");
    if (Nmu < 1 || Nmu > 64) return set_error(ERR_ARG, "Nmu must be in [1, 64]");
    b->Ng = Ng;
    b->L = L;
    b->dK = dK;
    for (int a = 0; a < 3; ++a) b->los[a] = los_hat[a];
    b->Nmu = Nmu;
    b->KF = 2 * M_PI / L;
    b->dKinv = b->KF / dK;
    // src/power.c:34-36
    b->NK = (int)floor(kSqrt3 * (Ng / 2) * b->dKinv) + 1;
    if (b->NK < 1 || b->NK > (1 << 20)) return set_error(ERR_ARG, "NK = %d out of range", b->NK);
    return OK;
}

// ---- geometry: exact (n2, imu) multiplicities -----------------------------------------------
__global__ void geometry_kernel(BinDev d, uint32_t *__restrict__ hist) {
    const long n = (long)d.Ng * d.Ng * d.nh;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
        if (e == 0) continue;  // the k = 0 mode is skipped (src/power.c:52-54)
        const int k = (int)(e % d.nh);
        const long row = e / d.nh;
        const int j = (int)(row % d.Ng), i = (int)(row / d.Ng);
        const int ki = kval(i, d.Ng), kj = kval(j, d.Ng), kk = kval(k, d.Ng);
        const uint32_t n2 = (uint32_t)(ki * ki + kj * kj + kk * kk);
        const uint32_t count = 1 + ((2 * k) % d.Ng > 0);
        float mu2;
        const int imu = wedge_index(ki, kj, kk, sqrtf((float)n2), d, mu2);
        atomicAdd(&hist[(size_t)n2 * d.W + imu], count);
    }
}

void bin_geometry_free(BinGeometry *g) {
    delete[] g->N;
    delete[] g->K;
    delete[] g->Nw;
    delete[] g->Kw;
    cudaFree(g->d_thr);
    cudaFree(g->d_acc);
    *g = BinGeometry();
}

int bin_geometry_build(BinGeometry *g, const BinSpec &s, cudaStream_t st) {
    bin_geometry_free(g);
    g->spec = s;
    const int Ng = s.Ng, NK = s.NK, W = s.Nmu + 1;
    const int h = Ng / 2;
    const uint32_t n2max = (uint32_t)(3L * h * h);
    // exact k-bin thresholds from the reference expression floor(sqrt(n2) * dKinv)
    std::vector<uint32_t> thr(NK + 2, n2max + 1);
    std::vector<int> ik(n2max + 1);
    for (uint32_t n2 = 0; n2 <= n2max; ++n2) {
        volatile double kamp = sqrt((double)n2);
        volatile double t = kamp * s.dKinv;
        ik[n2] = (int)floor(t);
    }
    thr[0] = 0;
    {
        int b = 1;
        for (uint32_t n2 = 0; n2 <= n2max && b <= NK; ++n2)
            while (b <= NK && ik[n2] >= b) thr[b++] = n2;
    }
    FG_CUDA(cudaMalloc(&g->d_thr, sizeof(uint32_t) * (NK + 2)));
    FG_CUDA(cudaMemcpyAsync(g->d_thr, thr.data(), sizeof(uint32_t) * (NK + 2), cudaMemcpyHostToDevice, st));
    // multiplicity histogram over (n2, imu)
    const size_t hlen = (size_t)(n2max + 1) * W;
    uint32_t *d_hist = nullptr;
    FG_CUDA(cudaMalloc(&d_hist, sizeof(uint32_t) * hlen));
    FG_CUDA(cudaMemsetAsync(d_hist, 0, sizeof(uint32_t) * hlen, st));
    const BinDev d = make_dev(s);
    const long nmodes = (long)Ng * Ng * (h + 1);
    long nb = ceil_div(nmodes, 256);
    if (nb > 64L * num_sms()) nb = 64L * num_sms();
    geometry_kernel<<<(unsigned)nb, 256, 0, st>>>(d, d_hist);
    note_launches(1);
    cudaError_t e = cudaGetLastError();
    std::vector<uint32_t> hh(hlen);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hh.data(), d_hist, sizeof(uint32_t) * hlen, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_hist);
    if (e != cudaSuccess) return cuda_check(e, "geometry histogram");
    g->N = new long[NK]();
    g->K = new double[NK]();
    g->Nw = new long[(size_t)NK * W]();
    g->Kw = new double[(size_t)NK * W]();
    g->bad = 0;
    for (uint32_t n2 = 1; n2 <= n2max; ++n2) {
        const uint32_t *row = &hh[(size_t)n2 * W];
        long tot = 0;
        for (int m = 0; m < W; ++m) tot += row[m];
        if (!tot) continue;
        const int b = ik[n2];
        if (b < 0 || b >= NK) {
            g->bad = 1;
            continue;
        }
        const double kamp = sqrt((double)n2);
        g->N[b] += tot;
        g->K[b] += (double)tot * kamp;
        for (int m = 0; m < W; ++m)
            if (row[m]) {
                g->Nw[(size_t)b * W + m] += row[m];
                g->Kw[(size_t)b * W + m] += (double)row[m] * kamp;
            }
    }
    g->acc_len = (size_t)NK * (4 + W);
    FG_CUDA(cudaMalloc(&g->d_acc, sizeof(double) * g->acc_len));
    g->valid = true;
    return OK;
}

// ---- power sums ---------------------------------------------------------------------------------

constexpr int kBinThreads = 256;
constexpr int kChunkRows = 64;

// inclusive segmented sum over runs of equal `key` within the warp; returns
// true on the last lane of each run (which then owns the run's sum)
template <int NV>
__device__ __forceinline__ bool warp_segsum(int key, float (&v)[NV], int lane) {
    const unsigned full = 0xffffffffu;
    const int kprev = __shfl_up_sync(full, key, 1);
    const bool head = lane == 0 || kprev != key;
    const unsigned hm = __ballot_sync(full, head);
    const int seg = __popc(hm & (0xffffffffu >> (31 - lane)));
    if (hm != 1u) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int sseg = __shfl_up_sync(full, seg, o);
            float t[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) t[q] = __shfl_up_sync(full, v[q], o);
            if (lane >= o && sseg == seg) {
#pragma unroll
                for (int q = 0; q < NV; ++q) v[q] += t[q];
            }
        }
        const int snext = __shfl_down_sync(full, seg, 1);
        return lane == 31 || snext != seg;
    }
    // a single run: butterfly reduction, lane 31 owns the total
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] += __shfl_xor_sync(full, v[q], o);
    return lane == 31;
}

// One warp walks one k row (fixed i, j) at a time, 32 modes per step, so the
// k bin is non-decreasing along the step and the row constants are computed
// once.  The CTA advances through chunks of kChunkRows rows and folds its FP32
// partial sums into FP64 after each chunk.
template <typename T, int MODE>
__global__ void __launch_bounds__(kBinThreads)
bin_power_kernel(BinDev d, const T *__restrict__ f, T Vinv, T Pshot,
                 const uint32_t *__restrict__ thr_g, double *__restrict__ gacc, int Ng_pad) {
    using T2 = vec2_t<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int NK = d.NK, W = d.W, NQ = 4 + W;
    double *acc64 = reinterpret_cast<double *>(smem_raw);               // [NK * NQ]
    float *acc32 = reinterpret_cast<float *>(acc64 + (size_t)NK * NQ);  // [NK * NQ] (FP32 grids)
    uint32_t *thr = reinterpret_cast<uint32_t *>(acc32 + (sizeof(T) == 4 ? (size_t)NK * NQ : 0));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    for (int e = tid; e < NK * NQ; e += blockDim.x) {
        acc64[e] = 0;
        if constexpr (sizeof(T) == 4) acc32[e] = 0.f;
    }
    for (int e = tid; e < NK + 2; e += blockDim.x) thr[e] = thr_g[e];
    __syncthreads();

    const int Ng = d.Ng, nh = d.nh;
    const int nrows = Ng * Ng;
    const int nchunks = (nrows + kChunkRows - 1) / kChunkRows;
    for (int ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
        const int r1 = min(nrows, (ch + 1) * kChunkRows);
        for (int row = ch * kChunkRows + warp; row < r1; row += nwarp) {
            const int i = row / Ng, j = row - i * Ng;
            const int ki = kval(i, Ng), kj = kval(j, Ng);
            const int n2ij = ki * ki + kj * kj;
            const T *frow = f + (long)row * Ng_pad;
            for (int k0 = 0; k0 < nh; k0 += 32) {
                const int k = k0 + lane;
                int b = -1, imu = 0;
                T pc = 0, mu2t = 0;
                if (k < nh && (row | k) != 0) {
                    const int kk = kval(k, Ng);
                    const uint32_t n2 = (uint32_t)(n2ij + kk * kk);
                    const int count = 1 + ((2 * k) % Ng > 0);
                    T p;
                    if constexpr (MODE == 0) {
                        p = frow[2 * k];
                    } else {
                        const T2 v = reinterpret_cast<const T2 *>(frow)[k];
                        if constexpr (sizeof(T) == 8)
                            p = __dsub_rn(__dmul_rn(__dadd_rn(__dmul_rn(v.x, v.x), __dmul_rn(v.y, v.y)), Vinv), Pshot);
                        else
                            p = (v.x * v.x + v.y * v.y) * Vinv - Pshot;
                    }
                    pc = p * (T)count;
                    b = kbin(n2, thr, NK, d.dKinv_f);
                    if (b >= NK) b = -1;
                    float mu2f;
                    imu = wedge_index(ki, kj, kk, sqrtf((float)n2), d, mu2f);
                    if constexpr (sizeof(T) == 8) {
                        if (!d.zero_los) {
                            const double kamp = __dsqrt_rn((double)n2);
                            const double num = __dadd_rn(__dadd_rn(__dmul_rn((double)ki, d.l0), __dmul_rn((double)kj, d.l1)),
                                                         __dmul_rn((double)kk, d.l2));
                            const double mu = __ddiv_rn(num, kamp);
                            mu2t = __dmul_rn(mu, mu);
                        }
                    } else {
                        mu2t = mu2f;
                    }
                }
                if constexpr (sizeof(T) == 8) {
                    if (b >= 0) {
                        const double m2 = mu2t;
                        double *a = acc64 + (size_t)b * NQ;
                        atomicAdd(a + 0, pc);
                        atomicAdd(a + 1, pc * (1.5 * m2 - 0.5));
                        atomicAdd(a + 2, pc * ((4.375 * m2 - 3.75) * m2 + 0.375));
                        atomicAdd(a + 3, pc * (((14.4375 * m2 - 19.6875) * m2 + 6.5625) * m2 - 0.3125));
                        atomicAdd(a + 4 + imu, pc);
                    }
                } else {
                    const float m2 = mu2t;
                    float v[4] = {pc, pc * (1.5f * m2 - 0.5f), pc * ((4.375f * m2 - 3.75f) * m2 + 0.375f),
                                  pc * (((14.4375f * m2 - 19.6875f) * m2 + 6.5625f) * m2 - 0.3125f)};
                    if (warp_segsum<4>(b, v, lane) && b >= 0) {
                        float *a = acc32 + (size_t)b * NQ;
                        atomicAdd(a + 0, v[0]);
                        atomicAdd(a + 1, v[1]);
                        atomicAdd(a + 2, v[2]);
                        atomicAdd(a + 3, v[3]);
                    }
                    float w[1] = {pc};
                    const int wkey = b < 0 ? -1 : b * W + imu;
                    if (warp_segsum<1>(wkey, w, lane) && wkey >= 0) atomicAdd(acc32 + (size_t)b * NQ + 4 + imu, w[0]);
                }
            }
        }
        if constexpr (sizeof(T) == 4) {
            __syncthreads();
            for (int e = tid; e < NK * NQ; e += blockDim.x) {
                acc64[e] += (double)acc32[e];
                acc32[e] = 0.f;
            }
            __syncthreads();
        }
    }
    __syncthreads();
    for (int e = tid; e < NK * NQ; e += blockDim.x)
        if (acc64[e] != 0) atomicAdd(&gacc[e], acc64[e]);
}

// FP32 grids.  The half spectrum is cut into blocks of 16 (i) x 16 (j) x 32
// (k) modes.  Each warp of a CTA stages one 16 x 32 slab of the block (16
// rows of 32 consecutive k, from coalesced loads) as FP32 powers in shared
// memory, then walks the slab in runs of 16 modes along the grid axis whose
// |n_a| is smallest at the block's centre: along that axis |n| changes
// slowest, so a run crosses the fewest k-bin edges (about 0.3 per mode,
// against 0.55 along a fixed axis).  A thread keeps the run's sums in
// registers and adds them to the CTA's FP32 shared accumulators when the bin
// (or the wedge) changes; every `fold` blocks the CTA adds its FP32
// sums to the FP64 global accumulators.
//   MODE 0: the grid holds P in F_Re (after P()).
//   MODE 1: the grid holds delta; P = |delta|^2 Vinv - Pshot.
//   MODE 2: as 1, with the interlacing finish of the grid fused in: A <-
//           (A + B * phase) * W^-1 * scale is written back and binned.
//   MODE 3: as 2 without an interlacing grid: A <- A * W^-1 * scale (the
//           deconvolution of a single paint, src/fft.c:236-254).
//   MODE 4: as 3 with the deconvolved value binned but not written back.
//   MODE 5: as 2 with the finished value binned but not written back (the
//           fused calls under the lazy host view: 4.3 GB fewer writes at
//           Ng = 1024).
//
// Mirrored modes.  A mode's k bin, wedge and Legendre weights depend on n^2 and
// |n . los|, so modes that differ by the sign of n_i where los_i = 0 (or where
// los has no other component) share them exactly, and likewise for n_j; where
// only los_k = 0, (n_i, n_j) and (-n_i, -n_j) do.  The slabs then cover
// n_i >= 0 (n_j >= 0) only: a slab element sums the powers of its NP = 4 (lines
// of sight along an axis) or 2 (los with two components) mirrored modes, and the
// classification, which is most of a mode's instructions, is done once for
// them (slab_mirror; NP = 1 for other lines of sight).  Measured with their
// finish, interlaced: Ng = 1024, los z 4.51 -> 1.94 ms (8.6 GB read: 4.4 TB/s); Ng =
// 512 los z with ten wedges 594 -> 305 us, los (1, 1, 0) 590 -> 479 us; and with shorter
// slabs on small grids Ng = 128 45 -> 25 us, Ng = 64 54 -> 26 us.
constexpr int kSlabI = 16, kSlabJ = 16, kSlabK = 32, kSlabRow = 33;
constexpr int kSlabThreads = 512;  // one warp per slab of a block (fewer where there are few blocks)
// blocks between folds of the FP32 sums into FP64: FFTGAL_BIN_FOLD, default 8
static int fold_blocks() {
    static const int v = [] {
        const char *e = getenv("FFTGAL_BIN_FOLD");
        const int n = e ? atoi(e) : 0;
        return n >= 1 && n <= 1024 ? n : 8;
    }();
    return v;
}

struct SlabFinish {
    float2 *A = nullptr;
    const float2 *B = nullptr;
    const float2 *ph = nullptr;  // [3][Ng] phase of the interlacing grid (FP32)
    const float *w = nullptr;    // [Ng] PCS window inverse (FP32)
    float scale = 0.f;           // H^3 / 2
};

// which axes mirror, and the rows along i and j that the slabs cover
struct SlabMirror {
    bool fi = false, fj = false;  // n_i, n_j on their own
    bool joint = false;           // (n_i, n_j) together
    int NI = 0, NJ = 0;
    __host__ __device__ int modes() const { return fi && fj ? 4 : (fi || fj || joint ? 2 : 1); }
};

static SlabMirror slab_mirror(const BinSpec &s) {
    SlabMirror m;
    const bool z0 = s.los[0] == 0, z1 = s.los[1] == 0, z2 = s.los[2] == 0;
    const int nz = (z0 ? 0 : 1) + (z1 ? 0 : 1) + (z2 ? 0 : 1);
    m.fi = z0 || nz == 1;
    m.fj = z1 || nz == 1;
    m.joint = z2 && !m.fi && !m.fj;
    const int half = s.Ng / 2 + 1;
    m.NI = m.fi || m.joint ? half : s.Ng;
    m.NJ = m.fj ? half : s.Ng;
    return m;
}

// the kernels whose CTAs per SM a measured launch shape sets: it is measured on both
// interlacing grids with the line of sight along z, and the kernels of one grid, or of
// fewer mirrored modes, have an optimum of their own
static bool tuned_slab(int np, int mode) { return np == 4 && (mode == 2 || mode == 5); }

// The slab blocks cover k < kmain.  When the half spectrum's last k block
// would hold only one or two columns (nh = Ng/2 + 1: the Nyquist column of
// every even Ng that is a multiple of 32), those columns are binned mode by
// mode after the blocks instead, by all threads of the grid, rather than as
// 32-column blocks with one or two columns used (6 % of the lane slots at
// Ng = 1024).
__host__ __device__ __forceinline__ int slab_kmain(int nh) {
    const int r = nh % kSlabK;
    return (nh > kSlabK && r > 0 && r <= 2) ? nh - r : nh;
}

// A mode's value and its share of the slab element: |delta|^2 without the
// window and Vinv (MODE >= 2), |delta|^2 (MODE 1), P (MODE 0); p is the phase
// of element e, wk the window inverse (stored with the value by MODE 2 and 3)
struct ModeLoad {
    float2 a, b;
};
template <int MODE>
__device__ __forceinline__ ModeLoad mode_load(const SlabFinish &fin, const float2 *__restrict__ f, long e) {
    ModeLoad m;
    m.a = MODE == 2 || MODE == 3 ? fin.A[e] : f[e];  // these modes also write A
    m.b = MODE == 2 || MODE == 5 ? fin.B[e] : make_float2(0.f, 0.f);
    return m;
}
template <int MODE>
__device__ __forceinline__ float mode_value(const SlabFinish &fin, const ModeLoad &m, long e, float2 p, float wk,
                                            bool store) {
    if (MODE == 0) return m.a.x;
    float2 v = m.a;
    if (MODE == 2 || MODE == 5) {
        v.x += m.b.x * p.x - m.b.y * p.y;
        v.y += m.b.x * p.y + m.b.y * p.x;
    }
    if ((MODE == 2 || MODE == 3) && store) fin.A[e] = make_float2(v.x * wk, v.y * wk);
    return v.x * v.x + v.y * v.y;
}
// power of `count` modes whose mode_value()s sum to s
template <int MODE>
__device__ __forceinline__ float mode_power(float s, float count, float wk, float Vinv, float Pshot) {
    if (MODE == 0) return s;
    if (MODE == 1) return s * Vinv - count * Pshot;
    return (s * wk) * wk * Vinv - count * Pshot;
}

// One mode by itself, by one thread (the columns and rows beside the slabs)
template <int MODE>
__device__ __forceinline__ void bin_single(const BinDev &d, const SlabFinish &fin, const float2 *__restrict__ f,
                                           const uint32_t *thr, float *acc32, int i, int j, int k, float Vinv,
                                           float Pshot) {
    const int Ng = d.Ng;
    const long e = ((long)i * Ng + j) * d.nh + k;
    float2 p = make_float2(0.f, 0.f);
    float wk = 0.f;
    if (MODE == 2 || MODE == 5) p = cmul(cmul(fin.ph[Ng + j], fin.ph[2 * Ng + k]), fin.ph[i]);
    if (MODE >= 2) wk = fin.w[j] * fin.w[k] * fin.scale * fin.w[i];
    const float s = mode_value<MODE>(fin, mode_load<MODE>(fin, f, e), e, p, wk, true);
    BinRun run;
    run.add(d, thr, acc32, kval(i, Ng), kval(j, Ng), kval(k, Ng), k, mode_power<MODE>(s, 1.f, wk, Vinv, Pshot));
    run.finish(d, acc32);
}

// MINB: CTAs per SM the registers are budgeted for, chosen by the CTAs per SM
// that the launch's shared memory allows and the tuned launch shape.
// nr: rows of a slab and modes of a run, 16 or, on small grids, 8 or 4, so that
// a block makes 16 x 16 / nr slabs for as many warps (a warp takes 20 us or more
// for 16 rows, whatever the grid; the CTA's blockDim.x / 32 warps take as many
// slabs of a block per turn).  FULL: 16 rows and 16 warps, known to the compiler, for
// the one-mode slabs, whose row loop is most of their work.
template <int MODE, int NP, int MINB, bool FULL>
__global__ void __launch_bounds__(kSlabThreads, MINB)
bin_power_slab_kernel(BinDev d, const float2 *__restrict__ f, SlabFinish fin, SlabMirror mir, float Vinv, float Pshot,
                      const uint32_t *__restrict__ thr_g, double *__restrict__ gacc, const DevScalars *__restrict__ ds,
                      int fold, int nr_) {
    if (ds) {
        Vinv = ds->Vinv;
        Pshot = ds->Pshot;
    }
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int NK = d.NK, W = d.W, NQ = 4 + W;
    float *acc32 = reinterpret_cast<float *>(smem_raw);                        // [NQ][NK]
    uint32_t *thr = reinterpret_cast<uint32_t *>(acc32 + (size_t)NK * NQ);     // [NK + 2]
    float *slabs = reinterpret_cast<float *>(thr + ((NK + 2 + 3) & ~3));        // [warps][16][kSlabRow]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = FULL ? kSlabThreads / 32 : blockDim.x >> 5;
    const int nr = FULL ? kSlabJ : nr_;
    float *slab = slabs + warp * kSlabJ * kSlabRow;
    for (int e = tid; e < NK * NQ; e += blockDim.x) acc32[e] = 0.f;
    for (int e = tid; e < NK + 2; e += blockDim.x) thr[e] = thr_g[e];
    __syncthreads();
    const int Ng = d.Ng, nh = d.nh, kmain = slab_kmain(nh), NI = NP == 1 ? d.Ng : mir.NI, NJ = NP == 1 ? d.Ng : mir.NJ;
    const int nbi = (NI + kSlabI - 1) / kSlabI, nbj = (NJ + kSlabJ - 1) / kSlabJ, nbk = (kmain + kSlabK - 1) / kSlabK;
    const int nsub = kSlabI * (kSlabJ / nr) / nwarp;  // CTA turns per block
    const int nblk = nbi * nbj * nbk * nsub;
    const long si = (long)Ng * nh, sj = nh;  // element strides
    int since_fold = 0;
    for (int turn = blockIdx.x; turn < nblk; turn += gridDim.x) {
        const int blk = turn / nsub, sub = turn - blk * nsub;
        const int bk = blk % nbk, bj = (blk / nbk) % nbj, bi = blk / (nbk * nbj);
        const int i0 = bi * kSlabI, j0 = bj * kSlabJ, k0 = bk * kSlabK;
        const int ci = abs(kval(min(i0 + kSlabI / 2, NI - 1), Ng));
        const int cj = abs(kval(min(j0 + kSlabJ / 2, NJ - 1), Ng));
        const int ck = min(k0 + kSlabK / 2, nh - 1);
        const int axis = (ck <= ci && ck <= cj) ? 2 : (cj <= ci ? 1 : 0);  // run axis
        // the warp's slab: for runs along i it fixes j and its rows are i,
        // otherwise it fixes i and its rows are j
        const bool rows_i = axis == 0;
        const int unit = sub * nwarp + warp;
        const int fixed = (rows_i ? j0 : i0) + (unit & (kSlabI - 1));
        const int r0 = (rows_i ? i0 : j0) + unit / kSlabI * nr;
        const int nfix = rows_i ? NJ : NI, nrow = rows_i ? NI : NJ;
        const int k = k0 + lane;
        if (fixed < nfix) {
            // mirrored index along the rows (cr) and of the fixed axis (cf)
            const bool cr = NP == 4 || (NP == 2 && (mir.joint || (rows_i ? mir.fi : mir.fj)));
            const bool cf = NP == 4 || (NP == 2 && (mir.joint || (rows_i ? mir.fj : mir.fi)));
            const bool has_f = fixed > 0 && 2 * fixed != Ng;
            const int fm = fixed ? Ng - fixed : 0;
            float2 q0 = make_float2(0.f, 0.f), q1 = q0;
            float wfk = 0.f;
            if (MODE >= 2 && k < kmain) {
                if (MODE == 2 || MODE == 5) {
                    const float2 pf = fin.ph[(rows_i ? Ng : 0) + fixed], pk = fin.ph[2 * Ng + k];
                    q0 = cmul(pf, pk);
                    if (NP > 1) q1 = cf ? cmul(cconj(pf), pk) : q0;
                }
                wfk = fin.w[fixed] * fin.w[k] * fin.scale;
            }
            // the row tables of the slab's rows: lane r holds row r's, the
            // loop takes them by shuffle
            float2 phl = make_float2(0.f, 0.f);
            float wl = 0.f;
            if (MODE >= 2 && lane < nr && r0 + lane < nrow) {
                if (MODE == 2 || MODE == 5) phl = fin.ph[(rows_i ? 0 : Ng) + r0 + lane];
                wl = fin.w[r0 + lane];
            }
            const long rs = rows_i ? si : sj, fs = rows_i ? sj : si;
            const float2 *fk = f;
            const long eF = fixed * fs + k, eG = (cf ? fm : fixed) * fs + k;
            long en = r0 * rs + eF;
            // unrolled for 8 or 16 loads in flight, as far as the registers go
            constexpr int UNR = MINB >= 3 ? (NP == 1 ? 8 : 4 / NP) : (NP == 1 ? 8 : 8 / NP);
#pragma unroll UNR
            for (int r = 0; r < nr; ++r, en += rs) {
                float2 pr = make_float2(0.f, 0.f);
                float wr = 0.f;
                if (MODE == 2 || MODE == 5) {
                    pr.x = __shfl_sync(0xffffffffu, phl.x, r);
                    pr.y = __shfl_sync(0xffffffffu, phl.y, r);
                }
                if (MODE >= 2) wr = __shfl_sync(0xffffffffu, wl, r);
                float pv = 0.f;
                const int x = r0 + r;
                if (x < nrow && k < kmain) {
                    const float wk = wfk * wr;
                    const long e0 = NP == 1 ? en : x * rs + eF;
                    if (NP == 1) {
                        // one mode per element: with the same arithmetic as below, written as
                        // its own product, the compiler keeps eight pairs of loads in flight
                        // (los (1, 1, 1), Ng = 1024, interlaced 5.02 -> 4.48 ms, with FULL and
                        // the running index, which also take single paints from 4.15 to 3.77)
                        if (MODE == 2 || MODE == 5) {
                            const float2 p = cmul(q0, pr);
                            const float2 bv = fin.B[e0], av = fin.A[e0];
                            const float2 dv = cmul(bv, p);
                            const float2 v = make_float2((dv.x + av.x) * wk, (dv.y + av.y) * wk);
                            if (MODE == 2) fin.A[e0] = v;
                            pv = (v.x * v.x + v.y * v.y) * Vinv - Pshot;
                        } else {
                            const float s = mode_value<MODE>(fin, mode_load<MODE>(fin, fk, e0), e0, q0, wk, true);
                            pv = mode_power<MODE>(s, 1.f, wk, Vinv, Pshot);
                        }
                    } else {
                        const bool has_r = x > 0 && 2 * x != Ng;
                        const long xm = x ? Ng - x : 0;
                        const float2 pc = cconj(pr);
                        if (NP == 2) {
                            // one partner; jointly mirrored modes need both indices off the Nyquist
                            // row and n_i off 0
                            bool has = cr ? has_r : has_f;
                            if (mir.joint)
                                has = rows_i ? has_r && 2 * fixed != Ng : has_f && 2 * x != Ng;
                            const long e1 = has ? (cr ? xm : x) * rs + eG : e0;
                            const ModeLoad m0 = mode_load<MODE>(fin, fk, e0), m1 = mode_load<MODE>(fin, fk, e1);
                            float s = mode_value<MODE>(fin, m0, e0, cmul(q0, pr), wk, true);
                            const float t = mode_value<MODE>(fin, m1, e1, cmul(q1, cr ? pc : pr), wk, has);
                            s += has ? t : 0.f;
                            pv = mode_power<MODE>(s, has ? 2.f : 1.f, wk, Vinv, Pshot);
                        } else {
                            const long e1 = has_r ? xm * rs + eF : e0, e2 = has_f ? x * rs + eG : e0;
                            const long e3 = has_r && has_f ? xm * rs + eG : e0;
                            const ModeLoad m0 = mode_load<MODE>(fin, fk, e0), m1 = mode_load<MODE>(fin, fk, e1);
                            const ModeLoad m2 = mode_load<MODE>(fin, fk, e2), m3 = mode_load<MODE>(fin, fk, e3);
                            float s = mode_value<MODE>(fin, m0, e0, cmul(q0, pr), wk, true);
                            const float t1 = mode_value<MODE>(fin, m1, e1, cmul(q0, pc), wk, has_r);
                            const float t2 = mode_value<MODE>(fin, m2, e2, cmul(q1, pr), wk, has_f);
                            const float t3 = mode_value<MODE>(fin, m3, e3, cmul(q1, pc), wk, has_r && has_f);
                            s += has_r ? t1 : 0.f;
                            s += has_f ? t2 : 0.f;
                            s += has_r && has_f ? t3 : 0.f;
                            pv = mode_power<MODE>(s, (has_r ? 2.f : 1.f) * (has_f ? 2.f : 1.f), wk, Vinv, Pshot);
                        }
                    }
                }
                slab[r * kSlabRow + lane] = pv;
            }
        }
        __syncwarp();
        if (fixed < nfix) {
            // runs along k: lane = (row, stretch of nr of the 32 k); else lane = k
            if (axis == 2) {
                const int r = lane & (nr - 1), c = lane - r, rr = r0 + r, kc = k0 + c;
                const int n = rr < nrow ? min(nr, kmain - kc) : 0;
                bin_run<2>(d, thr, acc32, fixed, rr, kc, n, slab + r * kSlabRow + c, 1);
            } else {
                const int kc = k0 + lane;
                const int n = kc < kmain ? min(nr, nrow - r0) : 0;
                if (axis == 1)
                    bin_run<1>(d, thr, acc32, fixed, r0, kc, n, slab + lane, kSlabRow);
                else
                    bin_run<0>(d, thr, acc32, r0, fixed, kc, n, slab + lane, kSlabRow);
            }
        }
        __syncwarp();
        if (++since_fold == fold) {
            since_fold = 0;
            __syncthreads();
            bin_fold(acc32, gacc, NK, NQ);
            __syncthreads();
        }
    }
    // beside the slabs, one mode per thread (consecutive threads take consecutive
    // k and j): the columns k >= kmain, and, where (n_i, n_j) mirror together, the
    // modes (-n_i, Ng/2) whose partner's n_j = -Ng/2 keeps its sign
    const long step = (long)gridDim.x * blockDim.x, first = (long)blockIdx.x * blockDim.x + tid;
    if (kmain < nh) {
        const int ncol = nh - kmain;
        for (long m = first; m < (long)ncol * Ng * Ng; m += step) {
            const long ij = m / ncol;
            bin_single<MODE>(d, fin, f, thr, acc32, (int)(ij / Ng), (int)(ij % Ng), kmain + (int)(m % ncol), Vinv,
                             Pshot);
        }
    }
    if (NP == 2 && mir.joint && Ng % 2 == 0) {
        for (long m = first; m < (long)(Ng / 2 - 1) * kmain; m += step)
            bin_single<MODE>(d, fin, f, thr, acc32, Ng / 2 + 1 + (int)(m / kmain), Ng / 2, (int)(m % kmain), Vinv,
                             Pshot);
    }
    __syncthreads();
    for (int e = tid; e < NK * NQ; e += blockDim.x) {
        const float v = acc32[e];
        if (v != 0.f) {
            const int q = e / NK, b = e - q * NK;
            atomicAdd(&gacc[(size_t)b * NQ + q], (double)v);
        }
    }
}

static size_t slab_smem(int NK, int NQ, int warps = kSlabThreads / 32) {
    return sizeof(float) * (size_t)NK * NQ + sizeof(uint32_t) * (size_t)((NK + 2 + 3) & ~3) +
           sizeof(float) * warps * kSlabJ * kSlabRow;
}

// the launch of the slab kernel: mirrored modes, rows of a slab, warps of a CTA, slabs,
// CTAs per SM, shared memory
struct SlabShape {
    SlabMirror mir;
    int np = 1, nr = kSlabJ, warps = kSlabThreads / 32, per_sm = 1;
    long units = 0;
    size_t smem = 0;
};

static SlabShape slab_shape(const BinSpec &s, int mode) {
    SlabShape h;
    h.mir = slab_mirror(s);
    h.np = h.mir.modes();
    // small grids: shorter slabs until there are 16 warps' worth per SM, and
    // smaller CTAs until there are two per SM
    const long blocks = ceil_div(h.mir.NI, kSlabI) * ceil_div(h.mir.NJ, kSlabJ) *
                        ceil_div(slab_kmain(s.Ng / 2 + 1), kSlabK);
    // three CTAs per SM hide the loads best, except where four mirrored modes of
    // two grids want 16 loads in flight and the grid is large: two CTAs without
    // spills (interlaced, los along z: Ng = 1024 1.94 against 2.27 ms, 512 305 against
    // 348 us, 384 158 against 180, but 256 84 against 76, 128 28.7 against 24.6; two
    // mirrored modes at 512 524 against 479 us)
    const int most = tuned_slab(h.np, mode) && blocks * kSlabI >= 64L * num_sms() ? 2 : 3;
    auto fill = [&](int nr) {  // slabs of nr rows; returns the rows that a warp takes one after the other
        h.nr = nr;
        h.units = blocks * kSlabI * (kSlabJ / nr);
        h.warps = kSlabThreads / 32;
        while (h.warps > 4 && h.units / h.warps < 2L * num_sms()) h.warps /= 2;
        h.smem = slab_smem(s.NK, 4 + s.Nmu + 1, h.warps);
        const int per_sm = (int)((224 * 1024) / (h.smem + 1024));
        h.per_sm = per_sm < 1 ? 1 : (per_sm > most ? most : per_sm);
        return ceil_div(h.units / h.warps, (long)num_sms() * h.per_sm) * nr;
    };
    int nr = kSlabJ;
    while (nr > 4 && blocks * kSlabI * (kSlabJ / nr) < 16L * num_sms()) nr /= 2;
    // with few rounds of CTAs a last one of few takes as long as a full one: shorter
    // slabs where that leaves an eighth fewer rows to do one after the other (interlaced,
    // los (1, 1, 1): Ng = 144 61 -> 39 us; (1, 1, 0): 192 76 -> 53; z: 240 100 -> 55.
    // With more rounds the shorter slabs' own cost counts: (1, 1, 1), 448 455 against 399)
    long rows = fill(nr);
    if (rows <= 3 * nr)
        for (long r; nr > 4 && 8 * (r = fill(nr / 2)) <= 7 * rows; rows = r) nr /= 2;
    fill(nr);
    return h;
}

int bin_cta_builtin(const BinSpec &s, int mode) { return slab_shape(s, mode).per_sm; }

static int bin_launch(BinGeometry *g, const void *f, int prec, int mode, double Vinv, double Pshot, cudaStream_t st,
                      const BinFinish *fin, const DevScalars *ds);

void bin_power_unpack(const BinGeometry *g, const double *h, double *Psum, double *Pw) {
    const int NK = g->spec.NK, W = g->spec.Nmu + 1, NQ = 4 + W;
    for (int b = 0; b < NK; ++b) {
        for (int l = 0; l < 4; ++l) Psum[b * 4 + l] = h[(size_t)b * NQ + l];
        for (int m = 0; m < W; ++m) Pw[(size_t)b * W + m] = h[(size_t)b * NQ + 4 + m];
    }
}

int bin_power_launch(BinGeometry *g, int mode, double Vinv, double Pshot, cudaStream_t st, const BinFinish *fin,
                     const DevScalars *ds) {
    if (mode < 2 || mode > 5) return set_error(ERR_ARG, "bin_power_launch: modes 2 to 5 only");
    return bin_launch(g, nullptr, 4, mode, Vinv, Pshot, st, fin, ds);
}

int bin_power(BinGeometry *g, const void *f, int prec, int mode, double Vinv, double Pshot,
              double *Psum, double *Pw, cudaStream_t st, cudaEvent_t *ev_end, const BinFinish *fin) {
    FG_TRY(bin_launch(g, f, prec, mode, Vinv, Pshot, st, fin, nullptr));
    if (ev_end) FG_CUDA(cudaEventRecord(*ev_end, st));
    std::vector<double> h(g->acc_len);
    FG_CUDA(cudaMemcpyAsync(h.data(), g->d_acc, sizeof(double) * g->acc_len, cudaMemcpyDeviceToHost, st));
    FG_CUDA(cudaStreamSynchronize(st));
    bin_power_unpack(g, h.data(), Psum, Pw);
    return OK;
}

static int bin_launch(BinGeometry *g, const void *f, int prec, int mode, double Vinv, double Pshot, cudaStream_t st,
                      const BinFinish *fin, const DevScalars *ds) {
    if (!g->valid) return set_error(ERR_STATE, "bin geometry not built");
    if (mode >= 2 && (prec != 4 || !fin)) return set_error(ERR_ARG, "fused finish needs an FP32 grid");
    const BinSpec &s = g->spec;
    const BinDev d = make_dev(s);
    const int NK = s.NK, W = s.Nmu + 1, NQ = 4 + W;
    size_t smem = prec == 4 ? slab_smem(NK, NQ) : (size_t)NK * NQ * 8 + sizeof(uint32_t) * (NK + 2);
    if (smem > 220 * 1024)
        return set_error(ERR_UNSUPPORTED, "binning: %d k bins x %d wedges exceed shared memory", NK, s.Nmu);
    FG_CUDA(cudaMemsetAsync(g->d_acc, 0, sizeof(double) * g->acc_len, st));
    if (prec == 4) {
        const SlabShape h = slab_shape(s, mode);
        const SlabMirror mir = h.mir;
        const int np = h.np, nr = h.nr, warps = h.warps;
        smem = h.smem;
        int per_sm = h.per_sm;
        if (tuned_slab(np, mode) && g->cta_per_sm > 0 && g->cta_per_sm < per_sm) per_sm = g->cta_per_sm;
        const long nturn = h.units / warps;
        const bool full = nr == kSlabJ && warps == kSlabThreads / 32;
        long nb = (long)num_sms() * per_sm;
        if (nb > nturn) nb = nturn;
        SlabFinish sf;
        if (fin) {
            sf.A = static_cast<float2 *>(fin->A);
            sf.B = static_cast<const float2 *>(fin->B);
            sf.ph = static_cast<const float2 *>(fin->ph32);
            sf.w = static_cast<const float *>(fin->w32);
            sf.scale = (float)fin->scale;
        }
        const float2 *fv = static_cast<const float2 *>(mode >= 2 ? fin->A : f);
#define FG_SLAB_LAUNCH3(M, N, B, F)                                                                          \
    do {                                                                                                    \
        FG_CUDA(cudaFuncSetAttribute(bin_power_slab_kernel<M, N, B, F>,                                      \
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));               \
        bin_power_slab_kernel<M, N, B, F><<<(unsigned)nb, 32 * warps, smem, st>>>(                              \
            d, fv, sf, mir, (float)Vinv, (float)Pshot, g->d_thr, g->d_acc, ds,                               \
            g->fold > 0 ? g->fold : fold_blocks(), nr);                                                      \
    } while (0)
#define FG_SLAB_LAUNCH2(M, B)                \
    do {                                     \
        if (np == 4)                         \
            FG_SLAB_LAUNCH3(M, 4, B, false); \
        else if (np == 2)                    \
            FG_SLAB_LAUNCH3(M, 2, B, false); \
        else if (full)                       \
            FG_SLAB_LAUNCH3(M, 1, B, true);  \
        else                                 \
            FG_SLAB_LAUNCH3(M, 1, B, false); \
    } while (0)
#define FG_SLAB_LAUNCH(M)             \
    do {                              \
        if (per_sm >= 3)              \
            FG_SLAB_LAUNCH2(M, 3);    \
        else                          \
            FG_SLAB_LAUNCH2(M, 2);    \
    } while (0)
        if (mode == 0)
            FG_SLAB_LAUNCH(0);
        else if (mode == 1)
            FG_SLAB_LAUNCH(1);
        else if (mode == 2)
            FG_SLAB_LAUNCH(2);
        else if (mode == 3)
            FG_SLAB_LAUNCH(3);
        else if (mode == 4)
            FG_SLAB_LAUNCH(4);
        else
            FG_SLAB_LAUNCH(5);
#undef FG_SLAB_LAUNCH3
#undef FG_SLAB_LAUNCH2
#undef FG_SLAB_LAUNCH
    } else {
        const int Ng_pad = 2 * (s.Ng / 2 + 1);
        const long nchunks = ceil_div((long)s.Ng * s.Ng, kChunkRows);
        int per_sm = (int)((220 * 1024) / smem);
        per_sm = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
        long nb = (long)num_sms() * per_sm;
        if (nb > nchunks) nb = nchunks;
#define FG_BIN_LAUNCH(M)                                                                                     \
    do {                                                                                                     \
        FG_CUDA(cudaFuncSetAttribute(bin_power_kernel<double, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     (int)smem));                                                            \
        bin_power_kernel<double, M><<<(unsigned)nb, kBinThreads, smem, st>>>(                                \
            d, (const double *)f, Vinv, Pshot, g->d_thr, g->d_acc, Ng_pad);                                  \
    } while (0)
        if (mode == 0)
            FG_BIN_LAUNCH(0);
        else
            FG_BIN_LAUNCH(1);
#undef FG_BIN_LAUNCH
    }
    FG_LAUNCHED(1);
    return OK;
}

}  // namespace fg
