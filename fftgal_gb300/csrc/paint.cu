// PCS (piecewise cubic spline) mass assignment for sm_103a.
//
// Restates the arithmetic of the reference's fft_p2g (src/fft.c:57-131):
// u = x * Ng/L - offset, base cell floor(u), fraction d = u - floor(u), the four
// cubic B-spline weights of src/fft.c:83-88, cells wrapped mod Ng.  The GPU
// organisation is new:
//
//  1. count   : every particle gets the key (tile, class) of its base cell.  The
//               grid is cut into tiles of at most 32 x 16 x 32 cells (i, j, k;
//               FP32 grids with Ng >= 64), 16 x 16 x 32 (smaller FP32 grids) or
//               8 x 8 x 16 (FP64 grids, whose key is the tile alone); per axis
//               the class says whether the particle's stencil (over all painted
//               grids) reaches into the lower (1) or upper (2) neighbour tile, or
//               neither (0).  Only the key histogram is
//               written (fire-and-forget atomics).
//  2. scan    : exclusive prefix sum of the key histogram, written to a cursor
//               array too.
//  3. scatter : the key is formed again and each particle's record is written
//               at the slot its key's cursor atomic returns.  The order within
//               a key depends on the atomics' order; the FP32 paint sums in
//               fixed point, so the painted grid does not.
//  4. paint   : FP32 grids: one CTA per tile owns its cells.  It pulls the particles
//               of its own tile and only the boundary classes of its 26 neighbours,
//               accumulates their weights in shared memory and writes every
//               owned cell exactly once (no global atomics, no zeroing pass).
//               FP64 grids: the grid is zeroed, and a warp adds the weights of its
//               tile's own particles, halo included, with global atomics.
//
// FP32 grids with Ng >= 64 (paint_rot_kernel, persistent over tiles of
// 32 x 16 x 32 cells, two 512-thread CTAs per SM): one thread deposits one
// particle, each lane of a warp visiting its particle's 64 cells in an order that
// puts the warp's 32 atomics of every step in 32 distinct banks.  The two
// interlacing grids are painted by separate CTAs, one grid each, from one sort.
// Both grids of 1e8 particles at Ng = 1024: 6.67 ms, against 10.67 ms of a warp
// that staged 32 particles' weights in shared memory and deposited two
// particles per step, lane = (particle, i row, j row).
// Smaller FP32 grids (paint_coop_kernel, 16 x 16 x 32 tiles, one or both grids per
// CTA, tiles that may span the periodic box) keep that staged deposit: each lane
// prepares one particle (cell indices and the 3 x 4 weights of one grid) in
// shared memory, then the warp deposits the particles one (two grids) or two
// (one grid) at a time, each lane adding its 4 k cells.
// Sums are 32-bit fixed point with a
// per-tile scale 2^-s, s the largest value for which no cell can exceed 2^32 (a
// particle adds at most (2/3)^3 of its weight to a cell): the tile's particle
// total bounds every cell, and only where that bound leaves fewer than 21
// fraction bits does a first pass count particles per 4^3-cell block.  A tile
// whose bound still leaves fewer than 16 bits (a dense clump: more than about
// 2e5 particles near one cell) paints one grid at a time into 64-bit sums
// with 22 fraction bits over the same shared memory, since at 12-15 bits the
// many tiny products at a stencil's edge round to zero and bias the edge cells
// low by several percent.  Integer sums are order independent, so the painted
// grid is bit-reproducible run to run.
// FP64 grids (paint_warp_f64_kernel) reproduce the reference's FP64 weight
// arithmetic op for op and accumulate in FP64: a warp owns a tile's cells and their
// halo in shared memory and adds them to the zeroed grid.
#include "internal.h"
#include "common.cuh"

#include <math.h>
#include <string.h>
#include <vector>

namespace fg {

constexpr int kTileExt[3] = {16, 16, 32};    // i, j, k
constexpr int kTileExt1[3] = {32, 16, 32};   // FP32 grids with Ng >= 64
constexpr int kMaxPaintGrids = 2;
// dense tiles (fewer 32-bit fraction bits than kWideBelow): 64-bit sums with
// kWideBits fraction bits, one grid per pass.  At 16-19 bits the 32-bit sums
// round the tiny products at a dense clump's stencil edge by up to 1.4 % of
// those cells' values (1e-6 of the clump's peak cell, 1e-5 of its mass); the
// clustered 1e8-galaxy lognormal mock has many such tiles, whose tile paint
// the 64-bit passes took from 13.0 to 15.8 ms (Ng = 1024) at a threshold of 20
constexpr int kWideBelow = 16;
constexpr int kWideBits = 22;
// FP32 shared layout: cell (li, lj, lk) of grid g at g*kGS + li*kSI + lj*kSJ +
// kPadK + lk.  kSI = 8 and kSJ = 6 (mod 32) put the 16 rows (li+a, lj+b), a, b
// < 4, of one stencil in 16 distinct banks of one parity, and the odd kGS gives
// the other grid the other parity: with each lane of the second grid taking
// its 4 k cells in the order s ^ ((b1 - b0) & 1) (its stencil is shifted by
// b1 - b0 cells along k), every one of the 4 atomic steps of a particle touches
// 32 distinct banks.  kPadK columns on either side of a row take the stencil
// cells beyond the tile along k, so a particle's 4 k cells are always
// contiguous; stencil rows outside the tile in i or j (local index kOut) are
// skipped.
constexpr int kPadK = 3;
constexpr int kSJ = 38, kSI = 616, kGS = 9849;
constexpr uint32_t kOut = 255u;
static_assert(15 * kSI + 15 * kSJ + kSJ <= kGS, "tile does not fit the layout");
static_assert(32 + 2 * kPadK <= kSJ, "row padding");
static_assert(kSI % 32 == 8 && kSJ % 32 == 6 && kGS % 2 == 1, "bank layout");
// two grids of 16 i rows, or a dense tile's 64-bit sums of one
constexpr int kAccWords = 2 * kGS > 2 * 16 * kSI ? 2 * kGS : 2 * 16 * kSI;
constexpr size_t kAccBytes = (sizeof(uint32_t) * kAccWords + 15) / 16 * 16;
// largest fixed-point scale: products stay below 2^22 so the FMA trick of
// deposit4 converts them to integers exactly
constexpr int kMaxFixBits = 23;
// the per-block count that can raise a dense tile's scale runs only when its
// particle total leaves fewer bits than this (tiles of more than about 6900
// particles): at >= 21 fraction bits a deposit rounds by at most 2^-22 of a
// unit weight, inside FP32 grid accuracy even where the deconvolution
// amplifies the noise of the corner bins, so the extra pass over the tile's
// records (most of 1 ms of the tile paint for a 1e8-galaxy lognormal mock at
// Ng=1024) is skipped for moderately dense tiles
constexpr int kBlockCountBelow = 21;
// per-tile block counts: 4^3-cell blocks over the tile plus a 4-cell margin
constexpr int kBlk = 4;
__host__ __device__ constexpr int blk_dim(int a) { return a == 1 ? (16 + 8) / kBlk : (32 + 8) / kBlk; }  // 10, 6, 10
constexpr int kBlkN = blk_dim(0) * blk_dim(1) * blk_dim(2);

struct AxisParams {
    // FP32 path: x * h - o as double-float (h = Ng/L, o = offset of grid g)
    float h_hi, h_lo;
    float o_hi[kMaxPaintGrids], o_lo[kMaxPaintGrids];
    // FP32 path: u_g = u_0 + delta_g, delta_g = o_0 - o_g in units of 2^-fb
    int dq[kMaxPaintGrids];
    // FP64 path
    double h;
    double o[kMaxPaintGrids];
};

struct PaintParams {
    AxisParams ax[3];
    // FP32 redshift-space displacement (v[0] null: none)
    const float *v[3];
    float los[3], aHinv;
    int Ng, Ng_pad, ngrids;
    int fb;                  // FP32 path: fraction bits of the packed cell coordinate
    int nt[3], tmax[3];      // tiles per axis, and their largest extents
    const int *tile_of[3];   // [Ng] per axis
    int tshift[3];           // log2 of the tile extent when every tile of the axis has it, else -1
    const int *start[3];     // [nt + 1] per axis
};

// ---- redshift-space displacement ---------------------------------------------
// x + ((los . v) / aH) los, the operation order of src/gal.c:69-72 in FP32 with
// explicit FMAs, so the key and scatter kernels displace a particle identically
__device__ __forceinline__ void rsd_displace(const PaintParams &pp, long p, float pos[3]) {
    if (!pp.v[0]) return;
    const float vd = fmaf(pp.los[2], pp.v[2][p], fmaf(pp.los[1], pp.v[1][p], pp.los[0] * pp.v[0][p]));
    const float s = pp.aHinv * vd;
#pragma unroll
    for (int a = 0; a < 3; ++a) pos[a] = fmaf(s, pp.los[a], pos[a]);
}
__device__ __forceinline__ void rsd_displace(const PaintParams &, long, double *) {}

// ---- per-axis cell coordinate ----------------------------------------------

__device__ __forceinline__ void coord(float x, const AxisParams &a, int g, int Ng, int &b, float &d) {
    // u = x*h - o with the rounding errors of the product and the subtraction
    // carried in a second float, then split into floor and fraction
    const float p = x * a.h_hi;
    const float pe = fmaf(x, a.h_hi, -p) + x * a.h_lo;
    const float s = p - a.o_hi[g];
    const float bv = s - p;
    const float se = (p - (s - bv)) + (-a.o_hi[g] - bv);
    const float lo = (pe + se) - a.o_lo[g];
    const float fb = floorf(s);
    float fr = (s - fb) + lo;
    int ib = (int)fb;
    if (fr < 0.f) {
        fr += 1.f;
        ib -= 1;
    } else if (fr >= 1.f) {
        fr -= 1.f;
        ib += 1;
    }
    ib %= Ng;
    if (ib < 0) ib += Ng;
    b = ib;
    d = fr;
}

__device__ __forceinline__ void coord(double x, const AxisParams &a, int g, int Ng, int &b, double &d) {
    // src/fft.c:68-82, evaluated without contraction so it rounds like the host
    const double u = __dsub_rn(__dmul_rn(x, a.h), a.o[g]);
    const int g1 = (int)floor(u);
    d = __dsub_rn(u, (double)g1);
    b = (g1 % Ng + Ng) % Ng;
}

// (explicit operations: every kernel rounds the weights alike; s = 1/6 times a
// power of two, which scales the weights exactly)
__device__ __forceinline__ void pcs_weights(float d, float w[4], float s = 1.f / 6.f) {
    const float e = __fsub_rn(1.f, d), d2 = __fmul_rn(d, d);
    w[0] = __fmul_rn(__fmul_rn(__fmul_rn(e, e), e), s);
    w[1] = __fmul_rn(__fmaf_rn(__fmaf_rn(3.f, d, -6.f), d2, 4.f), s);
    w[2] = __fmul_rn(__fmaf_rn(__fmaf_rn(__fmaf_rn(-3.f, d, 3.f), d, 3.f), d, 1.f), s);
    w[3] = __fmul_rn(__fmul_rn(d2, d), s);
}

// x / 6 rounded to nearest: with r = RN(1/6) and q = RN(x r) within an ulp of x / 6,
// RN(q + (x - 6 q) r) is the correctly rounded quotient (Markstein 1990); the
// weights' numerators (0 .. 6, or below by roundings of 0) never make it
// underflow.  Three operations of the FP64 pipe, which does two lanes per cycle
// and SM.
__device__ __forceinline__ double sixth(double x) {
    const double r = 1.0 / 6.0;
    const double q = __dmul_rn(x, r);
    return __fma_rn(__fma_rn(-6.0, q, x), r, q);
}

__device__ __forceinline__ void pcs_weights(double d, double w[4]) {
    // src/fft.c:83-88 in the reference's operation order, no FMA contraction
    const double e = __dsub_rn(1.0, d);
    const double d2 = __dmul_rn(d, d);
    w[0] = sixth(__dmul_rn(__dmul_rn(e, e), e));
    w[1] = sixth(__dadd_rn(__dmul_rn(__dsub_rn(__dmul_rn(3.0, d), 6.0), d2), 4.0));
    w[2] = sixth(
        __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(-3.0, d), 3.0), d), 3.0), d), 1.0));
    w[3] = sixth(__dmul_rn(d2, d));
}

// FP32 path: the grid-0 base cell b0 and the fraction as fb-bit fixed point;
// every other grid's cell is derived from these with an exact integer shift,
// identically in the key and the paint kernels.
__device__ __forceinline__ void cell0(float x, const AxisParams &a, int Ng, int fb, int &b0, uint32_t &dq) {
    float d;
    coord(x, a, 0, Ng, b0, d);
    const uint32_t one = 1u << fb;
    dq = (uint32_t)(d * (float)one);
    dq = dq >= one ? one - 1 : dq;
}

__device__ __forceinline__ void cell_g(int b0, uint32_t dq, int delta, int fb, int Ng, int &bg, uint32_t &dgq) {
    const int t = (int)dq + delta;  // |delta| <= 2^fb
    dgq = (uint32_t)t & ((1u << fb) - 1);
    bg = b0 + (t >> fb);            // arithmetic shift: floor division
    bg += bg < 0 ? Ng : 0;
    bg -= bg >= Ng ? Ng : 0;
}

// local index of stencil cell s (0..3) of base cell b: (b - 1 + s) mod Ng
// relative to the tile start t0, or -1 outside [0, te)
__device__ __forceinline__ int local_cell(int b, int s, int Ng, int t0, int te) {
    int c = b - 1 + s;
    c = c < 0 ? c + Ng : (c >= Ng ? c - Ng : c);
    const int l = c - t0;
    return (l >= 0 && l < te) ? l : -1;
}

template <typename P> struct Rec;
template <> struct Rec<float> { using type = uint4; };  // per axis (b0 << fb) | fraction
template <> struct Rec<double> { struct type { double x, y, z; }; };

// ---- 1. key + histogram -------------------------------------------------------

// the key of a particle; for FP32 positions also its packed record words
// (b0 << fb) | fraction per axis
template <typename P>
__device__ __forceinline__ uint32_t paint_key_of(const P pos[3], const PaintParams &pp, uint32_t *rec = nullptr) {
    const int Ng = pp.Ng;
    int t[3], cls[3] = {0, 0, 0};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int b0;
        uint32_t dq0 = 0;
        if constexpr (sizeof(P) == 4) {
            cell0(pos[a], pp.ax[a], Ng, pp.fb, b0, dq0);
            if (rec) rec[a] = ((uint32_t)b0 << pp.fb) | dq0;
        } else {
            P d;
            coord(pos[a], pp.ax[a], 0, Ng, b0, d);
        }
        int ta, t0, te;
        if (pp.tshift[a] >= 0) {
            ta = b0 >> pp.tshift[a];
            t0 = ta << pp.tshift[a];
            te = 1 << pp.tshift[a];
        } else {
            ta = pp.tile_of[a][b0];
            t0 = pp.start[a][ta];
            te = pp.start[a][ta + 1] - t0;
        }
        t[a] = ta;
        if constexpr (sizeof(P) == 8) continue;  // the FP64 paint goes by the tile alone
        int rmin = b0 - t0, rmax = b0 - t0;
        for (int g = 1; g < pp.ngrids; ++g) {
            int bg;
            uint32_t dgq;
            cell_g(b0, dq0, pp.ax[a].dq[g], pp.fb, Ng, bg, dgq);
            int dl = bg - b0;  // -1, 0 or +1 after undoing a wrap
            dl -= dl > 1 ? Ng : 0;
            dl += dl < -1 ? Ng : 0;
            rmin = min(rmin, b0 - t0 + dl);
            rmax = max(rmax, b0 - t0 + dl);
        }
        cls[a] = pp.nt[a] == 1 ? 0 : (rmin - 1 < 0 ? 1 : (rmax + 2 >= te ? 2 : 0));
    }
    const long tile = ((long)t[0] * pp.nt[1] + t[1]) * pp.nt[2] + t[2];
    if constexpr (sizeof(P) == 8) return (uint32_t)tile;
    return (uint32_t)(tile * 27 + cls[0] * 9 + cls[1] * 3 + cls[2]);
}

template <typename P>
__global__ void paint_key_kernel(const P *__restrict__ x, const P *__restrict__ y,
                                 const P *__restrict__ z, long Np, PaintParams pp,
                                 uint32_t *__restrict__ hist, const DevScalars *__restrict__ ds) {
    if (ds) Np = ds->Np;
    for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < Np; p += (long)gridDim.x * blockDim.x) {
        P pos[3] = {x[p], y[p], z[p]};
        rsd_displace(pp, p, pos);
        atomicAdd(&hist[paint_key_of<P>(pos, pp)], 1u);
    }
}

// Few keys (small grids): thousands of particles share a key, and atomics on one
// address come one after another (1e6 particles, Ng = 128, 3456 keys: 35 us, their
// 12 bytes per particle taking 2 us).  A CTA then counts in shared memory and
// adds its nonzero counts.  (Ranking chunks of 2048 particles in shared memory for
// the scatter as well was slower there: 51 against 37 us, Ng = 64 27 against 16.)
constexpr long kFewKeys = 8192;
template <typename P>
__global__ void __launch_bounds__(256)
paint_key_few_kernel(const P *__restrict__ x, const P *__restrict__ y, const P *__restrict__ z, long Np,
                     PaintParams pp, uint32_t *__restrict__ hist, int nkeys, const DevScalars *__restrict__ ds) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t *h = reinterpret_cast<uint32_t *>(smem_raw);  // [nkeys]
    if (ds) Np = ds->Np;
    for (int e = threadIdx.x; e < nkeys; e += blockDim.x) h[e] = 0u;
    __syncthreads();
    for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < Np; p += (long)gridDim.x * blockDim.x) {
        P pos[3] = {x[p], y[p], z[p]};
        rsd_displace(pp, p, pos);
        atomicAdd(&h[paint_key_of<P>(pos, pp)], 1u);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nkeys; e += blockDim.x)
        if (h[e]) atomicAdd(&hist[e], h[e]);
}

// ---- 2. exclusive scan of the histogram (in place, n + 1 entries) ------------------
// The offsets are written to a second array too: the scatter's cursors.

constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr int kScanBlock = kScanThreads * kScanPer;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *warp_sums, uint32_t *total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) warp_sums[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        uint32_t ws = lane < nw ? warp_sums[lane] : 0;
        uint32_t wi = ws;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += u;
        }
        if (lane < nw) warp_sums[lane] = wi - ws;
        if (lane == 31) *total = wi;
    }
    __syncthreads();
    const uint32_t r = warp_sums[wid] + inc - v;
    __syncthreads();
    return r;
}

__global__ void scan_block_sums(const uint32_t *__restrict__ a, long n, uint32_t *__restrict__ bsum) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t tot;
    const long base = (long)blockIdx.x * kScanBlock + threadIdx.x * kScanPer;
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanPer; ++i)
        if (base + i < n) s += a[base + i];
    block_exclusive_scan(s, ws, &tot);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

// a block adds up the sums of the blocks before it itself: a launch less than a scan
// of the sums in between (Ng = 256, 27649 entries: 13 us against 17; one CTA for all of
// them, as for short arrays, 24)
__global__ void scan_apply(uint32_t *__restrict__ a, uint32_t *__restrict__ cursor, long n,
                           const uint32_t *__restrict__ bsum) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t tot;
    const long base = (long)blockIdx.x * kScanBlock + threadIdx.x * kScanPer;
    uint32_t v[kScanPer];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
        v[i] = base + i < n ? a[base + i] : 0;
        s += v[i];
    }
    uint32_t before = 0;
    for (unsigned i = threadIdx.x; i < blockIdx.x; i += blockDim.x) before += bsum[i];
    block_exclusive_scan(before, ws, &tot);
    before = tot;
    uint32_t e = before + block_exclusive_scan(s, ws, &tot);
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) {
        if (base + i < n) a[base + i] = cursor[base + i] = e;
        e += v[i];
    }
}

// short arrays: one CTA runs through them in one launch
constexpr long kScanOne = 4L * kScanBlock;
__global__ void __launch_bounds__(kScanThreads)
scan_one(uint32_t *__restrict__ a, uint32_t *__restrict__ cursor, int n) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t tot;
    uint32_t carry = 0;
    for (int c0 = 0; c0 < n; c0 += kScanBlock) {
        const int base = c0 + threadIdx.x * kScanPer;
        uint32_t v[kScanPer], s = 0;
#pragma unroll
        for (int i = 0; i < kScanPer; ++i) {
            v[i] = base + i < n ? a[base + i] : 0;
            s += v[i];
        }
        uint32_t e = carry + block_exclusive_scan(s, ws, &tot);
        carry += tot;
#pragma unroll
        for (int i = 0; i < kScanPer; ++i) {
            if (base + i < n) a[base + i] = cursor[base + i] = e;
            e += v[i];
        }
        __syncthreads();  // tot is rewritten by the next stretch
    }
}

static int exclusive_scan(uint32_t *a, uint32_t *cursor, long n, uint32_t *bsum, cudaStream_t st) {
    if (n <= kScanOne) {
        scan_one<<<1, kScanThreads, 0, st>>>(a, cursor, (int)n);
        FG_LAUNCHED(1);
        return OK;
    }
    const long nb = ceil_div(n, kScanBlock);
    scan_block_sums<<<(unsigned)nb, kScanThreads, 0, st>>>(a, n, bsum);
    scan_apply<<<(unsigned)nb, kScanThreads, 0, st>>>(a, cursor, n, bsum);
    FG_LAUNCHED(2);
    return OK;
}

// ---- 3. scatter into key order ------------------------------------------------------

// the record of a displaced particle, and its key
template <typename P>
__device__ __forceinline__ uint32_t paint_record(const P pos[3], const PaintParams &pp, typename Rec<P>::type &r) {
    if constexpr (sizeof(P) == 4) {
        uint32_t w[3];
        const uint32_t k = paint_key_of<P>(pos, pp, w);
        r = make_uint4(w[0], w[1], w[2], 0u);
        return k;
    } else {
        r.x = pos[0];
        r.y = pos[1];
        r.z = pos[2];
        return paint_key_of<P>(pos, pp);
    }
}

template <typename P>
__global__ void paint_scatter_kernel(const P *__restrict__ x, const P *__restrict__ y,
                                     const P *__restrict__ z, long Np, PaintParams pp,
                                     uint32_t *__restrict__ cursor,
                                     typename Rec<P>::type *__restrict__ sorted,
                                     const DevScalars *__restrict__ ds) {
    if (ds) Np = ds->Np;
    for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < Np; p += (long)gridDim.x * blockDim.x) {
        P pos[3] = {x[p], y[p], z[p]};
        rsd_displace(pp, p, pos);
        typename Rec<P>::type r;
        const uint32_t k = paint_record<P>(pos, pp, r);
        sorted[atomicAdd(&cursor[k], 1u)] = r;
    }
}

// ---- 4. tile paint ---------------------------------------------------------------------

constexpr int kPaintThreads = 512;
constexpr int kStageParts = 16;  // particles staged per warp and round
constexpr int kMaxSeg = 125;

struct PaintOut {
    void *out[kMaxPaintGrids];
    double scale[kMaxPaintGrids];
    int accumulate[kMaxPaintGrids];
    const DevScalars *ds;  // if set, the scales are ds->scale
};

// Tile geometry and the flattened list of particle segments a tile pulls:
// its own key range for every class and the boundary classes of the (up to
// 26, deduplicated for 1 or 2 tiles per axis) neighbours.
struct TileSegs {
    int t0[3], te[3];
    int nseg;
    uint32_t total;
};

__device__ void tile_geometry(const PaintParams &pp, unsigned tile, TileSegs &ts) {
    const int nt1 = pp.nt[1], nt2 = pp.nt[2];
    const int tt[3] = {(int)(tile / (nt1 * nt2)), (int)((tile / nt2) % nt1), (int)(tile % nt2)};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        ts.t0[a] = pp.start[a][tt[a]];
        ts.te[a] = pp.start[a][tt[a] + 1] - ts.t0[a];
    }
}

// thread q's segment of `tile` (q < the returned count): first sorted index b
// and length cnt.  Issued a tile ahead so the loads overlap the write-out.
__device__ int tile_segment(const PaintParams &pp, const uint32_t *__restrict__ off, unsigned tile, int q,
                            uint32_t &b, uint32_t &cnt) {
    const int nt1 = pp.nt[1], nt2 = pp.nt[2];
    const int tt[3] = {(int)(tile / (nt1 * nt2)), (int)((tile / nt2) % nt1), (int)(tile % nt2)};
    // per axis the options (tile, class): the own tile with every class, then
    // the lower neighbour's particles reaching up (class 2) and the upper
    // neighbour's reaching down (class 1); both from the same tile when nt = 2
    int nopt[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) nopt[a] = pp.nt[a] == 1 ? 1 : 5;
    const int ncomb = nopt[0] * nopt[1] * nopt[2];  // <= 125
    b = 0;
    cnt = 0;
    if (q < ncomb) {
        const int idx[3] = {q / (nopt[1] * nopt[2]), (q / nopt[2]) % nopt[1], q % nopt[2]};
        int ot[3], oc[3];
        bool own = true;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int nt = pp.nt[a], x = idx[a];
            if (x < 3) {
                ot[a] = tt[a];
                oc[a] = nt == 1 ? 0 : x;
            } else {
                own = false;
                const int lo = (tt[a] + nt - 1) % nt, hi = (tt[a] + 1) % nt;
                if (nt == 2) {
                    ot[a] = hi;
                    oc[a] = x == 3 ? 1 : 2;
                } else {
                    ot[a] = x == 3 ? lo : hi;
                    oc[a] = x == 3 ? 2 : 1;
                }
            }
        }
        const long key = (((long)ot[0] * nt1 + ot[1]) * nt2 + ot[2]) * 27 + oc[0] * 9 + oc[1] * 3 + oc[2];
        if (!own) {
            b = off[key];
            cnt = off[key + 1] - b;
        } else if (q == 0) {  // every class of the own tile: 27 adjacent keys, one segment
            b = off[key];
            cnt = off[key + 27] - b;
        }
    }
    return ncomb;
}

// publish the fetched segments in shared memory (every thread takes part)
__device__ void tile_publish(int ncomb, uint32_t b, uint32_t cnt, uint32_t *seg_begin, uint32_t *seg_pref,
                             uint32_t *scan_ws, TileSegs &ts) {
    const int q = threadIdx.x;
    const uint32_t pref = block_exclusive_scan(cnt, scan_ws, &scan_ws[32]);  // scan_ws[33]
    const uint32_t tot = scan_ws[32];
    if (q < ncomb) {
        seg_begin[q] = b;
        seg_pref[q] = pref;
    }
    if (q == 0) seg_pref[ncomb] = tot;
    __syncthreads();
    ts.nseg = ncomb;
    ts.total = tot;
}

// index of particle q of the flattened segment list (largest segment whose
// prefix is <= q; empty segments are skipped automatically)
__device__ __forceinline__ uint32_t seg_index(uint32_t q, const uint32_t *seg_begin, const uint32_t *seg_pref,
                                              int nseg) {
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (seg_pref[mid] <= q) lo = mid;
        else hi = mid - 1;
    }
    return seg_begin[lo] + (q - seg_pref[lo]);
}

// per warp: the staged particles of one round, slot = particle + 16 * grid
struct __align__(16) StageBuf {
    uint4 loc[32];     // per axis: 4 packed local cell indices (255 = outside the tile); .w unused
    float4 w[3][32];   // per axis: PCS weights (k weights pre-scaled by 2^s)
};

__device__ __forceinline__ uint32_t pack_local(int b, int Ng, int t0, int te, uint32_t outv) {
    uint32_t r = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        int cs = b - 1 + s;  // in [-1, Ng + 2): one correction each way (Ng >= 2)
        cs += cs < 0 ? Ng : 0;
        cs -= cs >= Ng ? Ng : 0;
        const int l = cs - t0;
        r |= ((unsigned)l < (unsigned)te ? (uint32_t)l : outv) << (8 * s);
    }
    return r;
}

// deposit staged particles: lane = (grid, i row, j row), or (particle parity,
// i row, j row) when one grid is painted; every lane adds its row's 4 k
// cells.  By the bank layout each of the 4 atomic steps is a single
// shared-memory wavefront (two grids).  The loop is unrolled so that the
// shared loads of the next particles overlap the atomics of the current one.
// Stencil cells outside the tile (local index kOut) are skipped.
// slot of particle p of grid g in the stage buffer: the two grids' records
// interleave so that lanes reading both fall in different banks
__device__ __forceinline__ int stage_slot(int p, int g) { return 2 * p + g; }

// add round(w * wz) to the cell at offset `off`: 32-bit sums, or 64-bit sums
// (WIDE, offsets counted in 64-bit cells); w * wz < 2^22
template <bool WIDE>
__device__ __forceinline__ void dep_one(uint32_t *acc, int off, float w, float wz) {
    const float M = 12582912.0f;  // 1.5 * 2^23: FMA onto it rounds w * wz to an integer
    const uint32_t q = __float_as_uint(fmaf(w, wz, M)) - 0x4B400000u;
    if (WIDE)
        atomicAdd(reinterpret_cast<unsigned long long *>(acc) + off, (unsigned long long)q);
    else
        atomicAdd(acc + off, q);
}

// One particle of grid g for lane (a, b).
// FAST (no tile spans a periodic axis): loc.x / loc.y are the offsets of the
// particle's cells s ^ par for s = 0 and 1 in the stencil row (a, b) = (0, 0),
// relative to the accumulator, with par the cell-order bit; row (a, b) adds
// a*kSI + b*kSJ (lane_off).  loc.z has bit 4a + b set for the rows inside the
// tile.  The 4 k cells are contiguous (kPadK columns take those beyond the tile).
// Otherwise loc.x / loc.y hold the 4 local i / j indices as bytes (kOut outside
// the tile) and loc.z the 4 padded k cells as bytes, in step order.
// The k weights are stored in step order.
template <bool WIDE, bool FAST>
__device__ __forceinline__ void deposit_one(uint32_t *acc, const StageBuf &sb, int slot, int g, int a, int b,
                                            int lane_off) {
    const uint4 loc = sb.loc[slot];
    const float w = reinterpret_cast<const float *>(&sb.w[0][slot])[a] *
                    reinterpret_cast<const float *>(&sb.w[1][slot])[b];
    const float4 wz = sb.w[2][slot];
    if (FAST) {
        if (!((loc.z >> (4 * a + b)) & 1u)) return;  // a stencil row outside the tile
        const int o0 = (int)loc.x + lane_off, o1 = (int)loc.y + lane_off;
        dep_one<WIDE>(acc, o0, w, wz.x);
        dep_one<WIDE>(acc, o1, w, wz.y);
        dep_one<WIDE>(acc, o0 + 2, w, wz.z);
        dep_one<WIDE>(acc, o1 + 2, w, wz.w);
    } else {
        const uint32_t li = (loc.x >> (8 * a)) & 255u;
        const uint32_t lj = (loc.y >> (8 * b)) & 255u;
        if ((li | lj) >= 32u) return;  // kOut: a stencil row outside the tile
        const int row = g * kGS + (int)(li * kSI + lj * kSJ);
        dep_one<WIDE>(acc, row + (int)(loc.z & 255u), w, wz.x);
        dep_one<WIDE>(acc, row + (int)((loc.z >> 8) & 255u), w, wz.y);
        dep_one<WIDE>(acc, row + (int)((loc.z >> 16) & 255u), w, wz.z);
        dep_one<WIDE>(acc, row + (int)(loc.z >> 24), w, wz.w);
    }
}

template <bool WIDE, bool FAST>
__device__ __forceinline__ void deposit_all(uint32_t *acc, const StageBuf &sb, int np, int ngr, int lane) {
    const int h = lane >> 4, a = (lane >> 2) & 3, b = lane & 3;
    const int lane_off = a * kSI + b * kSJ;
    if (ngr > 1) {
#pragma unroll 4
        for (int p = 0; p < np; ++p) deposit_one<WIDE, FAST>(acc, sb, stage_slot(p, h), h, a, b, lane_off);
    } else {
        // one grid: 32 particles staged in slots 0..31, the half warps
        // deposit alternate ones; unrolled fully, so that the shared loads of
        // later particles are issued among the atomics of earlier ones
#pragma unroll 16
        for (int p = h; p < np; p += 2) deposit_one<WIDE, FAST>(acc, sb, p, 0, a, b, lane_off);
    }
}

// largest fixed-point exponent s <= kMaxFixBits for which `n` contributors to
// one cell cannot overflow its 32-bit sum: each adds round(w 2^s) <= 8/27 2^s +
// 1/2 (the largest PCS weight product is (2/3)^3), so n (16 2^s + 28) <= 54 2^32
// suffices; -1 if none.  Exact integer arithmetic; a result below kWideBelow
// selects the 64-bit sums.
__device__ __forceinline__ int fix_bits_for(uint32_t n) {
    int s = kMaxFixBits;
    while (s >= 0 && (unsigned long long)n * ((16u << s) + 28u) > (54ull << 32)) --s;
    return s;
}

// Fixed-point exponent of a tile of `total` particles.  The total bounds
// every cell's contributor count; only when that bound leaves fewer than
// kBlockCountBelow bits are the particles counted per 4^3 block of grid-0 base
// cells (over the tile plus a 4-cell margin, or the whole periodic axis when
// one tile spans it).  index(q) is the sorted index of the tile's q-th
// particle; blk (kBlkN words) and tmp (kBlkN words) are scratch.  Every thread
// of the CTA takes part.
template <typename Index>
__device__ __forceinline__ int tile_fixbits(uint32_t total, const uint4 *__restrict__ sorted, Index index,
                                            const PaintParams &pp, const TileSegs &ts, const bool *cyc, uint32_t *blk,
                                            uint32_t *tmp, uint32_t *scan_ws, int *fixbits_s) {
    const int fixbits = fix_bits_for(total);
    if (fixbits >= kBlockCountBelow) return fixbits;
    const int Ng = pp.Ng, fb = pp.fb, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nwarp = (int)blockDim.x / 32;
    int nb[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) nb[a] = cyc[a] ? (Ng + kBlk - 1) / kBlk : blk_dim(a);
    for (int e = tid; e < kBlkN; e += blockDim.x) blk[e] = 0u;
    __syncthreads();
    for (uint32_t q = tid; q < total; q += blockDim.x) {
        const uint4 r = sorted[index(q)];
        const uint32_t rw[3] = {r.x, r.y, r.z};
        int bidx = 0;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int b = (int)(rw[a] >> fb);
            int bb;
            if (cyc[a]) {
                bb = b / kBlk;
            } else {
                // a tile's particles have their base cells at -3 .. te + 1 (te <= Ng - 6), and
                // images are folded there as record_axis does: with two tiles along an
                // axis te and te + 1 are half a box away or more
                int l = b - ts.t0[a];
                l += l < -4 ? Ng : 0;
                l -= l >= Ng - 4 ? Ng : 0;
                bb = (l + 4) / kBlk;  // margin of 4 cells below the tile
                bb = bb < 0 ? 0 : (bb >= nb[a] ? nb[a] - 1 : bb);
            }
            bidx = bidx * blk_dim(a) + bb;
        }
        atomicAdd(&blk[bidx], 1u);
    }
    __syncthreads();
    // A cell's contributors have grid-0 base cells from 3 below to 3
    // above it per axis, within 3 consecutive blocks (cyclically on a
    // periodic axis): the largest 3x3x3 block sum bounds every cell's
    // contributor count.  Separable window sums along k, j, i.
    const int D1 = blk_dim(1), D2 = blk_dim(2);
    for (int e = tid; e < kBlkN; e += blockDim.x) {
        const int k = e % D2, j = (e / D2) % D1, i = e / (D2 * D1);
        uint32_t v = 0;
        const bool in = i < nb[0] && j < nb[1] && k < nb[2] && (cyc[2] || k + 2 < nb[2]);
        if (in)
            for (int c = 0; c < 3; ++c) v += blk[(i * D1 + j) * D2 + (cyc[2] ? (k + c) % nb[2] : k + c)];
        tmp[e] = v;
    }
    __syncthreads();
    for (int e = tid; e < kBlkN; e += blockDim.x) {
        const int k = e % D2, j = (e / D2) % D1, i = e / (D2 * D1);
        uint32_t v = 0;
        const bool in = i < nb[0] && j < nb[1] && k < nb[2] && (cyc[1] || j + 2 < nb[1]);
        if (in)
            for (int c = 0; c < 3; ++c) v += tmp[(i * D1 + (cyc[1] ? (j + c) % nb[1] : j + c)) * D2 + k];
        blk[e] = v;
    }
    __syncthreads();
    uint32_t mx = 0;
    for (int e = tid; e < kBlkN; e += blockDim.x) {
        const int k = e % D2, j = (e / D2) % D1, i = e / (D2 * D1);
        const bool in = i < nb[0] && j < nb[1] && k < nb[2] && (cyc[0] || i + 2 < nb[0]);
        if (in) {
            uint32_t v = 0;
            for (int c = 0; c < 3; ++c) v += blk[((cyc[0] ? (i + c) % nb[0] : i + c) * D1 + j) * D2 + k];
            mx = max(mx, v);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) scan_ws[warp] = mx;
    __syncthreads();
    if (tid == 0) {
        uint32_t m = 0;
        for (int w = 0; w < nwarp; ++w) m = max(m, scan_ws[w]);
        *fixbits_s = fix_bits_for(m);
    }
    __syncthreads();
    const int bits = *fixbits_s;
    return bits;
}

// Pass B over the tile's records: each warp stages 16 particles for both
// grids (NGS = 2: lanes 0..15 grid 0, 16..31 grid 1) or 32 particles of grid
// g1 (NGS = 1), then deposits them, into 32-bit sums or (WIDE) the 64-bit sums
// of grid g1; the records of the warp's next batch are loaded before the
// deposit so their latency hides behind it
template <int NGS, bool WIDE>
__device__ __forceinline__ void paint_records(uint32_t *acc, StageBuf &sb, const uint4 *__restrict__ sorted,
                                              const uint32_t *seg_begin, const uint32_t *seg_pref,
                                              const TileSegs &ts, const PaintParams &pp, const bool *cyc,
                                              bool fast, float fscale, int g1, const uint32_t (*loctab)[40],
                                              const uint32_t (*masktab)[40], int lane, int warp) {
    const int Ng = pp.Ng, fb = pp.fb, nseg = ts.nseg;
    const uint32_t total = ts.total;
    constexpr int nwarp = kPaintThreads / 32;
    const int parts = NGS > 1 ? kStageParts : 2 * kStageParts;  // particles per warp and round
    const int gs = NGS > 1 ? lane / kStageParts : g1;             // the grid this lane stages
    const int gofs = (WIDE || NGS == 1) ? 0 : gs * kGS;           // and its accumulator
    const float inv = __int_as_float((127 - fb) << 23);            // 2^-fb (fb <= 24)
    const uint32_t bstride = (uint32_t)nwarp * parts;
    uint32_t base = (uint32_t)warp * parts;
    uint4 rec = make_uint4(0, 0, 0, 0);
    {
        const uint32_t q = base + (lane & (parts - 1));
        if (q < total) rec = sorted[seg_index(q, seg_begin, seg_pref, nseg)];
    }
    for (; base < total; base += bstride) {
        const uint32_t q = base + (lane & (parts - 1));
        const bool valid = q < total;
        const int slot = NGS > 1 ? stage_slot(lane & (kStageParts - 1), gs) : lane;
        int bgv[3] = {0, 0, 0}, lv[3] = {0, 0, 0};
        uint32_t par = 0;
        float4 wk = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid) {
            const uint32_t rw[3] = {rec.x, rec.y, rec.z};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const int b0 = (int)(rw[a] >> fb);
                int bg;
                uint32_t dgq;
                cell_g(b0, rw[a] & ((1u << fb) - 1), pp.ax[a].dq[gs], fb, Ng, bg, dgq);
                float w[4];
                pcs_weights((float)dgq * inv, w);
                if (a == 2) {
                    wk = make_float4(w[0] * fscale, w[1] * fscale, w[2] * fscale, w[3] * fscale);
                    par = (uint32_t)(bg - b0) & 1u;
                } else {
                    sb.w[a][slot] = make_float4(w[0], w[1], w[2], w[3]);
                }
                // local index of the first stencil cell (periodic images
                // folded to the nearest copy of the tile)
                int l = bg - 1 - ts.t0[a];
                l -= l > Ng / 2 ? Ng : 0;
                l += l < -Ng / 2 ? Ng : 0;
                bgv[a] = bg;
                lv[a] = l;
            }
        }
        if (NGS == 1) {
            // one grid: the half warps deposit particles 2m and 2m + 1 together.
            // A first cell's bank parity is that of lv[2] + kPadK (the row
            // offsets kSI, kSJ are even), so particle 2m + 1 takes its k cells in
            // the order s ^ par that puts the pair's cells of every step in banks
            // of opposite parity, 16 distinct banks each: one wavefront per step
            const int other = __shfl_xor_sync(0xffffffffu, lv[2], 1);
            par = (lane & 1) ? (uint32_t)(((lv[2] ^ other) & 1) ^ 1) : 0u;
        }
        if (valid) {
            if (par) wk = make_float4(wk.y, wk.x, wk.w, wk.z);  // k cells in the order s ^ 1
            sb.w[2][slot] = wk;
            const bool kmiss = !cyc[2] && (lv[2] < -3 || lv[2] >= ts.te[2]);  // stencil misses the tile
            uint4 loc;
            if (fast) {
                const uint32_t mi = (unsigned)(lv[0] + 4) < 40u ? masktab[0][lv[0] + 4] : 0u;
                const uint32_t mj = (unsigned)(lv[1] + 4) < 40u ? masktab[1][lv[1] + 4] : 0u;
                const int b0 = gofs + lv[0] * kSI + lv[1] * kSJ + lv[2] + kPadK + (int)par;
                loc = make_uint4((uint32_t)b0, (uint32_t)(b0 + 1 - 2 * (int)par), kmiss ? 0u : mi * mj, 0u);
            } else {
                uint32_t li, lj, lk;
                li = cyc[0] ? pack_local(bgv[0], Ng, ts.t0[0], ts.te[0], kOut)
                            : ((unsigned)(lv[0] + 4) < 40u ? loctab[0][lv[0] + 4] : 0xFFFFFFFFu);
                lj = cyc[1] ? pack_local(bgv[1], Ng, ts.t0[1], ts.te[1], kOut)
                            : ((unsigned)(lv[1] + 4) < 40u ? loctab[1][lv[1] + 4] : 0xFFFFFFFFu);
                if (cyc[2])
                    lk = pack_local(bgv[2], Ng, ts.t0[2], ts.te[2], 0u) + 0x01010101u * kPadK;
                else
                    lk = (uint32_t)(kmiss ? 0 : lv[2] + kPadK) * 0x01010101u + 0x03020100u;
                if (par) lk = ((lk & 0x00FF00FFu) << 8) | ((lk >> 8) & 0x00FF00FFu);
                loc = make_uint4(kmiss ? 0xFFFFFFFFu : li, lj, lk, 0u);
            }
            sb.loc[slot] = loc;
        }
        __syncwarp();
        {
            const uint32_t qn = base + bstride + (lane & (parts - 1));
            if (qn < total) rec = sorted[seg_index(qn, seg_begin, seg_pref, nseg)];
        }
        const int np = min((uint32_t)parts, total - base);
        if (fast)
            deposit_all<WIDE, true>(acc, sb, np, NGS, lane);
        else
            deposit_all<WIDE, false>(acc, sb, np, NGS, lane);
        __syncwarp();
    }
}

// Persistent: each CTA paints tiles blockIdx.x, blockIdx.x + gridDim.x, ...
// The next tile's segment offsets are loaded during the write-out, the
// accumulators are cleared as they are written out, and each warp loads its
// next batch of records before depositing the current one.
// NGR = pp.ngrids (1 or 2), a template parameter so that the staging and
// deposit loops are specialised for one grid or the interlaced pair.
template <int NGR>
__global__ void __launch_bounds__(kPaintThreads, 2)
paint_coop_kernel(PaintParams pp, const uint32_t *__restrict__ off, const uint4 *__restrict__ sorted,
                  PaintOut po, unsigned ntiles) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t *acc = reinterpret_cast<uint32_t *>(smem_raw);                 // [2][kGS]
    StageBuf *stage = reinterpret_cast<StageBuf *>(smem_raw + kAccBytes);  // [warps]
    // the per-block counts and their window sums (before pass B) use the stage area
    uint32_t *blk = reinterpret_cast<uint32_t *>(stage) + kBlkN;  // [kBlkN]
    static_assert(2 * kBlkN * sizeof(uint32_t) <= sizeof(StageBuf) * (kPaintThreads / 32), "block counts");
    __shared__ uint32_t seg_begin[kMaxSeg];
    __shared__ uint32_t seg_pref[kMaxSeg + 1];
    __shared__ uint32_t scan_ws[33];
    __shared__ int fixbits_s;
    // packed local indices of the 4 stencil cells along i and j for a first
    // cell at l = -4 .. 35 relative to the tile start (kOut outside the tile);
    // they depend only on the tile extent, so they are rebuilt only when it changes
    __shared__ uint32_t loctab[2][40];
    // and as row masks: bit a (one bit per nibble for i, for the product with
    // the j mask) set when stencil row a lies inside the tile
    __shared__ uint32_t masktab[2][40];
    int tab_te0 = -1, tab_te1 = -1;
    // rebuild the tables for tile extents te0 x te1 (if they changed)
    auto build_tabs = [&](int te0, int te1) {
        if (te0 == tab_te0 && te1 == tab_te1) return;
        __syncthreads();
        if (threadIdx.x < 80) {
            const int a = threadIdx.x / 40, l = threadIdx.x % 40 - 4, te = a == 0 ? te0 : te1;
            uint32_t v = 0, m = 0;
#pragma unroll
            for (int s4 = 0; s4 < 4; ++s4) {
                const bool in = (unsigned)(l + s4) < (unsigned)te;
                v |= (in ? (uint32_t)(l + s4) : kOut) << (8 * s4);
                m |= (in ? 1u : 0u) << (a == 0 ? 4 * s4 : s4);
            }
            loctab[a][l + 4] = v;
            masktab[a][l + 4] = m;
        }
        __syncthreads();
        tab_te0 = te0;
        tab_te1 = te1;
    };

    const int Ng = pp.Ng, ngr = NGR;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = kPaintThreads / 32;  // launched with kPaintThreads
    unsigned tile = blockIdx.x;
    if (tile >= ntiles) return;
    for (int e = tid; e < (int)(kAccBytes / 16); e += kPaintThreads)
        reinterpret_cast<uint4 *>(smem_raw)[e] = make_uint4(0, 0, 0, 0);
    TileSegs ts;
    {
        uint32_t b, cnt;
        const int ncomb = tile_segment(pp, off, tile, tid, b, cnt);
        tile_publish(ncomb, b, cnt, seg_begin, seg_pref, scan_ws, ts);  // also orders the clearing above
    }
    for (;;) {
        tile_geometry(pp, tile, ts);
        const uint32_t total = ts.total;
        const int nseg = ts.nseg;
        bool cyc[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) cyc[a] = ts.te[a] == Ng;
        build_tabs(ts.te[0], ts.te[1]);

        const int fixbits = tile_fixbits(
            total, sorted, [&](uint32_t q) { return seg_index(q, seg_begin, seg_pref, nseg); }, pp, ts, cyc, blk,
            reinterpret_cast<uint32_t *>(stage), scan_ws, &fixbits_s);
        // a dense tile paints one grid per pass into 64-bit sums; otherwise one
        // pass paints every grid into 32-bit sums
        const bool wide = fixbits < kWideBelow;
        const int npass = wide ? ngr : 1;
        const float fscale = ldexpf(1.0f, wide ? kWideBits : fixbits);
        if (wide) {
            // the 32-bit tiles leave sums in the row padding: clear all of it
            __syncthreads();
            for (int e = tid; e < (int)(kAccBytes / 16); e += kPaintThreads)
                reinterpret_cast<uint4 *>(smem_raw)[e] = make_uint4(0, 0, 0, 0);
            __syncthreads();
        }
        const bool fast = !(cyc[0] || cyc[1] || cyc[2]);
        const unsigned next = tile + gridDim.x;
        uint32_t nb_begin = 0, nb_cnt = 0;
        int nb_comb = 0;
        for (int pass = 0; pass < npass; ++pass) {
            const int pg = pass;  // the grid of a wide pass
            if (wide)
                paint_records<1, true>(acc, stage[warp], sorted, seg_begin, seg_pref, ts, pp, cyc, fast, fscale, pg,
                                       loctab, masktab, lane, warp);
            else
                paint_records<NGR, false>(acc, stage[warp], sorted, seg_begin, seg_pref, ts, pp, cyc, fast, fscale, 0,
                                          loctab, masktab, lane, warp);
            __syncthreads();

            // the next tile's segments, loaded now and published after the write-out
            if (pass == npass - 1 && next < ntiles) nb_comb = tile_segment(pp, off, next, tid, nb_begin, nb_cnt);

            // write the owned cells (and the row padding of the last k tile),
            // clearing them for the next tile: warp w writes the i rows w, w + 16,
            // ..., stepping along j with pointer increments; lanes along k
            {
                const bool last_k = (ts.t0[2] + ts.te[2] == Ng);
                const int rowlen = ts.te[2] + (last_k ? pp.Ng_pad - Ng : 0);
                const int te1 = ts.te[1], te2 = ts.te[2];
                const long rstride = (long)pp.Ng_pad;  // global floats between consecutive j
                const long istride = rstride * Ng;     // and between consecutive i
                const double s0 = po.ds ? po.ds->scale[0] : po.scale[0], s1 = po.ds ? po.ds->scale[1] : po.scale[1];
                const long obase = ((long)ts.t0[0] * Ng + ts.t0[1]) * rstride + ts.t0[2];
                if (wide) {
                    // grid pg's rows of this pass from the 64-bit sums, then clear them all
                    const double scd = ldexp(pg == 0 ? s0 : s1, -kWideBits);
                    const float scf = (float)scd;
                    const int accu = po.accumulate[pg];
                    const unsigned long long *acc64 = reinterpret_cast<const unsigned long long *>(acc);
                    for (int li = warp; li < ts.te[0]; li += nwarp) {
                        float *o = reinterpret_cast<float *>(po.out[pg]) + obase + li * istride;
                        const unsigned long long *a = acc64 + kPadK + li * kSI;
                        for (int lj = 0; lj < te1; ++lj, o += rstride, a += kSJ) {
                            float v = 0.f * scf;
                            if (lane < te2) v = (float)((double)a[lane] * scd);
                            if (lane < rowlen) {
                                if (!accu) o[lane] = v;
                                else if (lane < te2) o[lane] += v;
                            }
                            if (lane + 32 < rowlen && !accu) o[lane + 32] = 0.f * scf;
                        }
                    }
                    __syncthreads();
                    for (int e = tid; e < (int)(kAccBytes / 16); e += kPaintThreads)
                        reinterpret_cast<uint4 *>(smem_raw)[e] = make_uint4(0, 0, 0, 0);
                    __syncthreads();
                    continue;
                }
                const float sc0 = (float)ldexp(s0, -fixbits);
                const float sc1 = ngr > 1 ? (float)ldexp(s1, -fixbits) : 0.f;
                const int accu0 = po.accumulate[0];
                for (int li = warp; li < ts.te[0]; li += nwarp) {
                    float *o0 = reinterpret_cast<float *>(po.out[0]) + obase + li * istride;
                    float *o1 = ngr > 1 ? reinterpret_cast<float *>(po.out[1]) + obase + li * istride : nullptr;
                    uint32_t *a0 = acc + kPadK + li * kSI;
                    uint32_t *a1 = a0 + kGS;
                    for (int lj = 0; lj < te1; ++lj, o0 += rstride, o1 += rstride, a0 += kSJ, a1 += kSJ) {
                        // padding cells take 0 x scale, as the reference scales the
                        // whole padded grid (src/fft.c:127-129): NaN for an empty catalog
                        float v0 = 0.f * sc0, v1 = 0.f * sc1;
                        if (lane >= te2) {
                            // a narrower tile's columns beyond te2 took its stencils'
                            // outer cells: they are cells of a wider tile to come
                            a0[lane] = 0u;
                            if (ngr > 1) a1[lane] = 0u;
                        } else {
                            const uint32_t c0 = a0[lane];
                            a0[lane] = 0u;
                            v0 = __uint2float_rn(c0) * sc0;
                            if (ngr > 1) {
                                const uint32_t c1 = a1[lane];
                                a1[lane] = 0u;
                                v1 = __uint2float_rn(c1) * sc1;
                            }
                        }
                        if (lane < rowlen) {
                            if (!accu0) o0[lane] = v0;
                            else if (lane < te2) o0[lane] += v0;
                            if (ngr > 1) {
                                if (!po.accumulate[1]) o1[lane] = v1;
                                else if (lane < te2) o1[lane] += v1;
                            }
                        }
                        if (lane + 32 < rowlen) {  // row padding beyond a full 32-cell tile
                            if (!accu0) o0[lane + 32] = 0.f * sc0;
                            if (ngr > 1 && !po.accumulate[1]) o1[lane + 32] = 0.f * sc1;
                        }
                    }
                }
            }
        }
        if (next >= ntiles) break;
        // the clearing above completes before the next deposit: tile_publish
        // synchronises the CTA
        tile_publish(nb_comb, nb_begin, nb_cnt, seg_begin, seg_pref, scan_ws, ts);
        tile = next;
    }
}

// ---- 4b. tile paint of FP32 grids with Ng >= 64: one thread per particle ------------------
// A tile holds one grid's sums of 32 x 16 x 32 cells in blocks of 2 x 4 x 4
// cells: cell (i, j, k') of a tile is word (i & 1) * 16 + (j & 3) * 4 + (k' & 3) of
// block ((i >> 1) * 4 + (j >> 2)) * kRotKB + (k' >> 2), so its bank is the triple
// of digits (i & 1, j & 3, k' & 3).  The 4 x 4 x 4 stencil of any particle holds
// every triple exactly twice (rows i and i + 2).  Lane l, which deposits a
// particle of its own, therefore visits its 64 cells in an order of its own: at
// step (ta, tb, tk) it adds the two cells whose digits are its lane's digits
// plus (ta, tb, tk) (mod 2, 4, 4).  The 32 lanes of a warp have distinct digits,
// so every one of the 64 atomics takes one shared-memory wavefront whatever the
// particles' positions; only the weights and the address parts of each axis
// have to be rotated, once per particle.  Random banks instead measured 2.6
// cycles per atomic against 1.0.
// k' = k + a shift of 0..3 chosen per row so that blocks of 4 k' are 16-byte
// aligned in the grid, whose rows are Ng_pad floats apart: the write-out
// then stores float4s.  A row's shift depends only on the tile and the row's
// j parity (Ng even) and keeps the digits of a step distinct.
// Cells outside the tile: along i two blocks on either side of the sums take
// them and along k one more block (of both sides), none of which is read; along
// j they get weight 0 and the block 0 cell of their digit.  A dense tile paints
// 16 rows at a time into 64-bit sums of the same layout (rot_deposit_wide).
// Bound by instruction issue (67 % of the slots at Ng = 512) and the barriers
// between a tile's phases; 54 instructions per particle for both grids against
// 94 of the staged deposit, 10 of them per-tile work.  Both grids of 1e8
// uniform particles at Ng = 1024: 6.67 ms against 10.67; of the clustered 1e7 at
// Ng = 512 with ten wedges, the whole call 3.31 ms against 3.73.
constexpr int kRotKB = 10;                             // k' blocks of a row: 9 of the tile, 1 outside
constexpr int kRotJB = kRotKB * 128;                   // bytes of one j block
constexpr int kRotIB = 4 * kRotJB;                     // bytes of one i block (2 rows)
constexpr int kRotJunk = 2;                            // i blocks below and above the tile
constexpr size_t kRotAccBytes = (size_t)(16 + 2 * kRotJunk) * kRotIB;
constexpr size_t kRotSmem = kRotAccBytes + 2 * kBlkN * sizeof(uint32_t);
static_assert(16 / 2 * kRotIB * 2 <= (int)kRotAccBytes, "64-bit sums of 16 rows");
static_assert(2 * (kRotSmem + 1280 + 1024) <= 228 * 1024, "two CTAs per SM");

// first stencil cell (relative to the tile origin t0) along one axis of a record, in
// the grid shifted by delta (units of 2^-fb cells).  A tile's particles have it at
// -4 .. te (the base cell of one grid lies up to one cell beyond the reach of the
// other's stencil); in tiles at the box edge (fold) periodic images are folded there.
__device__ __forceinline__ int record_cell(uint32_t rw, int delta, int fb, int Ng, int t0, bool fold) {
    const int t = (int)(rw & ((1u << fb) - 1)) + delta;  // cell_g without its wrap
    int l = (int)(rw >> fb) + (t >> fb) - 1 - t0;
    if (fold) {
        l += l < -4 ? Ng : 0;
        l -= l >= Ng - 4 ? Ng : 0;
    }
    return l;
}

// the same, and the PCS weights (times 6 s)
__device__ __forceinline__ void record_axis(uint32_t rw, int delta, int fb, float inv, int Ng, int t0, bool fold,
                                            float s, int &l, float w[4]) {
    const uint32_t one = 1u << fb;
    const int t = (int)(rw & (one - 1)) + delta;
    pcs_weights((float)((uint32_t)t & (one - 1)) * inv, w, s);
    l = record_cell(rw, delta, fb, Ng, t0, fold);
}

// w[t] <- w[(t + r) & 3]
__device__ __forceinline__ void rotate4(float w[4], int r) {
    const bool r1 = r & 1, r2 = r & 2;
    const float a = r1 ? w[1] : w[0], b = r1 ? w[2] : w[1], c = r1 ? w[3] : w[2], d = r1 ? w[0] : w[3];
    w[0] = r2 ? c : a;
    w[1] = r2 ? d : b;
    w[2] = r2 ? a : c;
    w[3] = r2 ? b : d;
}

// add the bits of v at byte address a + OFF of shared memory
template <int OFF>
__device__ __forceinline__ void red_shared(uint32_t a, float v) {
    asm volatile("red.shared.add.u32 [%0+%2], %1;" ::"r"(a), "r"(__float_as_uint(v)), "n"(OFF) : "memory");
}

// (x, y) * (m, m), one packed instruction
__device__ __forceinline__ void mul2(float x, float y, float m, float &px, float &py) {
    asm("{\n .reg .b64 a, b, c;\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %4};\n mul.rn.f32x2 c, a, b;\n mov.b64 {%0, %1}, c;\n}"
        : "=f"(px), "=f"(py)
        : "f"(x), "f"(y), "f"(m));
}

// what a CTA keeps for the tile it paints
struct RotTile {
    int t0[3], te[3];
    int sh0, sh1;  // k shifts of the rows of even and odd local j
    bool fold;     // the tile touches the box edge
};

// a lane's digits at steps 0 and 1 along j (in bytes: 16 each) and along k (4
// each, in the rows of its own j parity); steps 2 and 3 are these with bit 1
// flipped, and so are the rows of the other parity where the shifts differ
struct RotLane {
    int j0, j1, k0, k1, kflip;
};

// Deposit of one particle by its lane.  The products of the weights
// are formed as denormal floats: w_ij is scaled by 2^-64 and w_k by 2^(s - 85), so
// the FP32 multiplication itself rounds w_ij w_k 2^s to the nearest integer (its
// bit pattern, below 2^24) and no conversion is left.
__device__ __forceinline__ void rot_deposit(uint32_t acc, const uint4 &rec, int Ng, int fb, const RotTile &rt,
                                            const RotLane &rl, const int delta[3], float inv, float s6k, int lane) {
    const int lk = lane & 3, lb = (lane >> 2) & 3, la = lane >> 4;
    constexpr float s6i = (1.f / 6.f) * 5.421010862427522e-20f;  // 2^-64 / 6
    int li, lj, l0;
    float wi[4], wj[4], wk[4];
    record_axis(rec.x, delta[0], fb, inv, Ng, rt.t0[0], rt.fold, s6i, li, wi);
    record_axis(rec.y, delta[1], fb, inv, Ng, rt.t0[1], rt.fold, 1.f / 6.f, lj, wj);
    record_axis(rec.z, delta[2], fb, inv, Ng, rt.t0[2], rt.fold, s6k, l0, wk);
    // the sums' i and k blocks cover first cells -4 .. te
    if ((unsigned)(li + 4) > (unsigned)(rt.te[0] + 4) || (unsigned)(l0 + 4) > (unsigned)(rt.te[2] + 4)) return;
    // i: rows of parity la, then 1 - la, each with the row 2 above it
    const int ra = (la - li) & 1;
    const int i0 = li + ra, i1 = li + 1 - ra;
    const uint32_t ad_i0 = acc + (uint32_t)((i0 >> 1) * kRotIB + la * 64);
    const uint32_t ad_i1 = acc + (uint32_t)((i1 >> 1) * kRotIB + (1 - la) * 64);
    const float x00 = ra ? wi[1] : wi[0], x01 = ra ? wi[3] : wi[2];
    const float x10 = ra ? wi[0] : wi[1], x11 = ra ? wi[2] : wi[3];
    // j: the cells of digit D lie in block lj >> 2 if D >= lj & 3, else in the next
    int ad_j[4];
    {
        const int f = (lj & 3) * 16, b0 = lj >> 2;
#pragma unroll
        for (int u = 0; u < 4; ++u) wj[u] = (unsigned)(lj + u) < 16u ? wj[u] : 0.f;
        rotate4(wj, (lb - lj) & 3);
        const int base0 = (unsigned)b0 < 4u ? b0 * kRotJB : 0, base1 = (unsigned)(b0 + 1) < 4u ? (b0 + 1) * kRotJB : 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int D = ((t & 1) ? rl.j1 : rl.j0) ^ (t & 2 ? 32 : 0);
            ad_j[t] = (D < f ? base1 : base0) + D;
        }
    }
    // k: rows of the lane's own j parity (tb even) are shifted by shA, the others by shB
    int ad_kA[4], ad_kB[4];
    {
        rotate4(wk, (lk - l0 - rt.sh0) & 3);
        const int kA = l0 + ((lb & 1) ? rt.sh1 : rt.sh0), kB = l0 + ((lb & 1) ? rt.sh0 : rt.sh1);
        const int fA = (kA & 3) * 4, fB = (kB & 3) * 4;
        const int a1 = (kA >> 2) * 128 + 128, b1 = (kB >> 2) * 128 + 128;
        const int a0 = kA < 0 ? 9 * 128 : a1 - 128, b0 = kB < 0 ? 9 * 128 : b1 - 128;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int DA = ((t & 1) ? rl.k1 : rl.k0) ^ (t & 2 ? 8 : 0), DB = DA ^ rl.kflip;
            ad_kA[t] = (DA < fA ? a1 : a0) + DA;
            ad_kB[t] = (DB < fB ? b1 : b0) + DB;
        }
    }
#pragma unroll
    for (int ta = 0; ta < 2; ++ta) {
#pragma unroll
        for (int tb = 0; tb < 4; ++tb) {
            const uint32_t row = (ta ? ad_i1 : ad_i0) + (uint32_t)ad_j[tb];
            float w0, w1;
            mul2(ta ? x10 : x00, ta ? x11 : x01, wj[tb], w0, w1);
#pragma unroll
            for (int tk = 0; tk < 4; ++tk) {
                const uint32_t a = row + (uint32_t)((tb & 1) ? ad_kB[tk] : ad_kA[tk]);
                float p0, p1;
                mul2(w0, w1, wk[tk], p0, p1);
                red_shared<0>(a, p0);
                red_shared<kRotIB>(a, p1);
            }
        }
    }
}

// The same into the 64-bit sums of rows [h, h + rows) of a dense tile, in the same
// order: in a clump the particles of a warp share a cell, and lanes that walked the
// stencil in one order would meet at every step.  A 64-bit addition to shared memory
// is a compare-and-swap loop, so the low words are added first and the additions that
// wrap around (1 in 1024 or fewer) carry one to the high word.  Tile paint of both grids
// with a clump of 3e6 particles in one cell (Ng = 512): 451 ms in one order with 64-bit
// atomics, 149 in the lanes' own orders, 48 so; 200 particles per cell everywhere
// (Ng = 128): 216, 215 and, with the queues of paint_rot_kernel, 145 ms.
__device__ __forceinline__ void rot_deposit_wide(uint32_t *acc, const uint4 &rec, int Ng, int fb,
                                                 const RotTile &rt, int h, int rows, const int delta[3], float inv,
                                                 float kscale, int lane) {
    const int lk = lane & 3, lb = (lane >> 2) & 3, la = lane >> 4;
    int l[3];
    float w[3][4];
    record_axis(rec.x, delta[0], fb, inv, Ng, rt.t0[0], true, 1.f / 6.f, l[0], w[0]);
    record_axis(rec.y, delta[1], fb, inv, Ng, rt.t0[1], true, 1.f / 6.f, l[1], w[1]);
    record_axis(rec.z, delta[2], fb, inv, Ng, rt.t0[2], true, 1.f / 6.f, l[2], w[2]);
    const int ra = (la - l[0]) & 1, rb = (lb - l[1]) & 3, rk = (lk - l[2] - rt.sh0) & 3;
    const float x[2][2] = {{ra ? w[0][1] : w[0][0], ra ? w[0][3] : w[0][2]},
                           {ra ? w[0][0] : w[0][1], ra ? w[0][2] : w[0][3]}};
    rotate4(w[1], rb);
    rotate4(w[2], rk);
#pragma unroll
    for (int c = 0; c < 4; ++c) w[2][c] *= kscale;
#pragma unroll
    for (int ta = 0; ta < 4; ++ta) {
        const int i = l[0] + ((ra + ta) & 1) + (ta & 2) - h;
        if ((unsigned)i >= (unsigned)rows) continue;
#pragma unroll
        for (int tb = 0; tb < 4; ++tb) {
            const int j = l[1] + ((rb + tb) & 3);
            if ((unsigned)j >= (unsigned)rt.te[1]) continue;
            const float wij = (x[ta & 1][ta >> 1] * 5.421010862427522e-20f) * w[1][tb];
            const int sh = (j & 1) ? rt.sh1 : rt.sh0;
            uint32_t *row = acc + 2 * (((i >> 1) * 4 + (j >> 2)) * (kRotKB * 32) + (i & 1) * 16 + (j & 3) * 4);
            auto low = [&](int tk) {
                const int k = l[2] + ((rk + tk) & 3) + sh;
                return row + 2 * ((k >> 2) * 32 + (k & 3));
            };
            uint32_t v[4], sum[4];
#pragma unroll
            for (int tk = 0; tk < 4; ++tk) {
                const bool in = (unsigned)(l[2] + ((rk + tk) & 3)) < (unsigned)rt.te[2];
                v[tk] = in ? __float_as_uint(wij * w[2][tk]) : 0u;
                sum[tk] = v[tk] ? atomicAdd(low(tk), v[tk]) : 0u;
            }
#pragma unroll
            for (int tk = 0; tk < 4; ++tk)
                if (sum[tk] + v[tk] < v[tk]) atomicAdd(low(tk) + 1, 1u);
        }
    }
}

// Persistent like paint_coop_kernel.  split: even CTAs paint grid 0 and odd
// CTAs grid 1 of the same tiles, from one sort keyed for both grids.  The
// offsets of the next tile's segments are loaded before the deposits and its
// first records before the write-out, so their latencies hide behind them.
// T threads: 512, two CTAs per SM, or, where there are no more tiles (times
// grids) than SMs, one CTA of 1024 (two grids of Ng = 96, 54 tiles, 3e5 particles:
// 38 us against 45; of Ng = 64, 16 tiles, 4e4 particles: 20 against 22).
template <int T>
__global__ void __launch_bounds__(T, 1024 / T)
paint_rot_kernel(PaintParams pp, const uint32_t *__restrict__ off, const uint4 *__restrict__ sorted, PaintOut po,
                 unsigned ntiles, int split) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char *accb = smem_raw + kRotJunk * kRotIB;  // the tile's block 0
    uint32_t *blk = reinterpret_cast<uint32_t *>(smem_raw + kRotAccBytes);
    __shared__ uint32_t seg_begin[128];
    __shared__ uint32_t seg_pref[128 + 1];
    __shared__ uint32_t scan_ws[33];
    __shared__ int fixbits_s;
    __shared__ int geo[6];         // t0, te of the tile
    __shared__ uint32_t first[2];  // the next tile's own particles: first record, count
    const int Ng = pp.Ng, fb = pp.fb, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int nwarp = T / 32;
    const int g = split ? (int)(blockIdx.x & 1) : 0;
    const int delta[3] = {g ? pp.ax[0].dq[1] : pp.ax[0].dq[0], g ? pp.ax[1].dq[1] : pp.ax[1].dq[0],
                          g ? pp.ax[2].dq[1] : pp.ax[2].dq[0]};
    float *const out = reinterpret_cast<float *>(g ? po.out[1] : po.out[0]);
    const double scd = po.ds ? po.ds->scale[g] : (g ? po.scale[1] : po.scale[0]);
    const float scf = (float)scd;
    const int accu = g ? po.accumulate[1] : po.accumulate[0];
    const unsigned cta = split ? blockIdx.x >> 1 : blockIdx.x;
    const unsigned ncta = split ? gridDim.x >> 1 : gridDim.x;
    unsigned tile = cta;
    if (tile >= ntiles) return;
    for (int e = tid; e < (int)(kRotAccBytes / 16); e += T)
        reinterpret_cast<uint4 *>(smem_raw)[e] = make_uint4(0, 0, 0, 0);
    // the segments of a tile, one per thread of the first four warps, and its
    // geometry, loaded into registers that nothing reads until publish() ...
    uint32_t nb_begin = 0, nb_end = 0;
    int nb_t0 = 0, nb_t1 = 0;
    const int nt0 = pp.nt[0], nt1 = pp.nt[1], nt2 = pp.nt[2];
    // thread q's segment as an offset from the tile and a class, the options
    // per axis as in tile_segment (two tiles or more along every axis)
    int sd[3] = {0, 0, 0}, scls = 0, scnt = tid == 0 ? 27 : (tid < kMaxSeg ? 1 : 0);
    if (tid > 0 && tid < kMaxSeg) {
        const int idx[3] = {tid / 25, (tid / 5) % 5, tid % 5};
        bool own = true;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int x = idx[a], nt = pp.nt[a];
            int c = x;
            if (x >= 3) {
                own = false;
                sd[a] = nt > 2 && x == 3 ? -1 : 1;
                c = (x == 3) == (nt > 2) ? 2 : 1;
            }
            scls = 3 * scls + c;
        }
        if (own) scnt = 0;  // part of segment 0
    }
    auto fetch = [&](unsigned t) {
        if (warp >= 4) return;
        const unsigned ti = t / (unsigned)nt2, tk = t - ti * nt2, t0i = ti / (unsigned)nt1, tj = ti - t0i * nt1;
        int o0 = (int)t0i + sd[0], o1 = (int)tj + sd[1], o2 = (int)tk + sd[2];
        o0 = o0 < 0 ? o0 + nt0 : (o0 >= nt0 ? o0 - nt0 : o0);
        o1 = o1 < 0 ? o1 + nt1 : (o1 >= nt1 ? o1 - nt1 : o1);
        o2 = o2 < 0 ? o2 + nt2 : (o2 >= nt2 ? o2 - nt2 : o2);
        const uint32_t key = (uint32_t)((o0 * nt1 + o1) * nt2 + o2) * 27u + (uint32_t)scls;
        nb_begin = off[key];
        nb_end = off[key + (uint32_t)scnt];
        if (tid < 3) {
            const int *st = pp.start[tid];
            const unsigned q = tid == 0 ? t0i : tid == 1 ? tj : tk;
            nb_t0 = st[q];
            nb_t1 = st[q + 1];
        }
    };
    // ... and published in shared memory with the counts' prefix sums
    auto publish = [&]() {
        const uint32_t nb_cnt = nb_end - nb_begin;
        uint32_t inc = nb_cnt;
        if (warp < 4) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            if (lane == 31) scan_ws[warp] = inc;
            if (tid < 3) {
                geo[tid] = nb_t0;
                geo[3 + tid] = nb_t1 - nb_t0;
            }
        }
        __syncthreads();
        if (warp < 4) {
            uint32_t add = 0;
            for (int w = 0; w < warp; ++w) add += scan_ws[w];
            seg_begin[tid] = nb_begin;
            seg_pref[tid] = add + inc - nb_cnt;
            if (tid == 127) seg_pref[128] = add + inc;
        }
        __syncthreads();
    };
    fetch(tile);
    publish();  // also orders the clearing above
    constexpr int nseg = 128;  // segments 125 .. 127 are empty
    uint4 rec = make_uint4(0, 0, 0, 0);
    if ((uint32_t)tid < seg_pref[1]) rec = sorted[seg_begin[0] + tid];
    const float inv = __int_as_float((127 - fb) << 23);  // 2^-fb (fb <= 24)
    const uint32_t acc = (uint32_t)__cvta_generic_to_shared(accb);
    const bool flip = (pp.Ng_pad & 3) != 0;        // rows alternate between 16-byte alignment and 8 off it
    const bool vec = !flip || (Ng & 1) == 0;       // the shift depends on j alone
    const long rstride = (long)pp.Ng_pad, istride = rstride * Ng;
    RotLane rl;
    {
        const int lk = lane & 3, lb = (lane >> 2) & 3;
        rl.kflip = vec && flip ? 8 : 0;
        rl.j0 = lb * 16;
        rl.j1 = ((lb + 1) & 3) * 16;
        rl.k0 = (lk * 4) ^ ((lb & 1) ? rl.kflip : 0);
        rl.k1 = (((lk + 1) & 3) * 4) ^ ((lb & 1) ? rl.kflip : 0);
    }
    for (;;) {
        const uint32_t total = seg_pref[128];
        RotTile rt;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            rt.t0[a] = geo[a];
            rt.te[a] = geo[3 + a];
        }
        rt.fold = rt.t0[0] == 0 || rt.t0[1] == 0 || rt.t0[2] == 0 || rt.t0[0] + rt.te[0] == Ng ||
                  rt.t0[1] + rt.te[1] == Ng || rt.t0[2] + rt.te[2] == Ng;
        rt.sh0 = rt.sh1 = 0;
        if (vec) {
            rt.sh0 = (rt.t0[2] + (flip ? 2 * rt.t0[1] : 0)) & 3;
            rt.sh1 = (rt.t0[2] + (flip ? 2 * (rt.t0[1] + 1) : 0)) & 3;
        }
        const unsigned next = tile + ncta;
        if (next < ntiles) fetch(next);
        const uint32_t own = seg_pref[1];  // segment 0: the tile's own particles
        auto index = [&](uint32_t q) -> uint32_t {
            return q < own ? seg_begin[0] + q : seg_index(q, seg_begin, seg_pref, nseg);
        };
        int fixbits = fix_bits_for(total);
        if (fixbits < kBlockCountBelow) {
            const bool cyc[3] = {false, false, false};  // Ng >= 64: two tiles or more along every axis
            TileSegs ts;
            for (int a = 0; a < 3; ++a) ts.t0[a] = rt.t0[a];
            fixbits = tile_fixbits(total, sorted, index, pp, ts, cyc, blk, blk + kBlkN, scan_ws, &fixbits_s);
        }
        const bool wide = fixbits < kWideBelow;
        const int te0 = rt.te[0], te1 = rt.te[1], te2 = rt.te[2];
        const int rowlen = te2 + (rt.t0[2] + te2 == Ng ? pp.Ng_pad - Ng : 0);  // with the padding of the last k tile
        float *obase = out + ((long)rt.t0[0] * Ng + rt.t0[1]) * rstride + rt.t0[2];
        if (!wide) {
            const float s6k = (1.f / 6.f) * __int_as_float((127 + fixbits - 85) << 23);  // 2^(s - 85) / 6
            if ((uint32_t)tid >= own && (uint32_t)tid < total) rec = sorted[index((uint32_t)tid)];
            for (uint32_t q = tid; q < total; q += T) {
                const uint4 r = rec;
                if (q + T < total) rec = sorted[index(q + T)];  // in flight during the deposit
                rot_deposit(acc, r, Ng, fb, rt, rl, delta, inv, s6k, lane);
            }
            if (tid == 0) {
                first[0] = nb_begin;
                first[1] = next < ntiles ? nb_end - nb_begin : 0u;
            }
            __syncthreads();
            if ((uint32_t)tid < first[1]) rec = sorted[first[0] + tid];
            // write the owned cells and clear the sums.  A warp takes a block row (2 x 4
            // rows): 8 lanes read the 8 rows of one block (one wavefront), the four
            // groups of 8 lanes blocks kq and kq + 4 along k; then lanes l and l ^ 4
            // exchange so that a store covers 4 whole rows of the tile.  (64-byte
            // pieces of 8 rows took 18 store wavefronts per instruction, and the
            // whole paint 7.36 ms.)
            const float sc = scf * __int_as_float((127 - fixbits) << 23);  // scale 2^-s
            const float padv = 0.f * sc;  // padding cells take 0 x scale, as the reference
                                          // scales the whole padded grid (src/fft.c:127-129)
            // shift, extent and padding are even and the rows 16-byte aligned up to their shift
            const bool pairs = vec && !accu && ((rt.sh0 | te2 | rowlen) & 1) == 0;
            static_assert(nwarp % 4 == 0, "a warp's block rows are nwarp / 2 rows apart, with one j");
            const int r = lane & 7, kq = lane >> 3, hi = r >> 2;
            const int j = 4 * (warp & 3) + (r & 3), sh = (r & 1) ? rt.sh1 : rt.sh0;
            const int k = 4 * (kq + 4 * hi) - sh;  // after the exchange
            const bool full = pairs && te0 == 32 && te1 == 16 && rowlen == 32;  // no checks but the ends of shifted rows
            int i = 2 * (warp >> 2);
            uint4 *src = reinterpret_cast<uint4 *>(accb) + (warp * kRotKB + kq) * 8 + r;
            float *o = obase + i * istride + j * rstride + k;
            const long tail_off = (hi ? istride - 16 : 0) + 32;  // o is at block 4 hi of row i
            auto take = [&](uint4 *sp) {
                const uint4 c = *sp;
                *sp = make_uint4(0, 0, 0, 0);
                return make_float4(__uint2float_rn(c.x) * sc, __uint2float_rn(c.y) * sc, __uint2float_rn(c.z) * sc,
                                   __uint2float_rn(c.w) * sc);
            };
            // cells kk .. kk + 3 of a row of the tile
            auto put = [&](float *op, const float4 &u, int kk) {
                if (pairs && kk >= 0 && kk + 4 <= te2) {
                    *reinterpret_cast<float4 *>(op) = u;
                } else if (pairs) {
                    // the ends of a row: kk, te2 and rowlen are even
                    if ((unsigned)kk < (unsigned)rowlen)
                        *reinterpret_cast<float2 *>(op) = kk < te2 ? make_float2(u.x, u.y) : make_float2(padv, padv);
                    if ((unsigned)(kk + 2) < (unsigned)rowlen)
                        *reinterpret_cast<float2 *>(op + 2) =
                            kk + 2 < te2 ? make_float2(u.z, u.w) : make_float2(padv, padv);
                } else {
                    const float v[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if ((unsigned)(kk + q) >= (unsigned)rowlen) continue;
                        if (!accu) op[q] = kk + q < te2 ? v[q] : padv;
                        else if (kk + q < te2) op[q] += v[q];
                    }
                }
            };
            // (rows that no tile has are never read: they need no clearing)
            for (; i < pp.tmax[0]; i += nwarp / 2, src += nwarp * kRotKB * 8, o += nwarp / 2 * istride) {
                float4 u = take(src), v = take(src + 4 * 8);
                const float4 snd = hi ? u : v;
                float4 rcv;
                rcv.x = __shfl_xor_sync(0xffffffffu, snd.x, 4);
                rcv.y = __shfl_xor_sync(0xffffffffu, snd.y, 4);
                rcv.z = __shfl_xor_sync(0xffffffffu, snd.z, 4);
                rcv.w = __shfl_xor_sync(0xffffffffu, snd.w, 4);
                if (hi) u = rcv;  // row i, blocks kq + 4 hi
                else v = rcv;     // row i + 1
                if (full) {
                    if (k >= 0) {
                        *reinterpret_cast<float4 *>(o) = u;
                        *reinterpret_cast<float4 *>(o + istride) = v;
                    } else {
                        *reinterpret_cast<float2 *>(o + 2) = make_float2(u.z, u.w);
                        *reinterpret_cast<float2 *>(o + istride + 2) = make_float2(v.z, v.w);
                    }
                } else if (j < te1) {
                    if (i < te0) put(o, u, k);
                    if (i + 1 < te0) put(o + istride, v, k);
                }
                if (kq == 0) {  // block 8 of row i + hi: the last cells of the shifted rows, and the padding
                    float *ot = o + tail_off;
                    const float4 w = take(src + 8 * 8);
                    if (full) {
                        if (sh) *reinterpret_cast<float2 *>(ot) = make_float2(w.x, w.y);
                    } else if (j < te1 && i + hi < te0) {
                        put(ot, w, 32 - sh);
                    }
                }
            }
        } else {
            // 16 rows at a time in 64-bit sums
            const float kscale = __int_as_float((127 + kWideBits - 85) << 23);
            const double sc = ldexp(scd, -kWideBits);
            uint32_t *acc64 = reinterpret_cast<uint32_t *>(smem_raw);  // low and high words
            static_assert(16 * kRotIB + T / 32 * 64 * sizeof(uint32_t) <= kRotAccBytes, "the warps' queues");
            for (int h = 0; h < te0; h += 16) {
                const int rows = min(16, te0 - h);
                __syncthreads();
                for (int e = tid; e < (int)(kRotAccBytes / 16); e += T)
                    reinterpret_cast<uint4 *>(smem_raw)[e] = make_uint4(0, 0, 0, 0);
                __syncthreads();
                // a warp queues the particles that reach these rows and deposits 32 at a
                // time (185 -> 145 ms at 200 particles per cell, where half of them do)
                uint32_t *queue = reinterpret_cast<uint32_t *>(smem_raw + 16 * kRotIB) + 64 * warp;
                int queued = 0;
                uint32_t at = 0, x = 0;
                if ((uint32_t)tid < total) {
                    at = index((uint32_t)tid);
                    x = sorted[at].x;
                }
                for (uint32_t q0 = 32 * warp; q0 < total; q0 += T) {
                    const int i = record_cell(x, delta[0], fb, Ng, rt.t0[0], true) - h;
                    const bool hit = q0 + lane < total && (unsigned)(i + 3) < (unsigned)(rows + 3);
                    const unsigned hits = __ballot_sync(0xffffffffu, hit);
                    if (hit) queue[queued + __popc(hits & ((1u << lane) - 1u))] = at;
                    queued += __popc(hits);
                    if (q0 + lane + T < total) {
                        at = index(q0 + lane + T);
                        x = sorted[at].x;
                    }
                    __syncwarp();
                    if (queued < 32) continue;
                    queued -= 32;
                    rot_deposit_wide(acc64, sorted[queue[lane]], Ng, fb, rt, h, rows, delta, inv, kscale, lane);
                    const uint32_t left = queue[32 + lane];
                    __syncwarp();
                    queue[lane] = left;
                    __syncwarp();
                }
                if (lane < queued)
                    rot_deposit_wide(acc64, sorted[queue[lane]], Ng, fb, rt, h, rows, delta, inv, kscale, lane);
                __syncthreads();
                for (int b = warp; b < 8 * 4 * kRotKB; b += nwarp) {
                    const int kb = b % kRotKB, rowb = b / kRotKB;
                    const int i = 2 * (rowb >> 2) + (lane >> 4), j = 4 * (rowb & 3) + ((lane >> 2) & 3);
                    const int k = 4 * kb + (lane & 3) - ((j & 1) ? rt.sh1 : rt.sh0);
                    if (i >= rows || j >= te1 || (unsigned)k >= (unsigned)rowlen) continue;
                    float *o = obase + (h + i) * istride + j * rstride + k;
                    const float v =
                        (float)((double)reinterpret_cast<const unsigned long long *>(acc64)[b * 32 + lane] * sc);
                    if (!accu) *o = v;
                    else if (k < te2) *o += v;
                }
            }
            if (tid == 0) {
                first[0] = nb_begin;
                first[1] = next < ntiles ? nb_end - nb_begin : 0u;
            }
            __syncthreads();
            if ((uint32_t)tid < first[1]) rec = sorted[first[0] + tid];
            for (int e = tid; e < (int)(kRotAccBytes / 16); e += T)
                reinterpret_cast<uint4 *>(smem_raw)[e] = make_uint4(0, 0, 0, 0);
        }
        if (next >= ntiles) break;
        publish();  // the clearing above completes before the next deposit
        tile = next;
    }
}

// FP64 grids: one warp per tile of 8 x 8 x 16 cells and grid (blockIdx.y), one
// lane per particle of the tile.  The FP64 pipe does two lanes per cycle and SM
// and bounds the kernel, so every operation counts: the sums cover the tile and
// the cells its particles' stencils reach beyond it, so that no particle is
// visited twice (the box is then added to the zeroed grid with FP64 atomics);
// the weights' divisions by 6 take three operations; and a deposit is one fused
// multiply-add on shared memory, without atomics.  That is safe because a warp
// owns its box and its lanes never meet: as in paint_rot_kernel, cell (i, j, k)
// lies at digits (i & 1, j & 3, k & 3) of a 2 x 4 x 4 block and lane l visits its
// particle's cells at its own digits plus the step's, so the 32 lanes of a step
// have 32 distinct digits (and the half warps 16 distinct bank pairs each).
// 1e6 particles at Ng = 128, both grids: 2.44 ms with 512-thread CTAs that
// pulled the neighbours' particles and added with shared FP64 atomics, whose
// compare-and-swap loops repeat the addition for a whole warp; 0.78 so.
constexpr int kF64Ext[3] = {8, 8, 16};
constexpr int kF64BJ = (8 + 4) / 4, kF64BK = (16 + 4) / 4;  // j and k blocks of the box
constexpr int kF64Blocks = (8 + 4) / 2 * kF64BJ * kF64BK;
// a warp deposits at most this many particles: the sorted particles are cut at
// multiples of it, and a crowded tile's later pieces go to warps of their own
// (blockIdx.x >= ntiles; the boxes are added atomically, so pieces may share a tile)
constexpr uint32_t kF64Piece = 4096;

// word of box cell (i, j, k)
__device__ __forceinline__ int f64_row(int i) { return (i >> 1) * (kF64BJ * kF64BK * 32) + (i & 1) * 16; }
__device__ __forceinline__ int f64_col(int j) { return (j >> 2) * (kF64BK * 32) + (j & 3) * 4; }
__device__ __forceinline__ int f64_k(int k) { return (k >> 2) * 32 + (k & 3); }

__device__ __forceinline__ void rotate4(double w[4], int r) {
    const bool r1 = r & 1, r2 = r & 2;
    const double a = r1 ? w[1] : w[0], b = r1 ? w[2] : w[1], c = r1 ? w[3] : w[2], d = r1 ? w[0] : w[3];
    w[0] = r2 ? c : a;
    w[1] = r2 ? d : b;
    w[2] = r2 ? a : c;
    w[3] = r2 ? b : d;
}

__global__ void __launch_bounds__(32, 9)
paint_warp_f64_kernel(PaintParams pp, const uint32_t *__restrict__ off,
                      const Rec<double>::type *__restrict__ sorted, PaintOut po, unsigned ntiles) {
    __shared__ __align__(16) double acc[32 * kF64Blocks];
    const int Ng = pp.Ng, g = blockIdx.y, lane = threadIdx.x;
    unsigned tile = blockIdx.x;
    uint32_t p0, p1;
    if (blockIdx.x < ntiles) {
        p0 = off[tile];
        p1 = min(off[tile + 1], (p0 / kF64Piece + 1) * kF64Piece);
    } else {
        // the piece from p0: part of the tile that holds p0, unless that begins there
        p0 = (blockIdx.x - ntiles + 1) * kF64Piece;
        if (p0 >= off[ntiles]) return;
        unsigned lo = 0, hi = ntiles - 1;  // the last tile with off[tile] <= p0
        while (lo < hi) {
            const unsigned mid = (lo + hi + 1) >> 1;
            if (off[mid] <= p0) lo = mid;
            else hi = mid - 1;
        }
        tile = lo;
        if (off[tile] == p0) return;
        p1 = min(off[tile + 1], p0 + kF64Piece);
    }
    TileSegs ts;
    tile_geometry(pp, tile, ts);
    double *out = reinterpret_cast<double *>(g ? po.out[1] : po.out[0]);
    const double sc = g ? po.scale[1] : po.scale[0];
    const int accu = g ? po.accumulate[1] : po.accumulate[0];
    const bool finite = isfinite(sc);
    // the row padding takes 0 x scale, like the reference's scaling of the whole grid
    const int pad = blockIdx.x < ntiles && ts.t0[2] + ts.te[2] == Ng && !accu ? pp.Ng_pad - Ng : 0;
    for (int e = lane; e < ts.te[0] * ts.te[1] * pad; e += 32) {
        const int q = e % pad, lj = (e / pad) % ts.te[1], li = e / (pad * ts.te[1]);
        out[((long)(ts.t0[0] + li) * Ng + ts.t0[1] + lj) * pp.Ng_pad + Ng + q] = __dmul_rn(0.0, sc);
    }
    // an empty tile leaves the zeroed grid as it is (1e5 particles, Ng = 512, half of the
    // tiles are empty: the whole fft_p2g 1.21 ms, 2.84 without this)
    if (p0 == p1 && finite) return;
#pragma unroll 6
    for (int e = lane; e < 32 * kF64Blocks; e += 32) acc[e] = 0.0;
    // the box starts `low` cells below the tile: 1, or 2 where the grid's base
    // cells can lie one below those of grid 0, which the sort went by
    int low[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) low[a] = pp.ax[a].o[g] > pp.ax[a].o[0] ? 2 : 1;
    const int lk = lane & 3, lb = (lane >> 2) & 3, la = lane >> 4;
    volatile double *vacc = acc;
    __syncwarp();
    for (uint32_t q0 = p0; q0 < p1; q0 += 32) {
        const bool valid = q0 + lane < p1;
        Rec<double>::type r;
        r.x = r.y = r.z = 0.0;
        if (valid) r = sorted[q0 + lane];
        const double pos[3] = {r.x, r.y, r.z};
        int l[3];
        double w[3][4];
        bool in = valid;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            int b;
            double d;
            coord(pos[a], pp.ax[a], g, Ng, b, d);
            pcs_weights(d, w[a]);
            int c = b - 1 - ts.t0[a] + low[a];
            c += c < 0 ? Ng : 0;
            c -= c >= Ng ? Ng : 0;
            in = in && (unsigned)c <= (unsigned)ts.te[a];  // a particle of the tile has its first cell at 0 .. te
            l[a] = c;
        }
        if (!in) {  // lanes without a particle go along with weight 0
            l[0] = l[1] = l[2] = 0;
#pragma unroll
            for (int s = 0; s < 4; ++s) w[0][s] = 0.0;
        }
        const int ra = (la - l[0]) & 1, rb = (lb - l[1]) & 3, rk = (lk - l[2]) & 3;
        const int row[2] = {f64_row(l[0] + ra), f64_row(l[0] + 1 - ra)};
        const double x[2][2] = {{ra ? w[0][1] : w[0][0], ra ? w[0][3] : w[0][2]},
                                {ra ? w[0][0] : w[0][1], ra ? w[0][2] : w[0][3]}};
        rotate4(w[1], rb);
        rotate4(w[2], rk);
        int col[4], kc[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            col[t] = f64_col(l[1] + ((rb + t) & 3));
            kc[t] = f64_k(l[2] + ((rk + t) & 3));
        }
#pragma unroll
        for (int ta = 0; ta < 2; ++ta)
#pragma unroll
            for (int tb = 0; tb < 4; ++tb) {
                const double w0 = __dmul_rn(x[ta][0], w[1][tb]), w1 = __dmul_rn(x[ta][1], w[1][tb]);
                const int rc = row[ta] + col[tb];
#pragma unroll
                for (int tk = 0; tk < 4; ++tk) {
                    volatile double *p = vacc + rc + kc[tk];
                    const double a0 = p[0], a1 = p[kF64BJ * kF64BK * 32];  // rows i and i + 2
                    p[0] = __fma_rn(w0, w[2][tk], a0);
                    p[kF64BJ * kF64BK * 32] = __fma_rn(w1, w[2][tk], a1);
                    __syncwarp();
                }
            }
    }
    __syncwarp();
    // Add the box to the grid.  A non-finite scale takes every cell of the tile (and none
    // beyond it): 0 x inf.  In a sparse tile this is most of the work, so the grid
    // indices are formed once per axis and block instead of with three remainders per
    // cell, and what is zero is told by its bits before the FP64 pipe sees it (1e6
    // particles, Ng = 512, 8 to a tile: the whole fft_p2g 3.66 -> 2.32 ms).
    auto wrap = [&](int c) {
        while (c < 0) c += Ng;
        while (c >= Ng) c -= Ng;
        return c;
    };
    int kk[kF64BK];
#pragma unroll
    for (int kb = 0; kb < kF64BK; ++kb) kk[kb] = wrap(ts.t0[2] + 4 * kb + lk - (finite ? low[2] : 0));
    const double *src = acc + lane;
    for (int li = la; li < 8 + 4; li += 2) {
        double *plane = out + (long)wrap(ts.t0[0] + li - (finite ? low[0] : 0)) * Ng * pp.Ng_pad;
#pragma unroll
        for (int jb = 0; jb < kF64BJ; ++jb, src += 32 * kF64BK) {
            const int lj = 4 * jb + lb;
            double *row = plane + (long)wrap(ts.t0[1] + lj - (finite ? low[1] : 0)) * pp.Ng_pad;
            const bool outside = li >= ts.te[0] || lj >= ts.te[1];
#pragma unroll
            for (int kb = 0; kb < kF64BK; ++kb) {
                const double v = src[32 * kb];
                if (finite ? __double_as_longlong(v) == 0 : (outside || 4 * kb + lk >= ts.te[2])) continue;
                atomicAdd(row + kk[kb], __dmul_rn(v, sc));
            }
        }
    }
}

// ---- host side -----------------------------------------------------------------------------

static int tiling_build(PaintTiling *t, int Ng, const int ext[3], int classes) {
    std::vector<int> tab;
    long nk = classes;
    for (int a = 0; a < 3; ++a) {
        int nt = (int)ceil_div(Ng, ext[a]);
        // with more than one tile per axis and boundary classes every extent must be
        // >= 5 so that a stencil reaches at most the adjacent tile and the classes
        // are exclusive
        while (classes > 1 && nt > 1 && Ng / nt < 5) --nt;
        t->tab_off[a] = (int)tab.size();
        const size_t base = tab.size();
        tab.resize(base + Ng + nt + 1);
        int tmax = 0;
        for (int q = 0; q <= nt; ++q) tab[base + Ng + q] = (int)((long)q * Ng / nt);
        for (int q = 0; q < nt; ++q) {
            const int s0 = tab[base + Ng + q], s1 = tab[base + Ng + q + 1];
            tmax = s1 - s0 > tmax ? s1 - s0 : tmax;
            for (int c = s0; c < s1; ++c) tab[base + c] = q;
        }
        if (tmax > ext[a]) return set_error(ERR_STATE, "paint tile extent %d > %d", tmax, ext[a]);
        t->nt[a] = nt;
        t->tmax[a] = tmax;
        nk *= nt;
    }
    t->Ng = Ng;
    t->nkeys = nk;
    if (t->nkeys >= (1L << 32)) return set_error(ERR_UNSUPPORTED, "too many paint tiles");
    FG_CUDA(cudaMalloc(&t->d_tables, sizeof(int) * tab.size()));
    FG_CUDA(cudaMemcpy(t->d_tables, tab.data(), sizeof(int) * tab.size(), cudaMemcpyHostToDevice));
    return OK;
}

int paint_tiling_create(PaintTiling *t, int Ng, int prec) {
    if (prec == 8) return tiling_build(t, Ng, kF64Ext, 1);
    FG_TRY(tiling_build(t, Ng, kTileExt, 27));
    if (Ng >= 64) {
        t->one = new PaintTiling();
        FG_TRY(tiling_build(t->one, Ng, kTileExt1, 27));
    }
    return OK;
}

void paint_tiling_destroy(PaintTiling *t) {
    if (t->one) {
        paint_tiling_destroy(t->one);
        delete t->one;
        t->one = nullptr;
    }
    cudaFree(t->d_tables);
    t->d_tables = nullptr;
}

void paint_scratch_free(PaintScratch *s) {
    cudaFree(s->sorted);
    cudaFree(s->hist);
    cudaFree(s->cursor);
    cudaFree(s->scan_tmp);
    *s = PaintScratch();
}

static int ensure_scratch(PaintScratch *s, long Np, long nkeys) {
    if (Np > s->cap_particles) {
        cudaFree(s->sorted);
        s->sorted = nullptr;
        const long cap = Np + Np / 8 + 1024;
        FG_CUDA(cudaMalloc(&s->sorted, 32 * (size_t)cap));  // fits float4 and 3 doubles
        s->cap_particles = cap;
    }
    if (nkeys + 1 > s->cap_keys) {
        cudaFree(s->hist);
        cudaFree(s->cursor);
        cudaFree(s->scan_tmp);
        s->hist = s->cursor = s->scan_tmp = nullptr;
        FG_CUDA(cudaMalloc(&s->hist, sizeof(uint32_t) * (nkeys + 1)));
        FG_CUDA(cudaMalloc(&s->cursor, sizeof(uint32_t) * (nkeys + 1)));
        FG_CUDA(cudaMalloc(&s->scan_tmp, sizeof(uint32_t) * (ceil_div(nkeys + 1, kScanBlock) + 1)));
        s->cap_keys = nkeys + 1;
    }
    s->bytes = (size_t)32 * s->cap_particles + 2 * sizeof(uint32_t) * (size_t)s->cap_keys;
    return OK;
}

int paint_reserve(const PaintTiling *t, PaintScratch *s, long Np) {
    return ensure_scratch(s, Np > 0 ? Np : 1, t->nkeys);
}

static void split(double v, float &hi, float &lo) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

int paint(const PaintTiling *t, PaintScratch *s, int grid_prec, const void *x, const void *y, const void *z,
          int pos_prec, long Np, double Hinv, const PaintGridSpec *grids, int ngrids, cudaStream_t st,
          cudaEvent_t *ev, const PaintRsd *rsd, const DevScalars *ds) {
    if (ngrids < 1 || ngrids > kMaxPaintGrids) return set_error(ERR_ARG, "paint: 1 or 2 grids");
    if (ds && (grid_prec != 4 || pos_prec != 4)) return set_error(ERR_ARG, "paint: device scalars need FP32");
    if (rsd && rsd->v[0] && pos_prec != 4) return set_error(ERR_ARG, "paint: displacement needs FP32 positions");
    if (pos_prec != grid_prec) return set_error(ERR_ARG, "paint: position precision must match grid precision");
    const int cta_per_sm = t->cta_per_sm;
    const bool big = grid_prec == 4 && t->one;  // FP32: the 32 x 16 x 32 tiles
    if (big) t = t->one;
    if (Np < 0 || Np >= (1L << 32)) return set_error(ERR_ARG, "paint: Np out of range");
    for (int g = 1; g < ngrids; ++g)
        for (int a = 0; a < 3; ++a)
            if (fabs(grids[g].offset[a] - grids[0].offset[a]) > 1.0)
                return set_error(ERR_ARG, "paint: grid offsets must lie within one cell");
    const int Ng = t->Ng;
    PaintParams pp;
    memset(&pp, 0, sizeof(pp));
    pp.Ng = Ng;
    pp.Ng_pad = 2 * (Ng / 2 + 1);
    pp.ngrids = ngrids;
    if (rsd && rsd->v[0]) {
        for (int a = 0; a < 3; ++a) {
            pp.v[a] = rsd->v[a];
            pp.los[a] = (float)rsd->los[a];
        }
        pp.aHinv = (float)rsd->aHinv;
    }
    int bits_b = 1;
    while ((1 << bits_b) < Ng) ++bits_b;
    pp.fb = 32 - bits_b < 24 ? 32 - bits_b : 24;  // 2^-24 cell: below FP32 resolution
    if (grid_prec == 4 && pp.fb < 16) return set_error(ERR_UNSUPPORTED, "FP32 paint: Ng=%d too large", Ng);
    for (int a = 0; a < 3; ++a) {
        pp.nt[a] = t->nt[a];
        pp.tmax[a] = t->tmax[a];
        pp.tile_of[a] = t->d_tables + t->tab_off[a];
        {
            const int ext = Ng / t->nt[a];
            pp.tshift[a] = -1;
            if (ext * t->nt[a] == Ng && (ext & (ext - 1)) == 0)
                for (int b = 0; (1 << b) <= ext; ++b)
                    if ((1 << b) == ext) pp.tshift[a] = b;
        }
        pp.start[a] = t->d_tables + t->tab_off[a] + Ng;
        split(Hinv, pp.ax[a].h_hi, pp.ax[a].h_lo);
        pp.ax[a].h = Hinv;
        for (int g = 0; g < ngrids; ++g) {
            split(grids[g].offset[a], pp.ax[a].o_hi[g], pp.ax[a].o_lo[g]);
            pp.ax[a].o[g] = grids[g].offset[a];
            pp.ax[a].dq[g] = (int)llrint((grids[0].offset[a] - grids[g].offset[a]) * (double)(1u << pp.fb));
        }
    }
    PaintOut po;
    memset(&po, 0, sizeof(po));
    for (int g = 0; g < ngrids; ++g) {
        po.out[g] = grids[g].out;
        po.scale[g] = grids[g].scale;
        po.accumulate[g] = grids[g].accumulate;
    }
    po.ds = ds;
    FG_TRY(ensure_scratch(s, Np > 0 ? Np : 1, t->nkeys));
    FG_CUDA(cudaMemsetAsync(s->hist, 0, sizeof(uint32_t) * (t->nkeys + 1), st));
    const int nsm = num_sms();
    const unsigned gp = (unsigned)(Np > 0 ? (ceil_div(Np, 256) < 32L * nsm ? ceil_div(Np, 256) : 32L * nsm) : 1);
    // few keys: counted in shared memory, two particles or more per thread
    const bool few = t->nkeys <= kFewKeys;
    const size_t ksm = sizeof(uint32_t) * (size_t)t->nkeys;
    const unsigned gf = (unsigned)(ceil_div(Np, 512) < 4L * nsm ? ceil_div(Np, 512) : 4L * nsm);
#define FG_KEY_LAUNCH(P, D)                                                                                      \
    do {                                                                                                        \
        if (few)                                                                                                \
            paint_key_few_kernel<P><<<gf, 256, ksm, st>>>((const P *)x, (const P *)y, (const P *)z, Np, pp,      \
                                                          s->hist, (int)t->nkeys, D);                           \
        else                                                                                                    \
            paint_key_kernel<P><<<gp, 256, 0, st>>>((const P *)x, (const P *)y, (const P *)z, Np, pp, s->hist, D); \
    } while (0)
    if (Np > 0) {
        if (pos_prec == 4)
            FG_KEY_LAUNCH(float, ds);
        else
            FG_KEY_LAUNCH(double, nullptr);
        FG_LAUNCHED(1);
    }
#undef FG_KEY_LAUNCH
    if (ev) FG_CUDA(cudaEventRecord(ev[0], st));
    FG_TRY(exclusive_scan(s->hist, s->cursor, t->nkeys + 1, s->scan_tmp, st));
    if (ev) FG_CUDA(cudaEventRecord(ev[1], st));
    if (Np > 0) {
        if (pos_prec == 4)
            paint_scatter_kernel<float><<<gp, 256, 0, st>>>((const float *)x, (const float *)y, (const float *)z,
                                                           Np, pp, s->cursor, (uint4 *)s->sorted, ds);
        else
            paint_scatter_kernel<double><<<gp, 256, 0, st>>>((const double *)x, (const double *)y,
                                                            (const double *)z, Np, pp, s->cursor,
                                                            (Rec<double>::type *)s->sorted, nullptr);
        FG_LAUNCHED(1);
    }
    if (ev) FG_CUDA(cudaEventRecord(ev[2], st));
    const unsigned ntiles = (unsigned)((long)t->nt[0] * t->nt[1] * t->nt[2]);
    if (grid_prec == 4) {
        const unsigned slots = (unsigned)((cta_per_sm == 1 ? 1 : 2) * num_sms());
        if (big) {
            // one grid per CTA: with two grids, even CTAs paint grid 0 and odd
            // CTAs grid 1 (the sort's keys cover both grids' stencils)
            const int split = ngrids == 2;
            unsigned nb = slots < ntiles * ngrids ? slots : ntiles * ngrids;
            if (split) nb &= ~1u;
            FG_CUDA(cudaFuncSetAttribute(paint_rot_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRotSmem));
            FG_CUDA(cudaFuncSetAttribute(paint_rot_kernel<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRotSmem));
            if (ntiles * ngrids <= (unsigned)num_sms())
                paint_rot_kernel<1024><<<nb, 1024, kRotSmem, st>>>(pp, s->hist, (const uint4 *)s->sorted, po, ntiles,
                                                                   split);
            else
                paint_rot_kernel<512><<<nb, 512, kRotSmem, st>>>(pp, s->hist, (const uint4 *)s->sorted, po, ntiles,
                                                                 split);
        } else {
            constexpr int T = kPaintThreads;
            const size_t smem = kAccBytes + sizeof(StageBuf) * (T / 32);
            const unsigned nb = slots < ntiles ? slots : ntiles;
            FG_CUDA(cudaFuncSetAttribute(paint_coop_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            FG_CUDA(cudaFuncSetAttribute(paint_coop_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            if (ngrids == 1)
                paint_coop_kernel<1><<<nb, T, smem, st>>>(pp, s->hist, (const uint4 *)s->sorted, po, ntiles);
            else
                paint_coop_kernel<2><<<nb, T, smem, st>>>(pp, s->hist, (const uint4 *)s->sorted, po, ntiles);
        }
    } else {
        for (int g = 0; g < ngrids; ++g)
            if (!grids[g].accumulate)
                FG_CUDA(cudaMemsetAsync(grids[g].out, 0, sizeof(double) * (size_t)Ng * Ng * pp.Ng_pad, st));
        paint_warp_f64_kernel<<<dim3(ntiles + (unsigned)(Np / kF64Piece), ngrids), 32, 0, st>>>(
            pp, s->hist, (const Rec<double>::type *)s->sorted, po, ntiles);
    }
    FG_LAUNCHED(1);
    if (ev) FG_CUDA(cudaEventRecord(ev[3], st));
    return OK;
}

}  // namespace fg
