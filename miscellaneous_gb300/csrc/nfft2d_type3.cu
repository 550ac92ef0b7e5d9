// nfft2d_type3.cu -- type-3 2D NUFFT (nonuniform points to nonuniform
// frequencies) by Gaussian gridding, the reference's other native NUFFT:
//     F_k = sum_j f_j exp(-i (s_k x_j + t_k y_j))
// following NUFFT_2D_CPU (NFFT/NFFT3/C/NFFT3_2D_C.cpp:199-312): extents and
// centres of both point sets, R = 2.2 and the Gaussian half-width msp for
// the requested accuracy (:234-238), a rescaling that maps the points onto
// [-pi/2, pi/2] around their centre (:243-264), then
//   1) Gaussian spreading of the phase-shifted values onto an Mry x Mrx grid
//      with the pre-compensation exp(b (Dy^2 n_j^2 + Dx^2 n_i^2)) (:38-85);
//   2) a forward 2D FFT (cuFFT here, MKL there, :283-292);
//   3) Gaussian gathering at the scaled frequencies with the
//      post-compensation and the phase of the centres (:156-194).
// The reference's circular shift by half the grid with the (-1)^(i+j)
// checkerboard (:135-151) is folded into the gather's indexing: no pass.
//
// Kernels: the Gaussian weight of a footprint tap factors into a row and a
// column weight, so a point or frequency needs 2(2 msp + 1) exponentials, not
// (2 msp + 1)^2.  Points and frequencies are binned by the 16 x 16 grid tile
// of their footprint's first cell; the footprints of a tile then lie in one
// patch of (16 + 2 msp)^2 cells, and with the weights zero-padded to the patch
// both directions are small dense products.  FP32 data: the spread adds the
// outer products of a tile's points into a patch held in registers, the gather
// multiplies the patch by 64 frequencies' column weights at a time, both with
// 8 x 8 register tiles.  FP64 data: the spread accumulates in a shared-memory
// patch (warps own disjoint rows), the gather runs one warp per frequency over
// the footprint.  One global atomic add per cell puts a patch into the grid.
#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "nfft2d_internal.h"

namespace {

constexpr double kPi = 3.141592653589793238463;  // the reference's PI (NFFT3_2D_C.cpp:24)
constexpr int kWarpsPerBlock = 8;

__device__ __forceinline__ unsigned long long ord_key(double v) {
    const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
double ord_value(unsigned long long k) {
    const unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    double v;
    std::memcpy(&v, &u, sizeof v);
    return v;
}

// Keys of min a, max a, min b, max b of two arrays of n values into mm[0..3]
// (blockIdx.y 0) and of two others into mm[4..7] (blockIdx.y 1).  Compared as
// ordered integer keys: FP64 min and max run on GB300's slow FP64 pipe, and
// one atomic a block instead of one a warp keeps the four words uncontended
// (22 us a pair of 2 * 10^5 values -> 5 for both pairs).  NaNs are left out.
constexpr int kMinmaxThreads = 256;
__global__ void __launch_bounds__(kMinmaxThreads)
    k_minmax2(const double *__restrict__ a0, const double *__restrict__ b0, long long n0,
              const double *__restrict__ a1, const double *__restrict__ b1, long long n1, unsigned long long *mm) {
    const double *a = blockIdx.y ? a1 : a0, *b = blockIdx.y ? b1 : b0;
    const long long n = blockIdx.y ? n1 : n0;
    unsigned long long v[4] = {ord_key(DBL_MAX), ord_key(-DBL_MAX), ord_key(DBL_MAX), ord_key(-DBL_MAX)};
    auto nan = [](double x) {
        return (static_cast<unsigned long long>(__double_as_longlong(x)) << 1) > 0xffe0000000000000ull;
    };
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const double x = a[i], y = b[i];
        if (!nan(x)) {
            v[0] = min(v[0], ord_key(x));
            v[1] = max(v[1], ord_key(x));
        }
        if (!nan(y)) {
            v[2] = min(v[2], ord_key(y));
            v[3] = max(v[3], ord_key(y));
        }
    }
    __shared__ unsigned long long sm[kMinmaxThreads / 32][4];
    for (int o = 16; o > 0; o >>= 1)
        for (int k = 0; k < 4; ++k) {
            const unsigned long long u = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k] = (k & 1) ? max(v[k], u) : min(v[k], u);
        }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 4; ++k) sm[threadIdx.x >> 5][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 4) {
        const int k = threadIdx.x;
        unsigned long long r = sm[0][k];
        for (int w = 1; w < kMinmaxThreads / 32; ++w) r = (k & 1) ? max(r, sm[w][k]) : min(r, sm[w][k]);
        if (k & 1)
            atomicMax(mm + 4 * blockIdx.y + k, r);
        else
            atomicMin(mm + 4 * blockIdx.y + k, r);
    }
}

struct Params {
    double xb, yb, sb, tb;   // centres after the rescaling
    double kx, ky;           // rescaling X1 / (pi/2), Y1 / (pi/2)
    double Dx, Dy;           // grid steps 2 pi / Mr
    double b, t1, fact;      // Gaussian constants, fact = (1 / (4 pi b))^2
    int Mrx, Mry, ms;        // grid and footprint half-width
};

__device__ __forceinline__ int wrap(long long i, int n) {
    long long r = i % n;
    return static_cast<int>(r < 0 ? r + n : r);
}

// ---------------------------------------------------------------------------
// Spreading (NFFT3_2D_C.cpp:38-85), binned.  Tap (r, c) of a point has the
// weight exp(ex(c) + ey(r)) with ex depending on the column only and ey on
// the row only (:61-74), so a point needs 2(2ms+1) exponentials, not
// (2ms+1)^2, and the products wr(r) wc(c) are formed in the data precision.
// Points are binned by the TS x TS grid tile of their footprint's first
// cell; a CTA accumulates one work item (at most kT3Item points of one
// tile) into a shared-memory patch of (TS + W - 1)^2 cells -- warp w owns
// the patch rows r = w (mod 8), so no two threads ever touch one cell and no
// shared atomics are needed -- and adds the patch into the grid with one
// global atomic add per cell and component.
// ---------------------------------------------------------------------------
constexpr int kT3Tile = 16;    // TS
constexpr int kT3Item = 1024;  // points per work item (FP64)
constexpr int kT3Warps = 8;    // warps of a spreading CTA (FP64)

struct T3Rec {
    double xt, yt;  // (x - xb) / Dx, (y - yb) / Dy (:53-54)
    double re, im;  // the value with the centre phase removed and the constant factor (:48-51)
    int i0, j0;     // first footprint column and row, unwrapped (floor(M/2 + t) - ms)
};
// FP32 data: the fractional parts of xt and yt (formed in FP64) in place of
// xt and yt, and the footprint's place in its tile's patch.
struct __align__(8) T3Rec32 {
    float fx, fy, re, im;
    int place;  // patch row << 8 | patch column of the first cell
    int pad;
};
// One output frequency of FP32 data: fractional offsets, place and index.
struct __align__(16) T3Freq {
    float fx, fy;
    int place;
    int orig;
};

// The pre-compensation factors exp(b D^2 ds^2) of every grid offset ds
// (FP64, stored as FP32 for the FP32 spread):
// tab[ds + off], ds in [-off, n - off).
__global__ void k_t3_table(float *__restrict__ tab, int n, int off, double bD2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double d = static_cast<double>(i - off);
    tab[i] = static_cast<float>(exp(bD2 * d * d));
}

// Per point: the record fields and its tile; the rank within the tile from
// the tile's counter.
template <typename C2, typename Rec>
__global__ void k_t3_prep(const double *__restrict__ x, const double *__restrict__ y, const C2 *__restrict__ f,
                          long long n, Params P, int tiles_x, Rec *__restrict__ tmp, int2 *__restrict__ tile_rank,
                          unsigned *__restrict__ counts) {
    const long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (p >= n) return;
    const double xs = x[p] / P.kx, ys = y[p] / P.ky;  // :245-246
    const double arg = P.sb * xs + P.tb * ys;
    double sa, ca;
    sincos(arg, &sa, &ca);
    const double fr = static_cast<double>(f[p].x), fi = static_cast<double>(f[p].y);
    const double re = (fr * ca + fi * sa) * P.fact, im = (fi * ca - fr * sa) * P.fact;
    const double xt = (xs - P.xb) / P.Dx, yt = (ys - P.yb) / P.Dy;
    Rec r;
    const int i0 = static_cast<int>(floor(P.Mrx / 2 + xt)) - P.ms, j0 = static_cast<int>(floor(P.Mry / 2 + yt)) - P.ms;
    const int row = wrap(j0, P.Mry), col = wrap(i0, P.Mrx);
    if constexpr (sizeof(C2) == sizeof(double2)) {
        r.i0 = i0;
        r.j0 = j0;
        r.re = re;
        r.im = im;
        r.xt = xt;
        r.yt = yt;
    } else {
        r.re = static_cast<float>(re);
        r.im = static_cast<float>(im);
        r.fx = static_cast<float>(xt - floor(xt));
        r.fy = static_cast<float>(yt - floor(yt));
        r.place = (row % kT3Tile) << 8 | (col % kT3Tile);
        r.pad = 0;
    }
    const int tile = (row / kT3Tile) * tiles_x + col / kT3Tile;
    tmp[p] = r;
    tile_rank[p] = make_int2(tile, static_cast<int>(atomicAdd(counts + tile, 1u)));
}

// Per output frequency of FP32 data (:163-172, :189): the record, its tile
// and rank, and the factor that finishes it -- the post-compensation times
// the centres' phase -- in FP64.
__global__ void k_t3_prep_freq(const double *__restrict__ s, const double *__restrict__ t, long long n, Params P,
                               int tiles_x, T3Freq *__restrict__ tmp, int2 *__restrict__ tile_rank,
                               unsigned *__restrict__ counts, double2 *__restrict__ factor) {
    const long long k = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (k >= n) return;
    const double ss = s[k] * P.kx, ts = t[k] * P.ky;                                      // :247-248
    const double us = P.Mrx / 2 + (ss - P.sb), ut = P.Mry / 2 + (ts - P.tb);  // Ds = Dt = 1
    const double fs = floor(us), ft = floor(ut);
    const int col = wrap(static_cast<long long>(fs) - P.ms + P.Mrx / 2, P.Mrx);
    const int row = wrap(static_cast<long long>(ft) - P.ms + P.Mry / 2, P.Mry);
    T3Freq r;
    r.fx = static_cast<float>(us - fs);
    r.fy = static_cast<float>(ut - ft);
    r.place = (row % kT3Tile) << 8 | (col % kT3Tile);
    r.orig = static_cast<int>(k);
    const int tile = (row / kT3Tile) * tiles_x + col / kT3Tile;
    tmp[k] = r;
    tile_rank[k] = make_int2(tile, static_cast<int>(atomicAdd(counts + tile, 1u)));
    double tmp1 = P.Dy * (ts - P.tb);
    tmp1 = tmp1 * tmp1;
    double tmp2 = P.Dx * (ss - P.sb);
    tmp2 = tmp2 * tmp2;
    const double comp = exp(P.b * (tmp1 + tmp2));                 // :170-172
    const double arg = (ss - P.sb) * P.xb + (ts - P.tb) * P.yb;   // :189
    double sa, ca;
    sincos(arg, &sa, &ca);
    factor[k] = make_double2(ca * comp, sa * comp);
}

// One CTA a set (points, frequencies): exclusive scan of the tile counts into
// starts, and of the work items per tile; counts[ntiles] receives the number of
// work items.  Serial in the tiles (1 us per 1024), so both sets go at once: on
// 1.4 * 10^9 cells a second scan took 4.5 ms of 220.
struct T3Set {
    unsigned *counts, *starts, *item_starts;
    unsigned item;
};
__global__ void __launch_bounds__(1024) k_t3_scan(const T3Set s0, const T3Set s1, int ntiles) {
    const T3Set &set = blockIdx.x ? s1 : s0;
    unsigned *__restrict__ const counts = set.counts, *__restrict__ const starts = set.starts;
    unsigned *__restrict__ const item_starts = set.item_starts;
    const unsigned item = set.item;
    __shared__ unsigned s_pts[32], s_items[32];
    __shared__ unsigned carry_pts, carry_items;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) carry_pts = carry_items = 0;
    __syncthreads();
    for (int base = 0; base < ntiles; base += 1024) {
        const int i = base + tid;
        const unsigned c = i < ntiles ? counts[i] : 0u;
        const unsigned it = (c + item - 1) / item;
        unsigned a = c, b = it;  // inclusive warp scans
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned ua = __shfl_up_sync(0xffffffffu, a, o), ub = __shfl_up_sync(0xffffffffu, b, o);
            if (lane >= o) {
                a += ua;
                b += ub;
            }
        }
        if (lane == 31) {
            s_pts[warp] = a;
            s_items[warp] = b;
        }
        __syncthreads();
        if (warp == 0) {
            unsigned wa = s_pts[lane], wb = s_items[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned ua = __shfl_up_sync(0xffffffffu, wa, o), ub = __shfl_up_sync(0xffffffffu, wb, o);
                if (lane >= o) {
                    wa += ua;
                    wb += ub;
                }
            }
            s_pts[lane] = wa;
            s_items[lane] = wb;
        }
        __syncthreads();
        const unsigned before_pts = carry_pts + (warp ? s_pts[warp - 1] : 0u) + a - c;
        const unsigned before_items = carry_items + (warp ? s_items[warp - 1] : 0u) + b - it;
        if (i < ntiles) {
            starts[i] = before_pts;
            item_starts[i] = before_items;
        }
        __syncthreads();
        if (tid == 0) {
            carry_pts += s_pts[31];
            carry_items += s_items[31];
        }
        __syncthreads();
    }
    if (tid == 0) counts[ntiles] = carry_items;
}

// Records to their tile's range; the tile's work items {tile, first, count}.
template <typename Rec>
__global__ void k_t3_scatter(const Rec *__restrict__ tmp, const int2 *__restrict__ tile_rank, long long n,
                             const unsigned *__restrict__ starts, Rec *__restrict__ recs) {
    const long long p = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (p >= n) return;
    const int2 tr = tile_rank[p];
    recs[starts[tr.x] + static_cast<unsigned>(tr.y)] = tmp[p];
}

__global__ void k_t3_items(const unsigned *__restrict__ counts, const unsigned *__restrict__ starts,
                           const unsigned *__restrict__ item_starts, int ntiles, unsigned item,
                           int4 *__restrict__ items) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    const unsigned c = counts[t];
    for (unsigned k = 0; k * item < c; ++k)
        items[item_starts[t] + k] = make_int4(t, static_cast<int>(starts[t] + k * item),
                                              static_cast<int>(min(item, c - k * item)), 0);
}

// Dynamic shared memory of an FP64 spreading CTA: the patch, then B points'
// row and column weights, values and patch origins.
__host__ __device__ inline size_t t3_spread_smem(int W, int B) {
    const size_t PP = static_cast<size_t>(kT3Tile + W - 1);
    return (PP * PP * 2 + static_cast<size_t>(B) * (2 * W + 2)) * sizeof(double) +
           static_cast<size_t>(B) * sizeof(int2) + 16;
}

__global__ void __launch_bounds__(kT3Warps * 32)
    k_t3_spread(const T3Rec *__restrict__ recs, const int4 *__restrict__ items, const unsigned *__restrict__ n_items,
                Params P, int tiles_x, int B, double *__restrict__ grid) {
    extern __shared__ __align__(16) unsigned char t3_smem[];
    const int it = blockIdx.x;
    if (it >= static_cast<int>(*n_items)) return;
    const int4 item = items[it];
    const int W = 2 * P.ms + 1, PP = kT3Tile + W - 1;
    double *patch = reinterpret_cast<double *>(t3_smem);   // PP x PP complex, row-major
    double *wgt = patch + 2 * PP * PP;                     // per point: W row weights, then W column weights
    double *pval = wgt + 2 * B * W;                        // per point: the value
    int2 *pinfo = reinterpret_cast<int2 *>(pval + 2 * B);  // per point: patch row, column of its first cell
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < 2 * PP * PP; i += blockDim.x) patch[i] = 0.0;
    const int tr0 = (item.x / tiles_x) * kT3Tile, tc0 = (item.x % tiles_x) * kT3Tile;  // tile origin (wrapped)
    for (int b0 = 0; b0 < item.z; b0 += B) {
        const int nb = min(B, item.z - b0);
        __syncthreads();  // the previous batch's weights are consumed (and the patch zeroed)
        // per point: its patch origin and value; weights: point q, k < W rows
        // then W columns (:61-74), FP64 exponentials
        for (int q = tid; q < nb; q += blockDim.x) {
            const T3Rec &r = recs[item.y + b0 + q];
            pinfo[q] = make_int2(wrap(r.j0, P.Mry) - tr0, wrap(r.i0, P.Mrx) - tc0);
            pval[2 * q] = r.re;
            pval[2 * q + 1] = r.im;
        }
        for (int e = tid; e < nb * 2 * W; e += blockDim.x) {
            const int q = e / (2 * W), k = e - q * 2 * W;
            const T3Rec &r = recs[item.y + b0 + q];
            const bool row = k < W;
            const int kk = row ? k : k - W;
            const int ds = row ? r.j0 + kk - P.Mry / 2 : r.i0 + kk - P.Mrx / 2;  // dsj or dsi (:61-74)
            const double d = static_cast<double>(ds);
            const double t = row ? r.yt : r.xt;
            const double D = row ? P.Dy : P.Dx;
            wgt[q * 2 * W + k] = exp(P.b * D * D * d * d - P.t1 * (t - d) * (t - d));
        }
        __syncthreads();
        for (int q = 0; q < nb; ++q) {
            // footprint origin in the patch: the tile offset of the first cell
            const int2 o = pinfo[q];
            const int lr = o.x, lc = o.y;
            const double *wr = wgt + q * 2 * W, *wc = wr + W;
            const double vr = pval[2 * q], vi = pval[2 * q + 1];
            // this lane's columns c = lane + 32 m of the footprint: v * wc(c)
            for (int c0 = 0; c0 < W; c0 += 32) {
                const int c = c0 + lane;
                if (c >= W) continue;
                const double ax = vr * wc[c], ay = vi * wc[c];
                double *col = patch + 2 * (lc + c);
#pragma unroll 4
                for (int k = (warp - lr % kT3Warps + kT3Warps) % kT3Warps; k < W; k += kT3Warps) {
                    double *cell = col + 2 * (lr + k) * PP;  // patch row lr + k = warp (mod 8)
                    const double w = wr[k];
                    cell[0] += ax * w;
                    cell[1] += ay * w;
                }
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < PP * PP; i += blockDim.x) {
        const double ax = patch[2 * i], ay = patch[2 * i + 1];
        if (ax == 0.0 && ay == 0.0) continue;
        const int pr = i / PP, pc = i - pr * PP;
        double *g = grid + 2 * (static_cast<size_t>(wrap(tr0 + pr, P.Mry)) * P.Mrx + wrap(tc0 + pc, P.Mrx));
        atomicAdd(g, ax);
        atomicAdd(g + 1, ay);
    }
}

// ---------------------------------------------------------------------------
// FP32 data: both directions as dense products over a tile's patch, PR rows x
// PC columns (the patch edge rounded up to the register tiles), the weights
// zero outside their window.
//
// Spread: thread (i, j) holds patch rows 8i .. 8i+7 x columns 4j .. 4j+3 in
// registers and adds the points' outer products, 32 points' Gaussian factors
// (FP32, on exact arguments) in shared memory at a time and the next 32
// evaluated beside them.  The pre-compensation exp(b (Dy^2 dsj^2 + Dx^2 dsi^2))
// (:61-74) belongs to the grid cell, not to the point: it multiplies the
// finished patch (no footprint of a point wraps: |ds| <= M/4 + ms < M/2, since
// M >= 4.4 msp).  Half the products are with padding (39 of 54 rows and
// columns carry weights at eps 1e-6), and it is still bound by FP32 FMAs and
// the operand loads beside them; a read-modify-write of a patch in shared
// memory cost 24 bytes a product: 652 -> 88 us for 2 * 10^5 points, W = 39.
// ---------------------------------------------------------------------------
constexpr int kT3Batch = 32;    // points whose weights are in shared memory at a time
constexpr int kT3Freqs = 64;    // frequencies of a gather product
constexpr long long kT3Slice = 1LL << 24;  // frequencies binned at a time (0.9 GB of work buffers)

__host__ __device__ constexpr int round_up(int v, int m) { return (v + m - 1) / m * m; }
// Register tiles cover the patch; whole warps.  Rows of shared arrays are
// padded against bank conflicts.
struct T3Shape {
    int PR, PC;         // patch rows (a multiple of 8) and columns (of 4)
    int spread_threads, gather_threads;
    int spread_smem, gather_smem;
};
inline T3Shape t3_shape(int W) {
    T3Shape h;
    const int pp = kT3Tile + W - 1;
    h.PR = round_up(pp, 8);
    h.PC = round_up(pp, 4);
    h.spread_threads = round_up(h.PR / 8 * (h.PC / 4), 32);
    h.gather_threads = round_up(kT3Freqs / 8 * (h.PR / 4), kT3Freqs);
    h.spread_smem = 2 * kT3Batch * ((h.PR + 4) + 2 * (h.PC + 2)) * 4;
    // the patch, column by column; column and row weights of the frequencies
    // (the partial sums take the column weights' place)
    h.gather_smem = (h.PC * 2 * (h.PR + 2) + (h.PC + h.PR) * kT3Freqs) * 4;
    return h;
}

// MAXT threads, MINB CTAs an SM: (128, 4) up to W = 41, (448, 1) above.
template <int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    k_t3_spread_f32(const T3Rec32 *__restrict__ recs, const int4 *__restrict__ items,
                    const unsigned *__restrict__ n_items, Params P, int tiles_x, int PR, int PC,
                    const float *__restrict__ prex, int tabo_x, const float *__restrict__ prey, int tabo_y,
                    float2 *__restrict__ grid) {
    extern __shared__ __align__(16) unsigned char t3_smem[];
    if (blockIdx.x >= *n_items) return;
    const int4 item = items[blockIdx.x];
    const int W = 2 * P.ms + 1, SR = PR + 4, SC = PC + 2;
    float *wr0 = reinterpret_cast<float *>(t3_smem);                       // [2][point][SR] row weights
    float2 *vc0 = reinterpret_cast<float2 *>(wr0 + 2 * kT3Batch * SR);     // [2][point][SC] value times column weight
    const float t1f = static_cast<float>(P.t1), msf = static_cast<float>(P.ms);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    const int i8 = tid / (PC / 4), j4 = tid - i8 * (PC / 4);
    const bool on = i8 < PR / 8;
    // weights of points b0 .. b0 + 31: a lane takes one point, a warp every
    // `warps`th row and column of the patch
    auto prepare = [&](int b0, float *wr, float2 *vc) {
        T3Rec32 r{};
        r.place = 1 << 20;  // no point: every row is outside its window
        if (b0 + lane < item.z) r = recs[item.y + b0 + lane];
        const int lr = r.place >> 8, lc = r.place & 255;
        for (int k = warp; k < PR; k += warps) {
            const int a = k - lr;  // footprint row
            const float g = r.fy + (msf - static_cast<float>(a));
            const float w = expf(-t1f * g * g);
            wr[lane * SR + k] = static_cast<unsigned>(a) < static_cast<unsigned>(W) ? w : 0.f;
        }
        for (int k = warp; k < PC; k += warps) {
            const int a = k - lc;
            const float g = r.fx + (msf - static_cast<float>(a));
            const float w = static_cast<unsigned>(a) < static_cast<unsigned>(W) ? expf(-t1f * g * g) : 0.f;
            vc[lane * SC + k] = make_float2(r.re * w, r.im * w);
        }
    };
    float2 acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = make_float2(0.f, 0.f);
    prepare(0, wr0, vc0);
    __syncthreads();
    int buf = 0;
    for (int b0 = 0; b0 < item.z; b0 += kT3Batch, buf ^= 1) {
        const int nb = min(kT3Batch, item.z - b0);
        if (b0 + kT3Batch < item.z)
            prepare(b0 + kT3Batch, wr0 + (buf ^ 1) * kT3Batch * SR, vc0 + (buf ^ 1) * kT3Batch * SC);
        if (on) {
            const float4 *w4 = reinterpret_cast<const float4 *>(wr0 + buf * kT3Batch * SR + 8 * i8);
            const float4 *v4 = reinterpret_cast<const float4 *>(vc0 + buf * kT3Batch * SC + 4 * j4);
            for (int q = 0; q < nb; ++q, w4 += SR / 4, v4 += SC / 2) {
                const float4 wa = w4[0], wb = w4[1], va = v4[0], vb = v4[1];
                const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
                const float2 v[4] = {make_float2(va.x, va.y), make_float2(va.z, va.w), make_float2(vb.x, vb.y),
                                     make_float2(vb.z, vb.w)};
#pragma unroll
                for (int r = 0; r < 8; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[r][c] = __ffma2_rn(v[c], make_float2(w[r], w[r]), acc[r][c]);
            }
        }
        __syncthreads();  // this batch's weights are consumed, the next one's there
    }
    if (!on) return;
    // two cells an atomic: the grid's sides are even, so a pair of columns
    // never straddles its edge and lies on 16 bytes.  What lies beyond the
    // grid's edge belongs to no footprint.
    const int row0 = (item.x / tiles_x) * kT3Tile + 8 * i8, col0 = (item.x % tiles_x) * kT3Tile + 4 * j4;
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
        if (col0 + c >= P.Mrx) continue;
        const float px0 = prex[col0 + c - P.Mrx / 2 + tabo_x], px1 = prex[col0 + c + 1 - P.Mrx / 2 + tabo_x];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float2 a = acc[r][c], b = acc[r][c + 1];
            if (row0 + r >= P.Mry || (a.x == 0.f && a.y == 0.f && b.x == 0.f && b.y == 0.f)) continue;
            const float py = prey[row0 + r - P.Mry / 2 + tabo_y], p0 = py * px0, p1 = py * px1;
            float2 *g = grid + static_cast<size_t>(row0 + r) * P.Mrx + (col0 + c);
            atomicAdd(reinterpret_cast<float4 *>(g), make_float4(a.x * p0, a.y * p0, b.x * p1, b.y * p1));
        }
    }
}

// Gather: Y[k][r] = sum_c wc_k[c] G[r][c] for 64 frequencies of one tile at a
// time, thread (i, j) holding frequencies 8i .. 8i+7 x rows 4j .. 4j+3 (real
// and imaginary) in registers; then F_k = sum_r wr_k[r] Y[k][r] over the row
// groups through shared memory, finished in FP64.  The shift's (-1)^(i+j)
// (:147-148) is a sign per column and per row.  347 -> 83 us for 1.5 * 10^5
// frequencies, W = 39, where a warp per frequency re-read 12 KB of the grid.
template <int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    k_t3_gather_f32(const T3Freq *__restrict__ recs, const int4 *__restrict__ items,
                    const unsigned *__restrict__ n_items, Params P, int tiles_x, int PR, int PC,
                    const float2 *__restrict__ grid, const double2 *__restrict__ factor, float2 *__restrict__ F) {
    extern __shared__ __align__(16) unsigned char t3_smem[];
    if (blockIdx.x >= *n_items) return;
    const int4 item = items[blockIdx.x];
    const int W = 2 * P.ms + 1, SR = PR + 2;
    float2 *G = reinterpret_cast<float2 *>(t3_smem);  // [column][SR]
    float *wc = reinterpret_cast<float *>(G + PC * SR);  // [column][64]
    float *wr = wc + PC * kT3Freqs;                      // [row][64]
    float2 *part = reinterpret_cast<float2 *>(wc);       // [row group][64], after the products
    const float t1f = static_cast<float>(P.t1), msf = static_cast<float>(P.ms);
    const int tid = threadIdx.x;
    const int tr0 = (item.x / tiles_x) * kT3Tile, tc0 = (item.x % tiles_x) * kT3Tile;
    for (int r = tid >> 5; r < PR; r += blockDim.x >> 5) {
        const float2 *src = grid + static_cast<size_t>((tr0 + r) % P.Mry) * P.Mrx;
        for (int c = tid & 31; c < PC; c += 32) G[c * SR + r] = src[(tc0 + c) % P.Mrx];
    }
    const int i8 = tid % (kT3Freqs / 8), j4 = tid / (kT3Freqs / 8);
    const bool on = j4 < PR / 4;
    const int k = tid % kT3Freqs;  // the frequency this thread prepares and finishes
    for (int b0 = 0; b0 < item.z; b0 += kT3Freqs) {
        T3Freq rec{};
        rec.place = 1 << 20;  // none: every row is outside its window
        if (b0 + k < item.z) rec = recs[item.y + b0 + k];
        __syncthreads();  // the previous batch's sums are consumed (and the patch stored)
        // FP32 Gaussians on exact arguments; tiles start on even cells and the
        // grid's sides are even, so a cell's parity is its patch column's (row's)
        for (int x = tid / kT3Freqs; x < PC + PR; x += blockDim.x / kT3Freqs) {
            const bool col = x < PC;
            const int at = col ? x : x - PC, a = at - (col ? rec.place & 255 : rec.place >> 8);
            const float g = (col ? rec.fx : rec.fy) - (static_cast<float>(a) - msf);
            float w = static_cast<unsigned>(a) < static_cast<unsigned>(W) ? expf(-t1f * g * g) : 0.f;
            if (at & 1) w = -w;
            wc[x * kT3Freqs + k] = w;  // wr follows wc
        }
        __syncthreads();
        float2 acc[8][4];
        if (on) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
#pragma unroll
                for (int r = 0; r < 4; ++r) acc[q][r] = make_float2(0.f, 0.f);
            const float4 *a4 = reinterpret_cast<const float4 *>(wc + 8 * i8);
            const float4 *g4 = reinterpret_cast<const float4 *>(G + 4 * j4);
#pragma unroll 2
            for (int c = 0; c < PC; ++c, a4 += kT3Freqs / 4, g4 += SR / 2) {
                const float4 wa = a4[0], wb = a4[1], ga = g4[0], gb = g4[1];
                const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
                const float2 v[4] = {make_float2(ga.x, ga.y), make_float2(ga.z, ga.w), make_float2(gb.x, gb.y),
                                     make_float2(gb.z, gb.w)};
#pragma unroll
                for (int q = 0; q < 8; ++q)
#pragma unroll
                    for (int r = 0; r < 4; ++r) acc[q][r] = __ffma2_rn(v[r], make_float2(w[q], w[q]), acc[q][r]);
            }
        }
        __syncthreads();  // the column weights are consumed
        if (on) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                float2 s = make_float2(0.f, 0.f);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float w = wr[(4 * j4 + r) * kT3Freqs + 8 * i8 + q];
                    s = __ffma2_rn(acc[q][r], make_float2(w, w), s);
                }
                part[j4 * kT3Freqs + 8 * i8 + q] = s;
            }
        }
        __syncthreads();
        if (tid < kT3Freqs && b0 + k < item.z) {
            float2 s = make_float2(0.f, 0.f);
            for (int j = 0; j < PR / 4; ++j) {
                const float2 v = part[j * kT3Freqs + k];
                s.x += v.x;
                s.y += v.y;
            }
            const double2 f = factor[rec.orig];
            const double a0 = static_cast<double>(s.x), a1 = static_cast<double>(s.y);
            F[rec.orig] = make_float2(static_cast<float>(a0 * f.x + a1 * f.y), static_cast<float>(a1 * f.x - a0 * f.y));
        }
    }
}

// ---------------------------------------------------------------------------
// Gathering (:156-194).  The Gaussian weight of tap (r, c) is
// exp(-t1 (difs - npj)^2) exp(-t1 (dift - npi)^2) and the shift's (-1)^(i+j)
// (:147-148) is (-1)^i (-1)^j, so both factor per column and per row.  A
// warp owns 32 output frequencies: each lane sets up one of them (FP64:
// scaling, cell, fractional offsets, the post-compensation and the centres'
// phase), then the warp sums the footprints one frequency after the other --
// lane l owns footprint columns l and l + 32 and runs down the rows -- and
// the lane that owns the frequency finishes it.  FP64 data.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
    k_t3_gather(const double *__restrict__ s, const double *__restrict__ t, long long n, Params P,
                const double2 *__restrict__ grid, double2 *__restrict__ F) {
    const long long k0 = (blockIdx.x * static_cast<long long>(kWarpsPerBlock) + (threadIdx.x >> 5)) * 32;
    const int lane = threadIdx.x & 31;
    if (k0 >= n) return;
    const long long k = k0 + lane;
    const bool mine = k < n;
    // this lane's frequency (:163-172, :189)
    double ss = 0.0, ts = 0.0;
    if (mine) {
        ss = s[k] * P.kx;  // :247-248
        ts = t[k] * P.ky;
    }
    const double us = P.Mrx / 2 + (ss - P.sb), ut = P.Mry / 2 + (ts - P.tb);  // Ds = Dt = 1
    const double fs = floor(us), ft = floor(ut);
    const double difs = us - fs, dift = ut - ft;
    const int ifirst = wrap(static_cast<long long>(fs) - P.ms + P.Mrx / 2, P.Mrx);
    const int jfirst = wrap(static_cast<long long>(ft) - P.ms + P.Mry / 2, P.Mry);
    const int W = 2 * P.ms + 1;
    const double t1 = P.t1;
    double res0 = 0.0, res1 = 0.0;
    const int nk = static_cast<int>(min(32LL, n - k0));
    for (int o = 0; o < nk; ++o) {
        const double ds = __shfl_sync(0xffffffffu, difs, o), dt = __shfl_sync(0xffffffffu, dift, o);
        const int i0 = __shfl_sync(0xffffffffu, ifirst, o), j0 = __shfl_sync(0xffffffffu, jfirst, o);
        // row weights of rows lane + 32 m (the grid has even sides: the
        // wrapped row's parity is that of j0 + r)
        double wrow[3];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            const int r = lane + 32 * m;
            const double g = dt - static_cast<double>(r - P.ms);
            const double e = r < W ? exp(-t1 * g * g) : 0.0;
            wrow[m] = ((j0 + r) & 1) ? -e : e;
        }
        double acc0 = 0.0, acc1 = 0.0;
        for (int c0 = 0; c0 < W; c0 += 32) {
            const int c = c0 + lane;
            const bool on = c < W;
            const int cc = on ? c : 0;
            const int i = i0 + cc >= P.Mrx ? i0 + cc - P.Mrx : i0 + cc;
            const double g = ds - static_cast<double>(cc - P.ms);
            const double es = exp(-t1 * g * g);
            // lanes past the footprint read a valid cell and weigh it by 0
            const double wcol = on ? (((i0 + cc) & 1) ? -es : es) : 0.0;
            const double2 *col = grid + i;
            double s0 = 0.0, s1 = 0.0;
            int j = j0;
#pragma unroll
            for (int m = 0; m < 3; ++m) {  // footprint rows 32 m .. 32 m + 31
                const int rn = min(32, W - 32 * m);
#pragma unroll 8
                for (int rr = 0; rr < rn; ++rr) {
                    const double wr = __shfl_sync(0xffffffffu, wrow[m], rr);
                    const double2 v = col[static_cast<size_t>(j) * P.Mrx];
                    s0 += v.x * wr;
                    s1 += v.y * wr;
                    j = j + 1 == P.Mry ? 0 : j + 1;
                }
            }
            acc0 += s0 * wcol;
            acc1 += s1 * wcol;
        }
        for (int x = 16; x > 0; x >>= 1) {
            acc0 += __shfl_xor_sync(0xffffffffu, acc0, x);
            acc1 += __shfl_xor_sync(0xffffffffu, acc1, x);
        }
        if (lane == o) {
            res0 = acc0;
            res1 = acc1;
        }
    }
    if (mine) {
        double tmp1 = P.Dy * (ts - P.tb);
        tmp1 = tmp1 * tmp1;
        double tmp2 = P.Dx * (ss - P.sb);
        tmp2 = tmp2 * tmp2;
        const double comp = exp(P.b * (tmp1 + tmp2));                 // :170-172
        const double arg = (ss - P.sb) * P.xb + (ts - P.tb) * P.yb;   // :189
        double sa, ca;
        sincos(arg, &sa, &ca);
        double2 out;
        out.x = (res0 * ca + res1 * sa) * comp;
        out.y = (res1 * ca - res0 * sa) * comp;
        F[k] = out;
    }
}

int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return NFFT2D_OK;
    return e == cudaErrorMemoryAllocation ? NFFT2D_ERR_OOM : NFFT2D_ERR_CUDA;
}

#define T3_CUDA(expr)                                   \
    do {                                                \
        const int st_ = cuda_status(expr);              \
        if (st_ != NFFT2D_OK) return st_;               \
    } while (0)

// Extents of both sets, {min, max} of x, y, s, t, with one read-back.
int minmax(const double *x, const double *y, long long nx, const double *s, const double *t, long long ns,
           unsigned long long *d_mm, cudaStream_t st, int sms, double out[8]) {
    const unsigned long long init[8] = {~0ull, 0ull, ~0ull, 0ull, ~0ull, 0ull, ~0ull, 0ull};
    T3_CUDA(cudaMemcpyAsync(d_mm, init, sizeof init, cudaMemcpyHostToDevice, st));
    const long long n = std::max(nx, ns);
    const int blocks = static_cast<int>(std::max<long long>(1, std::min<long long>((n + 1023) / 1024, sms)));
    k_minmax2<<<dim3(blocks, 2), kMinmaxThreads, 0, st>>>(x, y, nx, s, t, ns, d_mm);
    T3_CUDA(cudaGetLastError());
    unsigned long long h[8];
    T3_CUDA(cudaMemcpyAsync(h, d_mm, sizeof h, cudaMemcpyDeviceToHost, st));
    T3_CUDA(cudaStreamSynchronize(st));
    for (int i = 0; i < 8; ++i) out[i] = ord_value(h[i]);
    return NFFT2D_OK;
}

struct Scratch {
    cudaStream_t st;
    void *mm = nullptr, *grid = nullptr;
    cufftHandle plan = 0;
    bool plan_ok = false;
    ~Scratch() {
        if (plan_ok) {
            cudaStreamSynchronize(st);  // no FFT in flight when the handle goes back to the pool
            nfft2d::pooled_plan_release(plan);
        }
        if (grid) cudaFreeAsync(grid, st);
        if (mm) cudaFreeAsync(mm, st);
    }
};

}  // namespace

extern "C" int nfft2d_nufft3_2d(const double *x, const double *y, const double *s, const double *t, const void *f,
                                void *F, double eps, long long len_in, long long len_out, int precision,
                                void *stream) {
    if (!x || !y || !s || !t || !f || !F || len_in < 1 || len_out < 1) return NFFT2D_ERR_INVALID_ARG;
    if (!(eps > 0 && eps < 1)) return NFFT2D_ERR_INVALID_ARG;
    if (precision != NFFT2D_F32 && precision != NFFT2D_F64) return NFFT2D_ERR_INVALID_ARG;
    if (len_in > (1LL << 40) || len_out > (1LL << 40)) return NFFT2D_ERR_INVALID_ARG;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    Scratch S{st};
    int dev = 0, sms = 0;
    T3_CUDA(cudaGetDevice(&dev));
    T3_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    T3_CUDA(cudaMallocAsync(&S.mm, 8 * sizeof(unsigned long long), st));
    double ext[8];
    const int rc = minmax(x, y, len_in, s, t, len_out, static_cast<unsigned long long *>(S.mm), st, sms, ext);
    if (rc != NFFT2D_OK) return rc;
    for (double v : ext)
        if (!std::isfinite(v)) return NFFT2D_ERR_NONFINITE;
    const double *exy = ext, *est = ext + 4;
    // :214-232 (the reductions start from -+FLT_MAX, which finite data within
    // range never leaves)
    double Max_x = exy[1], min_x = exy[0], Max_y = exy[3], min_y = exy[2];
    double Max_s = est[1], min_s = est[0], Max_t = est[3], min_t = est[2];
    double xb = (Max_x + min_x) / 2, X1 = std::fabs(Max_x - xb);
    double yb = (Max_y + min_y) / 2, Y1 = std::fabs(Max_y - yb);
    double sb = (Max_s + min_s) / 2, Sx = std::fabs(Max_s - sb);
    double tb = (Max_t + min_t) / 2, Ty = std::fabs(Max_t - tb);
    if (!(X1 > 0) || !(Y1 > 0)) return NFFT2D_ERR_INVALID_ARG;  // all points on one line: no scale
    const double R = 2.2;
    double msp = 2 + 2 * (R * R) * (-std::log(eps / 76)) / (kPi * (R * R - 2));  // :235
    const double mrx = 2 * std::ceil((X1 * Sx / kPi) * R * R + R * msp);         // :237-238
    const double mry = 2 * std::ceil((Y1 * Ty / kPi) * R * R + R * msp);
    if (!(mrx <= 65536) || !(mry <= 65536) || mrx * mry > 1.5e9) return NFFT2D_ERR_UNSUPPORTED;
    Params P{};
    P.Mrx = static_cast<int>(mrx);
    P.Mry = static_cast<int>(mry);
    P.Dx = 2 * kPi / P.Mrx;
    P.Dy = 2 * kPi / P.Mry;
    P.kx = X1 / (kPi / 2);
    P.ky = Y1 / (kPi / 2);
    Max_x = Max_x / P.kx;
    min_x = min_x / P.kx;
    P.xb = (Max_x + min_x) / 2;
    Max_s = Max_s * P.kx;
    min_s = min_s * P.kx;
    P.sb = (Max_s + min_s) / 2;
    Max_y = Max_y / P.ky;
    min_y = min_y / P.ky;
    P.yb = (Max_y + min_y) / 2;
    Max_t = Max_t * P.ky;
    min_t = min_t * P.ky;
    P.tb = (Max_t + min_t) / 2;
    P.b = (msp - 2) / (4 * kPi);
    P.t1 = 1 / (4 * P.b);
    msp = std::floor(msp - 2);
    P.ms = static_cast<int>(msp);
    const double f0 = 1. / (4. * kPi * P.b);
    P.fact = f0 * f0;

    const bool dbl = precision == NFFT2D_F64;
    const int W = 2 * P.ms + 1;
    if (W > 96) return NFFT2D_ERR_UNSUPPORTED;  // the gather's lanes hold at most 96 row weights
    const size_t rb = dbl ? sizeof(double) : sizeof(float);
    const T3Shape shape = t3_shape(W);
    int B = 32;  // points per weight batch of the FP64 spread
    while (dbl && B > 4 && t3_spread_smem(W, B) > nfft2d::kMaxSmem) B /= 2;
    const size_t smem = dbl ? t3_spread_smem(W, B) : shape.spread_smem;
    if (smem > nfft2d::kMaxSmem || shape.gather_smem > nfft2d::kMaxSmem) return NFFT2D_ERR_UNSUPPORTED;
    const size_t cells = static_cast<size_t>(P.Mrx) * P.Mry;
    const size_t csz = 2 * rb;
    const int tiles_x = (P.Mrx + kT3Tile - 1) / kT3Tile, tiles_y = (P.Mry + kT3Tile - 1) / kT3Tile;
    const long long ntiles = static_cast<long long>(tiles_x) * tiles_y;
    // FP32 work items: enough of them for each SM to hold several CTAs, a few
    // batches each (a spread item ends in a patch of atomics, a gather item
    // begins by reading one)
    auto item_of = [sms](long long n) {
        const long long v = n / (sms * 8LL) / 64 * 64;
        return static_cast<unsigned>(std::max(128LL, std::min<long long>(v, 512)));
    };
    // FP32 frequencies go in slices, which bounds their work buffers
    const long long slice = std::min(len_out, kT3Slice);
    const unsigned item_in = dbl ? kT3Item : item_of(len_in), item_out = item_of(slice);
    // a tile that has any has at least one item, a full one an item per item_in
    const long long max_items = std::min(ntiles, len_in) + len_in / item_in + 1;
    const long long max_items_out = std::min(ntiles, slice) + slice / item_out + 1;
    if (len_in > 0x7fffffffLL || max_items > 0x7fffffffLL) return NFFT2D_ERR_UNSUPPORTED;
    // work buffers: the grid; of the points and (FP32) of the frequencies the
    // records (unsorted, sorted), tile and rank, counts, starts, item starts,
    // items; the frequencies' factors; pre-compensation tables over ds in
    // [-off, off]: |ds| <= M/4 + ms + 1 for points inside the extents, off =
    // M/2 + ms + 2 leaves margin
    const int tabo_x = P.Mrx / 2 + P.ms + 2, tabo_y = P.Mry / 2 + P.ms + 2;
    size_t total = 0;
    auto take = [&](size_t bytes) {
        const size_t at = total;
        total += (bytes + 255) / 256 * 256;
        return at;
    };
    struct Bins {
        size_t tmp, recs, tr, counts, starts, istarts, items;
    };
    auto take_bins = [&](long long n, size_t rec, long long n_items) {
        Bins o;
        o.tmp = take(static_cast<size_t>(n) * rec);
        o.recs = take(static_cast<size_t>(n) * rec);
        o.tr = take(static_cast<size_t>(n) * sizeof(int2));
        o.starts = take(static_cast<size_t>(ntiles) * sizeof(unsigned));
        o.istarts = take(static_cast<size_t>(ntiles) * sizeof(unsigned));
        o.items = take(static_cast<size_t>(n_items) * sizeof(int4));
        return o;
    };
    const size_t off_grid = take(cells * csz);  // then the counts: one memset
    const size_t off_counts = take(2 * static_cast<size_t>(ntiles + 1) * sizeof(unsigned)), zeroed = total;
    Bins bi = take_bins(len_in, dbl ? sizeof(T3Rec) : sizeof(T3Rec32), max_items), bo{};
    bi.counts = off_counts;
    if (!dbl) bo = take_bins(slice, sizeof(T3Freq), max_items_out);
    bo.counts = off_counts + static_cast<size_t>(ntiles + 1) * sizeof(unsigned);
    const size_t off_factor = take(dbl ? 0 : static_cast<size_t>(slice) * sizeof(double2));
    const size_t off_tx = take(static_cast<size_t>(2 * tabo_x + 1) * sizeof(float));
    const size_t off_ty = take(static_cast<size_t>(2 * tabo_y + 1) * sizeof(float));
    T3_CUDA(cudaMallocAsync(&S.grid, total, st));
    unsigned char *base = static_cast<unsigned char *>(S.grid);
    T3_CUDA(cudaMemsetAsync(base + off_grid, 0, zeroed - off_grid, st));
    auto words = [&](size_t o) { return reinterpret_cast<unsigned *>(base + o); };
    // counting sort by tile of n records: scan (k_t3_scan), move, work items
    auto set_of = [&](const Bins &o, unsigned item) {
        return T3Set{words(o.counts), words(o.starts), words(o.istarts), item};
    };
    auto bin = [&](auto *rec, const Bins &o, long long n, unsigned item) -> cudaError_t {
        using Rec = std::remove_pointer_t<decltype(rec)>;
        cudaError_t e;
        k_t3_scatter<Rec><<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(
            reinterpret_cast<const Rec *>(base + o.tmp), reinterpret_cast<const int2 *>(base + o.tr), n, words(o.starts),
            reinterpret_cast<Rec *>(base + o.recs));
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        k_t3_items<<<static_cast<unsigned>((ntiles + 255) / 256), 256, 0, st>>>(
            words(o.counts), words(o.starts), words(o.istarts), static_cast<int>(ntiles), item,
            reinterpret_cast<int4 *>(base + o.items));
        return cudaGetLastError();
    };
    T3Freq *const freqs = reinterpret_cast<T3Freq *>(base + bo.tmp);  // FP32 only
    double2 *const factor = reinterpret_cast<double2 *>(base + off_factor);
    auto prep_freq = [&](long long at) -> cudaError_t {  // the slice from `at`
        const long long n = std::min(slice, len_out - at);
        k_t3_prep_freq<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(
            s + at, t + at, n, P, tiles_x, freqs, reinterpret_cast<int2 *>(base + bo.tr), words(bo.counts), factor);
        return cudaGetLastError();
    };
    const unsigned pb = static_cast<unsigned>((len_in + 255) / 256);
    int2 *tr = reinterpret_cast<int2 *>(base + bi.tr);
    const int4 *items = reinterpret_cast<const int4 *>(base + bi.items);
    // one CTA per possible work item; those beyond the device-side count return
    if (dbl) {
        T3Rec *tmp = reinterpret_cast<T3Rec *>(base + bi.tmp);
        k_t3_prep<double2, T3Rec><<<pb, 256, 0, st>>>(x, y, static_cast<const double2 *>(f), len_in, P, tiles_x, tmp, tr,
                                                     words(bi.counts));
        T3_CUDA(cudaGetLastError());
        k_t3_scan<<<1, 1024, 0, st>>>(set_of(bi, item_in), T3Set{}, static_cast<int>(ntiles));
        T3_CUDA(cudaGetLastError());
        T3_CUDA(bin(tmp, bi, len_in, item_in));
        T3_CUDA(nfft2d::allow_smem(k_t3_spread, static_cast<int>(smem)));
        k_t3_spread<<<static_cast<unsigned>(max_items), kT3Warps * 32, smem, st>>>(
            reinterpret_cast<const T3Rec *>(base + bi.recs), items, words(bi.counts) + ntiles, P, tiles_x, B,
            static_cast<double *>(S.grid));
    } else {
        T3Rec32 *tmp = reinterpret_cast<T3Rec32 *>(base + bi.tmp);
        float *prex = reinterpret_cast<float *>(base + off_tx), *prey = reinterpret_cast<float *>(base + off_ty);
        k_t3_table<<<(2 * tabo_x + 1 + 255) / 256, 256, 0, st>>>(prex, 2 * tabo_x + 1, tabo_x, P.b * P.Dx * P.Dx);
        k_t3_table<<<(2 * tabo_y + 1 + 255) / 256, 256, 0, st>>>(prey, 2 * tabo_y + 1, tabo_y, P.b * P.Dy * P.Dy);
        T3_CUDA(cudaGetLastError());
        k_t3_prep<float2, T3Rec32><<<pb, 256, 0, st>>>(x, y, static_cast<const float2 *>(f), len_in, P, tiles_x, tmp, tr,
                                                      words(bi.counts));
        T3_CUDA(cudaGetLastError());
        T3_CUDA(prep_freq(0));
        k_t3_scan<<<2, 1024, 0, st>>>(set_of(bi, item_in), set_of(bo, item_out), static_cast<int>(ntiles));
        T3_CUDA(cudaGetLastError());
        T3_CUDA(bin(tmp, bi, len_in, item_in));
        auto spread = shape.spread_threads <= 128 ? k_t3_spread_f32<128, 4> : k_t3_spread_f32<448, 1>;
        T3_CUDA(nfft2d::allow_smem(spread, static_cast<int>(smem)));
        spread<<<static_cast<unsigned>(max_items), shape.spread_threads, smem, st>>>(
            reinterpret_cast<const T3Rec32 *>(base + bi.recs), items, words(bi.counts) + ntiles, P, tiles_x, shape.PR,
            shape.PC, prex, tabo_x, prey, tabo_y, reinterpret_cast<float2 *>(base + off_grid));
    }
    T3_CUDA(cudaGetLastError());
    // :283-292 -- rows are Mry, the fast (column) dimension Mrx
    if (nfft2d::pooled_plan_2d(&S.plan, P.Mry, P.Mrx, dbl ? CUFFT_Z2Z : CUFFT_C2C) != CUFFT_SUCCESS)
        return NFFT2D_ERR_CUFFT;
    S.plan_ok = true;
    if (cufftSetStream(S.plan, st) != CUFFT_SUCCESS) return NFFT2D_ERR_CUFFT;
    const cufftResult fr =
        dbl ? cufftExecZ2Z(S.plan, static_cast<cufftDoubleComplex *>(S.grid), static_cast<cufftDoubleComplex *>(S.grid),
                           CUFFT_FORWARD)
            : cufftExecC2C(S.plan, static_cast<cufftComplex *>(S.grid), static_cast<cufftComplex *>(S.grid),
                           CUFFT_FORWARD);
    if (fr != CUFFT_SUCCESS) return NFFT2D_ERR_CUFFT;
    if (dbl) {
        const long long warps_out = (len_out + 31) / 32;  // 32 frequencies per warp
        const unsigned blk_out = static_cast<unsigned>((warps_out + kWarpsPerBlock - 1) / kWarpsPerBlock);
        k_t3_gather<<<blk_out, kWarpsPerBlock * 32, 0, st>>>(s, t, len_out, P, static_cast<const double2 *>(S.grid),
                                                             static_cast<double2 *>(F));
    } else {
        auto gather = shape.gather_threads <= 128 ? k_t3_gather_f32<128, 4> : k_t3_gather_f32<448, 1>;
        T3_CUDA(nfft2d::allow_smem(gather, shape.gather_smem));
        for (long long at = 0; at < len_out; at += slice) {
            const long long n = std::min(slice, len_out - at);
            if (at > 0) {  // the first slice's counts are scanned with the points'
                T3_CUDA(cudaMemsetAsync(words(bo.counts), 0, static_cast<size_t>(ntiles + 1) * sizeof(unsigned), st));
                T3_CUDA(prep_freq(at));
                k_t3_scan<<<1, 1024, 0, st>>>(set_of(bo, item_out), T3Set{}, static_cast<int>(ntiles));
                T3_CUDA(cudaGetLastError());
            }
            T3_CUDA(bin(freqs, bo, n, item_out));
            gather<<<static_cast<unsigned>(max_items_out), shape.gather_threads, shape.gather_smem, st>>>(
                reinterpret_cast<const T3Freq *>(base + bo.recs), reinterpret_cast<const int4 *>(base + bo.items),
                words(bo.counts) + ntiles, P, tiles_x, shape.PR, shape.PC, static_cast<const float2 *>(S.grid), factor,
                static_cast<float2 *>(F) + at);
            T3_CUDA(cudaGetLastError());
        }
    }
    T3_CUDA(cudaGetLastError());
    return cuda_status(cudaStreamSynchronize(st));
}
