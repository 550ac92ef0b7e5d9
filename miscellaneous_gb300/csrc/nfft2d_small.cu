// nfft2d_small.cu -- whole transforms of small FP32 plans in one launch.
//
// At 64^2 coefficients and 4096 points every stage of a transform runs 1 to 2
// us of work behind 4 to 12 us of launch, fill and dependent latency.  Here
// one cooperative kernel goes through all stages, with grid barriers where the
// separate kernels have launch boundaries; the grid stays in L2.
//
//   type 2: pad + band-column FFTs | row FFTs + halo | gather
//   type 1: zero, spread patches | add them | fold + row FFTs | columns + crop
//
// A kernel that runs so short is bound by fetching its instructions, by its
// chains of loads and by its barriers (1.5 us each): a version with the
// separate kernels' unrolled radix-16 FFT and register patches spent 2 to 6 us
// in each piece of straight-line code.  So everything here is a short loop --
// radix-4 FFTs of one warp, patches in shared memory, a row of taps an
// iteration --, a phase issues its global loads together, the loads and
// weights of the points come before the barrier that their grid waits for, and
// the warps are spread over all SMs (on the 16 of one cluster shared memory
// bound the gather and the spread: 18 and 26 us).  64^2 coefficients, 4096
// points, w 6, back to back: forward 14.7 us, adjoint 16.5; the separate kernels,
// each starting while the one before ends, 14.4 and 25.7.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "nfft2d_device.cuh"
#include "nfft2d_internal.h"
#include "nfft2d_kargs.cuh"
#include "nfft2d_tile_ops.cuh"

namespace nfft2d {
namespace {

constexpr int kSmallCtas = kGridCtas;
constexpr int kSmallThreads = 128;
constexpr int kSmallWarpsCta = kSmallThreads / 32;
constexpr int kSmallWarps = kSmallCtas * kSmallWarpsCta;
constexpr int kSmallSide = 512;    // longest FFT

struct SmallArgs {
    int N1, N2, logn1, logn2;
    float s;      // exponent sign
    int give_up;  // grid_wait's
    const float *d1, *d2;
    const float2 *tw1, *tw2;  // exp(-2 pi i m / n)
};

// Loads of what this kernel itself writes (never the read-only path).
__device__ __forceinline__ float2 ld_rw(const float2 *p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_rw4(const float2 *p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 mul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}

// Stockham FFT of one sequence of n = 2^logn elements by one warp, X_k =
// sum_m x_m exp(s 2 pi i m k / n), from `a` into the returned one of the
// buffers a and b: radix 4, one radix-2 stage first when logn is odd.  tw:
// exp(-2 pi i m / n) in shared memory.
__device__ __forceinline__ float2 *warp_fft(float2 *a, float2 *b, int logn, float s, const float2 *tw) {
    const int lane = threadIdx.x & 31, n = 1 << logn;
    int logl = 0;  // 2^logl: length of the transforms done so far
    if (logn & 1) {
        for (int i = lane; i < n / 2; i += 32) {
            const float2 x = a[i], y = a[i + n / 2];
            b[2 * i] = add(x, y);
            b[2 * i + 1] = sub(x, y);
        }
        __syncwarp();
        float2 *t = a;
        a = b;
        b = t;
        logl = 1;
    }
    for (; logl < logn; logl += 2) {
        for (int i = lane; i < n / 4; i += 32) {
            // butterfly i: j within the transforms of length 2^logl, k which
            const int j = i & ((1 << logl) - 1), m = j << (logn - logl - 2);
            float2 w1 = tw[m], w2 = tw[2 * m], w3 = tw[3 * m];
            w1.y *= -s, w2.y *= -s, w3.y *= -s;
            const float2 x0 = a[i], x1 = mul(a[i + n / 4], w1), x2 = mul(a[i + n / 2], w2), x3 = mul(a[i + 3 * (n / 4)], w3);
            const float2 t0 = add(x0, x2), t1 = sub(x0, x2), t2 = add(x1, x3), d = sub(x1, x3);
            const float2 t3 = make_float2(-s * d.y, s * d.x);  // s i (x1 - x3)
            float2 *o = b + ((i >> logl) << (logl + 2)) + j;
            o[0] = add(t0, t2);
            o[1 << logl] = add(t1, t3);
            o[2 << logl] = sub(t0, t2);
            o[3 << logl] = sub(t1, t3);
        }
        __syncwarp();
        float2 *t = a;
        a = b;
        b = t;
    }
    return a;
}

// Twiddles of both dimensions to shared memory (n1, then n2).
__device__ __forceinline__ void load_twiddles(float2 *tw, const SmallArgs &a) {
    const int n1 = 1 << a.logn1, n2 = 1 << a.logn2;
    for (int i = threadIdx.x; i < n1 + n2; i += kSmallThreads) tw[i] = i < n1 ? __ldg(a.tw1 + i) : __ldg(a.tw2 + (i - n1));
}

// Work items are split while there are warps without one: unit u of n * split
// takes its share of an item's batches of B points.
struct SmallUnit {
    int first, count, r0, c0;
};
__device__ __forceinline__ int small_split(int n) { return n > 0 ? max(1, min(8, kSmallWarps / n)) : 1; }
template <int B>
__device__ __forceinline__ SmallUnit small_unit(const int4 *__restrict__ chunks, int u, int units, int split,
                                                const Geom &g) {
    if (u >= units) return {0, 0, 0, 0};
    const int4 ch = __ldg(&chunks[u / split]);
    const int part = u % split, batches = (ch.z + B - 1) / B;
    const int b0 = batches * part / split, b1 = batches * (part + 1) / split;
    const int tr = ch.x / g.tiles2;
    return {ch.y + B * b0, max(0, min(ch.z, B * b1) - B * b0), tr * kRegTile, (ch.x - tr * g.tiles2) * kRegTile};
}

// A tile's patch in a warp's shared memory, as the TMA boxes of the plan's
// tensor map (compute_layout), and its points' weights.
template <int K>
struct SmallPatch {
    static constexpr int W = 2 * K + 1, KE = K + (K & 1), PR = kRegTile + 2 * K, COLS = kRegTile + 2 * KE;
    static constexpr int SW = spread_strip_width(K);
    static constexpr int PITCH = (COLS + 15) / 16 * 16 + (SW < kRegTile ? SW : 0);
    static constexpr int ELEMS = (PR * PITCH + 15) / 16 * 16;  // whole 128 bytes
    static constexpr int WROW = 33;                            // weights [tap][point], padded
    static constexpr int BYTES = ELEMS * 8 + (2 * W * WROW * 4 + 127) / 128 * 128;  // a warp's patch and weights
};

// Shared memory: the twiddles, then a warp's two FFT buffers or its patch.
constexpr int kTwBytes = (kSmallSide + kSmallCells / kSmallSide) * 8;  // the longest pair of sides
template <int K>
constexpr int small_warp_bytes() {
    return std::max(2 * kSmallSide * 8, SmallPatch<K>::BYTES);
}
template <int K>
constexpr int small_smem() {
    return kTwBytes + kSmallWarpsCta * small_warp_bytes<K>() + 128;
}

// A warp transforms one line at a time; band column bc of the N2 is grid column
// c and column j of the coefficients.
template <int K>
__global__ void __launch_bounds__(kSmallThreads)
    k_small_type2(const float2 *__restrict__ F, float2 *grid, const Rec32 *__restrict__ recs,
                  const int4 *__restrict__ chunks, float2 *__restrict__ out, const SmallArgs a,
                  const __grid_constant__ KArgs ka) {
    extern __shared__ unsigned char sm_raw[];
    unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(sm_raw) + 127) & ~uintptr_t(127));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, gw = wid * kSmallCtas + blockIdx.x;
    float2 *tw = reinterpret_cast<float2 *>(base);
    unsigned char *mine = base + kTwBytes + wid * small_warp_bytes<K>();
    float2 *b0 = reinterpret_cast<float2 *>(mine), *b1 = b0 + kSmallSide;
    const Geom &g = ka.g;
    const int n1 = g.n1, n2 = g.n2, H = g.H, N1 = a.N1, N2 = a.N2;
    float2 *const inner = grid + static_cast<size_t>(H) * g.C + H;  // cell (0, 0)
    load_twiddles(tw, a);
    __syncthreads();
    for (int bc = gw; bc < N2; bc += kSmallWarps) {  // band columns
        const int j = bc < N2 / 2 ? bc + N2 / 2 : bc - N2 / 2, c = bc < N2 / 2 ? bc : n2 - N2 + bc;
        const float s2 = __ldg(a.d2 + j);
#pragma unroll 4
        for (int r = lane; r < n1; r += 32) {
            // rows outside the band load the band's edge: no load waits behind a branch
            const int k1 = r < n1 / 2 ? r : r - n1, i = min(max(k1 + N1 / 2, 0), N1 - 1);
            const float sc = __ldg(a.d1 + i) * s2;
            const float2 f = __ldg(F + static_cast<size_t>(i) * N2 + j);
            b0[r] = k1 >= -N1 / 2 && k1 < N1 / 2 ? make_float2(f.x * sc, f.y * sc) : make_float2(0.f, 0.f);
        }
        __syncwarp();
        const float2 *x = warp_fft(b0, b1, a.logn1, a.s, tw);
        for (int r = lane; r < n1; r += 32) inner[static_cast<size_t>(r) * g.C + c] = x[r];
        __syncwarp();
    }
    if (!grid_barrier(ka.status, 1, a.give_up)) {
        grid_done(ka.status, true);
        return;
    }
    for (int r = gw; r < n1; r += kSmallWarps) {  // rows, with their halo images
        float2 *row = inner + static_cast<size_t>(r) * g.C;
#pragma unroll 4
        for (int c = lane; c < n2; c += 32) {
            const int k2 = c < n2 / 2 ? c : c - n2;
            const float2 v = ld_rw(row + c);  // only the band is from this transform
            b0[c] = k2 >= -N2 / 2 && k2 < N2 / 2 ? v : make_float2(0.f, 0.f);
        }
        __syncwarp();
        const float2 *x = warp_fft(b0, b1, a.logn2, a.s, tw + n1);
        const int dr = r < H ? n1 : (r >= n1 - H ? -n1 : 0);
        for (int c = lane - H; c < n2 + H; c += 32) {
            const float2 v = x[c & (n2 - 1)];
            row[c] = v;
            if (dr) row[static_cast<ptrdiff_t>(dr) * g.C + c] = v;
        }
        __syncwarp();
    }
    grid_arrive(ka.status);
    // gather: the tile's patch to shared memory, then kLanes lanes a point, a
    // row of taps an iteration (the tiled gather's sums, split over the lanes).
    // The first points' weights are there before the grid is.
    using S = SmallPatch<K>;
    constexpr int kLanes = 4, B = 32 / kLanes;
    float2 *patch = reinterpret_cast<float2 *>(mine);
    float *w1s = reinterpret_cast<float *>(mine + S::ELEMS * 8) + lane;
    const int n = ka.n_chunks >= 0 ? ka.n_chunks : ka.status[0];  // < 0: counted on the device only
    const int split = small_split(n), units = n * split;
    const int first_row = lane % kLanes;
    bool waiting = true;
    int u = gw, p = lane / kLanes;
    SmallUnit q = small_unit<B>(chunks, u, units, split, g);
    do {
        bool have = p < q.count;
        const int4 raw = __ldg(reinterpret_cast<const int4 *>(recs) + (have ? q.first + p : 0));
        const int lr = static_cast<int>(static_cast<unsigned>(raw.z) >> 16) - q.r0, lc = (raw.z & 0xFFFF) - q.c0;
        if (have && (static_cast<unsigned>(lr) >= static_cast<unsigned>(kRegTile) ||
                     static_cast<unsigned>(lc) >= static_cast<unsigned>(kRegTile))) {
            latch_error(ka.status, kErrBounds);
            have = false;
        }
        float w1[S::W], w2[S::W];
        weights_poly2<K>(__int_as_float(raw.x), __int_as_float(raw.y), w1, w2, ka.poly);
#pragma unroll
        for (int k = 0; k < S::W; ++k) w1s[k * S::WROW] = w1[k];
        if (waiting && !grid_wait(ka.status, 2, a.give_up)) {
            grid_done(ka.status, true);
            return;
        }
        waiting = false;
        if (p < B && q.count > 0) {  // a new tile
            const float2 *src = grid + static_cast<size_t>(q.r0 - K + H) * g.C + (q.c0 - S::KE + H);
            constexpr int HALF = S::COLS / 2;
            __syncwarp();
#pragma unroll 8
            for (int i = lane; i < S::PR * HALF; i += 32) {
                const int r = i / HALF, c = 2 * (i - r * HALF);
                *reinterpret_cast<float4 *>(patch + r * S::PITCH + c) = ld_rw4(src + static_cast<size_t>(r) * g.C + c);
            }
            __syncwarp();
        }
        float sx = 0.f, sy = 0.f, ex = 0.f, ey = 0.f;
        if (have) {
            const float2 *tap = patch + (lr + first_row) * S::PITCH + lc + (S::KE - K);
#pragma unroll 1
            for (int r = first_row; r < S::W; r += kLanes, tap += kLanes * S::PITCH) {
                float rx = 0.f, ry = 0.f;
#pragma unroll
                for (int k = 0; k < S::W; ++k) {
                    const float2 v = tap[k];
                    rx = fmaf(w2[k], v.x, rx);
                    ry = fmaf(w2[k], v.y, ry);
                }
                const float w = w1s[r * S::WROW];
                if (ka.compensated) {
                    float e;
                    two_sum(sx, __fmul_rn(w, rx), sx, e);
                    ex = __fadd_rn(ex, e);
                    two_sum(sy, __fmul_rn(w, ry), sy, e);
                    ey = __fadd_rn(ey, e);
                } else {
                    sx = fmaf(w, rx, sx);
                    sy = fmaf(w, ry, sy);
                }
            }
        }
#pragma unroll
        for (int o = 1; o < kLanes; o *= 2) {
            const float ox = __shfl_xor_sync(0xffffffffu, sx, o), oy = __shfl_xor_sync(0xffffffffu, sy, o);
            ex = __fadd_rn(ex, __shfl_xor_sync(0xffffffffu, ex, o));
            ey = __fadd_rn(ey, __shfl_xor_sync(0xffffffffu, ey, o));
            if (ka.compensated) {
                float e;
                two_sum(sx, ox, sx, e);
                ex = __fadd_rn(ex, e);
                two_sum(sy, oy, sy, e);
                ey = __fadd_rn(ey, e);
            } else {
                sx = __fadd_rn(sx, ox);
                sy = __fadd_rn(sy, oy);
            }
        }
        if (have && first_row == 0) out[ka.binned_io ? q.first + p : raw.w] = make_float2(sx + ex, sy + ey);
        p += B;
        if (p - lane / kLanes >= q.count) {
            u += kSmallWarps;
            p = lane / kLanes;
            q = small_unit<B>(chunks, u, units, split, g);
        }
    } while (u < units);
    grid_done(ka.status, false);
}

template <int K>
__global__ void __launch_bounds__(kSmallThreads)
    k_small_type1(const __grid_constant__ CUtensorMap tmap, const float2 *__restrict__ f, float2 *grid,
                  const Rec32 *__restrict__ recs, const int4 *__restrict__ chunks, float2 *__restrict__ F,
                  const SmallArgs a, const __grid_constant__ KArgs ka) {
    extern __shared__ unsigned char sm_raw[];
    unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(sm_raw) + 127) & ~uintptr_t(127));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, gw = wid * kSmallCtas + blockIdx.x;
    float2 *tw = reinterpret_cast<float2 *>(base);
    unsigned char *mine = base + kTwBytes + wid * small_warp_bytes<K>();
    float2 *b0 = reinterpret_cast<float2 *>(mine), *b1 = b0 + kSmallSide;
    const Geom &g = ka.g;
    const int n1 = g.n1, n2 = g.n2, H = g.H, N1 = a.N1, N2 = a.N2;
    float2 *const inner = grid + static_cast<size_t>(H) * g.C + H;  // cell (0, 0)
    for (int i = blockIdx.x * kSmallThreads + threadIdx.x; i < g.Ra * (g.C >> 1); i += kSmallCtas * kSmallThreads)
        reinterpret_cast<float4 *>(grid)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    grid_arrive(ka.status);
    load_twiddles(tw, a);
    // spread: one point after another into the tile's patch in shared memory,
    // a lane per column and component; the patch leaves as one TMA reduction
    using S = SmallPatch<K>;
    float *patch = reinterpret_cast<float *>(mine);
    float *w1s = reinterpret_cast<float *>(mine + S::ELEMS * 8), *w2s = w1s + S::W * S::WROW;
    const int n = ka.n_chunks >= 0 ? ka.n_chunks : ka.status[0];  // < 0: counted on the device only
    const int split = small_split(n), units = n * split;
    bool pending = false;  // a reduction of this warp's patch
    bool waiting = true;
    for (int u = gw; u < units || waiting; u += kSmallWarps) {
        const SmallUnit q = small_unit<16>(chunks, u, units, split, g);
        if (pending && lane == 0) bulk_wait_read_all();  // the last patch has been read
        __syncwarp();
        for (int i = lane; i < S::ELEMS / 2; i += 32) reinterpret_cast<float4 *>(patch)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p0 = 0; p0 < q.count; p0 += 32) {
            int4 raw = make_int4(0, 0, 0, 0);
            if (p0 + lane < q.count) raw = __ldg(reinterpret_cast<const int4 *>(recs) + q.first + p0 + lane);
            float2 v = make_float2(0.f, 0.f);
            if (p0 + lane < q.count) v = __ldg(f + (ka.binned_io ? q.first + p0 + lane : raw.w));
            int lr = static_cast<int>(static_cast<unsigned>(raw.z) >> 16) - q.r0, lc = (raw.z & 0xFFFF) - q.c0;
            if (p0 + lane >= q.count) lr = lc = 0;
            if (static_cast<unsigned>(lr) >= static_cast<unsigned>(kRegTile) ||
                static_cast<unsigned>(lc) >= static_cast<unsigned>(kRegTile)) {
                latch_error(ka.status, kErrBounds);
                lr = lc = 0;
                v = make_float2(0.f, 0.f);  // contributes nothing
            }
            float w1[S::W], w2[S::W];
            weights_poly2<K>(__int_as_float(raw.x), __int_as_float(raw.y), w1, w2, ka.poly);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < S::W; ++k) {
                w1s[k * S::WROW + lane] = w1[k];
                w2s[k * S::WROW + lane] = w2[k];
            }
            __syncwarp();
            const int at = 2 * (lr * S::PITCH + lc + (S::KE - K));
            const int nb = min(32, q.count - p0);
#pragma unroll 1
            for (int p = 0; p < nb; ++p) {
                const float vx = __shfl_sync(0xffffffffu, v.x, p), vy = __shfl_sync(0xffffffffu, v.y, p);
                float *cell = patch + __shfl_sync(0xffffffffu, at, p) + lane;
                // columns 0 .. 15 of the window, then (W > 16) the last one
#pragma unroll
                for (int c0 = 0; c0 < S::W; c0 += 16) {
                    const int c = c0 + (lane >> 1);
                    if (c < S::W) {
                        const float vw = (lane & 1 ? vy : vx) * w2s[c * S::WROW + p];
                        float sum[S::W];  // all loads before the first store
#pragma unroll
                        for (int r = 0; r < S::W; ++r) sum[r] = cell[2 * (r * S::PITCH + c0)];
#pragma unroll
                        for (int r = 0; r < S::W; ++r) sum[r] = fmaf(vw, w1s[r * S::WROW + p], sum[r]);
#pragma unroll
                        for (int r = 0; r < S::W; ++r) cell[2 * (r * S::PITCH + c0)] = sum[r];
                    }
                }
                __syncwarp();
            }
        }
        fence_proxy_async_smem();  // the patch, before the TMA engine reads it
        // the zeros of the grid are there (and so is the loop's code) by now
        if (waiting && !grid_wait(ka.status, 1, a.give_up)) {
            grid_done(ka.status, true);
            return;
        }
        waiting = false;
        __syncwarp();
        pending = true;
        if (lane == 0 && q.count > 0) {
            asm volatile("fence.proxy.async;" ::: "memory");  // the zeros, before the TMA engine adds to them
            tma_reduce_add_2d(&tmap, patch, 2 * (H + q.c0 - S::KE), H + q.r0 - K);
            bulk_commit();
        }
    }
    if (lane == 0) bulk_wait_all();
    __syncwarp();
    if (!grid_barrier(ka.status, 2, a.give_up)) {
        grid_done(ka.status, true);
        return;
    }
    for (int r = gw; r < n1; r += kSmallWarps) {  // rows with their halo images folded in
        float2 *row = inner + static_cast<size_t>(r) * g.C;
        const bool edge = r < H || r >= n1 - H;
        // all images' loads together: a cell without one reads itself
        const ptrdiff_t dr = edge ? static_cast<ptrdiff_t>(r < H ? n1 : -n1) * g.C : 0;
#pragma unroll 4
        for (int c = lane; c < n2; c += 32) {
            const bool side = c < H || c >= n2 - H;
            const int dc = side ? (c < H ? n2 : -n2) : 0;
            const float2 *at = row + c;
            const float2 v0 = ld_rw(at), v1 = ld_rw(at + dc), v2 = ld_rw(at + dr), v3 = ld_rw(at + dr + dc);
            float2 v = v0;
            if (side) v = add(v, v1);
            if (edge) v = add(v, v2);
            if (side && edge) v = add(v, v3);
            b0[c] = v;
        }
        __syncwarp();
        const float2 *x = warp_fft(b0, b1, a.logn2, a.s, tw + n1);
        for (int c = lane; c < n2; c += 32) {
            const int k2 = c < n2 / 2 ? c : c - n2;
            if (k2 >= -N2 / 2 && k2 < N2 / 2) row[c] = x[c];
        }
        __syncwarp();
    }
    if (!grid_barrier(ka.status, 3, a.give_up)) {
        grid_done(ka.status, true);
        return;
    }
    for (int bc = gw; bc < N2; bc += kSmallWarps) {  // band columns, cropped
        const int j = bc < N2 / 2 ? bc + N2 / 2 : bc - N2 / 2, c = bc < N2 / 2 ? bc : n2 - N2 + bc;
        const float s2 = __ldg(a.d2 + j);
#pragma unroll 4
        for (int r = lane; r < n1; r += 32) b0[r] = ld_rw(inner + static_cast<size_t>(r) * g.C + c);
        __syncwarp();
        const float2 *x = warp_fft(b0, b1, a.logn1, a.s, tw);
#pragma unroll 2
        for (int i = lane; i < N1; i += 32) {
            const float2 v = x[(i - N1 / 2) & (n1 - 1)];
            const float sc = __ldg(a.d1 + i) * s2;
            F[static_cast<size_t>(i) * N2 + j] = make_float2(v.x * sc, v.y * sc);
        }
        __syncwarp();
    }
    grid_done(ka.status, false);
}

SmallArgs small_args(const nfft2d_plan_s *p, int sign) {
    SmallArgs a{};
    a.N1 = p->N1;
    a.N2 = p->N2;
    while ((1 << a.logn1) < p->g.n1) ++a.logn1;
    while ((1 << a.logn2) < p->g.n2) ++a.logn2;
    a.s = sign < 0 ? -1.f : 1.f;
    a.give_up = p->give_up;
    a.d1 = static_cast<const float *>(p->deap1);
    a.d2 = static_cast<const float *>(p->deap2);
    a.tw1 = p->tw1;
    a.tw2 = p->tw2;
    return a;
}

template <typename Kernel, typename... Args>
cudaError_t launch_grid(Kernel kernel, int smem, const nfft2d_plan_s *p, Args... args) {
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSmallCtas);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cfg.stream = p->stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int K>
cudaError_t type2_K(const nfft2d_plan_s *p, int sign, const void *F, void *f) {
    return launch_grid(k_small_type2<K>, small_smem<K>(), p, static_cast<const float2 *>(F),
                       static_cast<float2 *>(p->grid), static_cast<const Rec32 *>(p->recs),
                       static_cast<const int4 *>(p->chunks), static_cast<float2 *>(f), small_args(p, sign),
                       make_kargs(p));
}

template <int K>
cudaError_t type1_K(const nfft2d_plan_s *p, int sign, const void *f, void *F) {
    return launch_grid(k_small_type1<K>, small_smem<K>(), p, p->tmap, static_cast<const float2 *>(f),
                       static_cast<float2 *>(p->grid), static_cast<const Rec32 *>(p->recs),
                       static_cast<const int4 *>(p->chunks), static_cast<float2 *>(F), small_args(p, sign),
                       make_kargs(p));
}

template <typename Fn>
cudaError_t by_width(int K, Fn fn) {
    switch (K) {
        case 2: return fn(std::integral_constant<int, 2>{});
        case 3: return fn(std::integral_constant<int, 3>{});
        case 4: return fn(std::integral_constant<int, 4>{});
        case 5: return fn(std::integral_constant<int, 5>{});
        case 6: return fn(std::integral_constant<int, 6>{});
        case 7: return fn(std::integral_constant<int, 7>{});
        case 8: return fn(std::integral_constant<int, 8>{});
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

bool small_available(const nfft2d_plan_s *p) {
    // power-of-two sides (fused_ok); a CTA an SM, all of them resident
    const Geom &g = p->g;
    return p->precision == NFFT2D_F32 && !p->grid_external && p->fused_ok && p->tmap_ok && g.T == kRegTile &&
           g.n1 <= kSmallSide && g.n2 <= kSmallSide && 1LL * g.n1 * g.n2 <= kSmallCells && p->num_sms >= kSmallCtas;
}

cudaError_t launch_small_type2(const nfft2d_plan_s *p, int sign, const void *F, void *f) {
    return by_width(p->K, [&](auto k) { return type2_K<decltype(k)::value>(p, sign, F, f); });
}

cudaError_t launch_small_type1(const nfft2d_plan_s *p, int sign, const void *f, void *F) {
    return by_width(p->K, [&](auto k) { return type1_K<decltype(k)::value>(p, sign, f, F); });
}

}  // namespace nfft2d
