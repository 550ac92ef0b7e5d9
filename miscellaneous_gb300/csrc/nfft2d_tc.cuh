// nfft2d_tc.cuh -- the tile contraction of the FP32 gather on the tensor
// cores (tcgen05), shared by the single-transform and the batched kernels.
//
// All points of one tile draw on one patch of at most 32 columns x 32 rows, so
//     Y[p][r] = sum_c w2_p[c] G[r][c],   f_p = sum_r w1_p[r] Y[p][r]
// has a dense inner product: 128 points x 32 columns x (real and imaginary
// rows) is one accumulator of 128 lanes in tensor memory.  One thread owns one
// point from its record to its result: it evaluates the weights, leaves the
// column weights in shared memory as a row of the A operand, and finishes its
// own accumulator lane with the row weights.
//
// Precision: every operand is a sum of three bf16 parts, and the six largest of
// the nine products are taken, the leading one in an accumulator of its own.
// bf16 keeps FP32's exponent range: no scaling.  What is left out:
//   - values: nothing down to 2^-27 of the value.
//   - weights: 2^-27 of the window's peak, or 2^-18 of a weight below 2^-9 of it,
//     whose leading part is zero (see split_weight).
//   - the three smallest products: 2^-26 of peak times value, or 2^-17 of weight
//     times value for those weights.
//   - the unit's sums, truncated at about 2^-24 of the largest term: nothing of
//     the leading products while the cells under a window differ by less than 2^6
//     or so, up to that unit a product where they differ by more.
// Relative error against 64 bits, the FP32 gather -> here (512^2 coefficients,
// 2^20 points, w 6 | 7 | 8): random coefficients 2.41 -> 2.33e-7 | 2.71 -> 2.59 |
// 3.31 -> 3.15; a regridder's raster 4.29 -> 4.30 (w 6); 100 scatterers under a
// taper, whose peaks stand 2^30 above the cells around them, 1.58 -> 1.63 | 1.67 ->
// 1.74 | 1.72 -> 1.77; at points where only the tails of their windows meet such
// a peak the two agree to 2 digits, the FP32 window's own fit being larger.
#pragma once

#include <cuda_runtime.h>

#include "nfft2d_device.cuh"
#include "nfft2d_internal.h"

namespace nfft2d {

// ---------------------------------------------------------------------------
// tcgen05 primitives
// ---------------------------------------------------------------------------
// Tensor memory of one CTA: `cols` columns (a power of two, at least 32), the
// address left in shared memory.  One whole warp calls each.  An allocation
// waits until the SM's other CTAs leave enough columns; they hold theirs only
// while they run.
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Arrive on an mbarrier once the thread's MMAs so far have completed.
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// D (tensor memory) = A B or += A B; bf16 operands in shared memory, FP32 accumulation.
__device__ __forceinline__ void tc_mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(static_cast<uint32_t>(accumulate))
        : "memory");
}
// 8 columns of the calling warp's 32 lanes, one lane a thread.
__device__ __forceinline__ void tmem_ld8(float (&v)[8], uint32_t addr) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Values loaded before tmem_wait_ld are read only after it.
__device__ __forceinline__ void tmem_ready(float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) asm volatile("" : "+f"(v[i]));
}

// Operands in shared memory, K-major without swizzle: core matrices of 8 rows
// x 16 bytes, contiguous; neighbours along K LBO bytes apart, along M or N
// 4 LBO (32 bf16 columns are four core matrices a row group).  B's LBO is 160:
// a warp stores consecutive columns of one or two rows, and with 128 the
// columns' core matrices fall in the same banks.
constexpr uint32_t kLboA = 128, kLboB = 160;
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t addr, uint32_t lbo) {
    return static_cast<uint64_t>((addr & 0x3ffff) >> 4) | static_cast<uint64_t>(lbo >> 4) << 16 |
           static_cast<uint64_t>(lbo >> 2) << 32 | static_cast<uint64_t>(1) << 46;
}
// FP32 accumulators, bf16 A and B, both K-major, M x N.
__host__ __device__ constexpr uint32_t tc_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n / 8) << 17) |
           (static_cast<uint32_t>(m / 16) << 24);
}

// ---------------------------------------------------------------------------
// three-way bf16 splits
// ---------------------------------------------------------------------------
// Two FP32 values as three packed bf16 pairs: x = h + m + l.
struct Bf3 {
    uint32_t h, m, l;
};

__device__ __forceinline__ uint32_t pack_bf16(float x0, float x1) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(x1), "f"(x0));
    return d;
}

__device__ __forceinline__ float2 unpack_bf16(uint32_t p) {
    return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
}
// a - b, one rounding an element
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

// h and its rest given: m and l by rounding to nearest.
__device__ __forceinline__ void split_rest(Bf3 &s, float2 x) {
    s.m = pack_bf16(x.x, x.y);
    x = sub2(x, unpack_bf16(s.m));
    s.l = pack_bf16(x.x, x.y);
}

// Grid values: all three parts by rounding to nearest, an exact sum.
__device__ __forceinline__ Bf3 split_value(float x0, float x1) {
    const float2 x = make_float2(x0, x1);
    Bf3 s;
    s.h = pack_bf16(x0, x1);
    split_rest(s, sub2(x, unpack_bf16(s.h)));
    return s;
}

// Window weights, at most 1 in magnitude: h is a multiple of 2^-8 (rounded by
// adding and taking back 1.5 * 2^15), so that its products with 8-bit parts of
// values of one size, summed over a window, fit the accumulator's 24 bits: the
// tensor cores truncate, and with h rounded at each weight's own size a leading
// sum came out 0.9e-7 short.
__device__ __forceinline__ Bf3 split_weight(float x0, float x1) {
    constexpr float kMagic = 49152.f;
    const float2 x = make_float2(x0, x1);
    const float2 h = __fadd2_rn(__fadd2_rn(x, make_float2(kMagic, kMagic)), make_float2(-kMagic, -kMagic));
    Bf3 s;
    s.h = __byte_perm(__float_as_uint(h.x), __float_as_uint(h.y), 0x7632);
    split_rest(s, sub2(x, h));
    return s;
}

// ---------------------------------------------------------------------------
// the gather
// ---------------------------------------------------------------------------
constexpr int kTcPoints = 128;  // points of a batch: lanes of an accumulator, threads of a CTA
constexpr int kTcCtas = 4;      // CTAs an SM: 128 of its 512 columns of tensor memory each

// Work items of a run: neighbours share a tile and its patch, but each CTA
// should get several runs.
inline int tc_run_items(long long items, long long ctas) {
    const long long r = items / (8 * ctas);
    return static_cast<int>(r < 1 ? 1 : (r > 16 ? 16 : r));
}

template <int K>
struct TcGeo {
    static constexpr int W = 2 * K + 1;
    static constexpr int KE = K + (K & 1);               // column halo: even, rows stay on 16-byte boundaries
    static constexpr int PR = 16 + 2 * K;                // patch rows
    static constexpr int PC = 16 + 2 * KE;               // patch columns, at most 32
    static constexpr int NR = (PR + 7) / 8 * 8;          // rows of the accumulator, real and imaginary each
    static constexpr int N = 2 * NR;
    static constexpr uint32_t COLS = 128;                // tensor memory: leading and remaining products
    static constexpr int A_PLANE = kTcPoints * 64;       // bytes: 128 rows x 32 bf16
    static constexpr int B_PLANE = N / 2 * static_cast<int>(kLboB);
    static constexpr int W_BYTES = NR * kTcPoints * 4;   // row weights by patch row, one column a point
    static constexpr int SMEM = 3 * A_PLANE + 3 * B_PLANE + W_BYTES + 128;
    static_assert(PC <= 32 && NR <= 32 && 2 * N <= 128, "the patch fits the operands");
};

// The batches of a CTA: runs of `group` consecutive work items {tile, first
// point, points}, dealt round robin; an item is cut every kTcPoints points.
struct TcWalk {
    const int4 *chunks;
    int n, group, step;  // items; items a run; items from one run of this CTA to its next
    int tiles2, T;
    int i, end;          // this item, end of its run
    int first, count;    // this batch's points
    int left;            // points of the item after this batch
    int tile, r0, c0;    // its tile and the tile's origin
    int4 next;           // the next item of the run

    __device__ __forceinline__ TcWalk(const int4 *chunks_, int n_, int group_, const Geom &g)
        : chunks(chunks_), n(n_), group(group_), step(static_cast<int>(gridDim.x) * group_), tiles2(g.tiles2), T(g.T),
          tile(-1) {}

    __device__ __forceinline__ void item(const int4 &ch) {
        if (ch.x != tile) {
            tile = ch.x;
            const int tr = tile / tiles2;
            r0 = tr * T;
            c0 = (tile - tr * tiles2) * T;
        }
        first = ch.y;
        count = min(kTcPoints, ch.z);
        left = ch.z - count;
        if (i + 1 < end) next = __ldg(&chunks[i + 1]);
    }
    __device__ __forceinline__ bool open(int run) {
        i = run;
        end = min(run + group, n);
        if (i >= n) return false;
        item(__ldg(&chunks[i]));
        return true;
    }
    __device__ __forceinline__ bool advance() {
        if (left > 0) {
            first += count;
            count = min(kTcPoints, left);
            left -= count;
            return true;
        }
        if (++i == end) return open(end - group + step);  // a run cut short is the last
        item(next);
        return true;
    }
};

// One tile's patch on its way from the padded grid to the B operand: two
// columns of one row a slot, loaded ahead of their use.  Cells outside the
// logical padded grid are no one's: zero.
template <int K>
struct TcPatch {
    static constexpr int CELLS = TcGeo<K>::PR * TcGeo<K>::PC / 2;
    static constexpr int SLOTS = (CELLS + kTcPoints - 1) / kTcPoints;
    float4 v[SLOTS];

    __device__ __forceinline__ void load(const float2 *__restrict__ grid, const Geom &g, int r0, int c0) {
        using S = TcGeo<K>;
#pragma unroll
        for (int k = 0; k < SLOTS; ++k) {
            const int i = k * kTcPoints + threadIdx.x;
            const int r = i / (S::PC / 2), c = 2 * (i - r * (S::PC / 2));
            const int row = r0 - K + g.H + r, col = c0 - S::KE + g.H + c;
            v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < CELLS && row < g.R && col < g.Cl)
                v[k] = __ldg(reinterpret_cast<const float4 *>(grid + static_cast<size_t>(row) * g.C + col));
        }
    }
    __device__ __forceinline__ void store(unsigned char *b) const {
        using S = TcGeo<K>;
#pragma unroll
        for (int k = 0; k < SLOTS; ++k) {
            const int i = k * kTcPoints + threadIdx.x;
            const int r = i / (S::PC / 2), c = 2 * (i - r * (S::PC / 2));
            if (i >= CELLS) break;
            const Bf3 re = split_value(v[k].x, v[k].z), im = split_value(v[k].y, v[k].w);
            unsigned char *p = b + (4 * (r >> 3) + (c >> 3)) * static_cast<int>(kLboB) + (r & 7) * 16 + (c & 7) * 2;
            constexpr int kIm = S::NR / 2 * static_cast<int>(kLboB);
            *reinterpret_cast<uint32_t *>(p) = re.h;
            *reinterpret_cast<uint32_t *>(p + S::B_PLANE) = re.m;
            *reinterpret_cast<uint32_t *>(p + 2 * S::B_PLANE) = re.l;
            *reinterpret_cast<uint32_t *>(p + kIm) = im.h;
            *reinterpret_cast<uint32_t *>(p + kIm + S::B_PLANE) = im.m;
            *reinterpret_cast<uint32_t *>(p + kIm + 2 * S::B_PLANE) = im.l;
        }
    }
};

// The MMAs of a batch and their commit: one thread.  The leading part of A
// meets the leading and middle parts of B in one MMA of twice the rows (their
// planes adjoin, and so do the two accumulators), which reads A once: the MMAs
// are bound by their operand reads from shared memory, not by their products.
template <int K>
__device__ __forceinline__ void tc_gather_mma(uint32_t tmem, const unsigned char *a, const unsigned char *b,
                                              uint64_t *bar) {
    using S = TcGeo<K>;
    const uint64_t da = tc_smem_desc(smem_u32(a), kLboA), db = tc_smem_desc(smem_u32(b), kLboB);
    constexpr int pa[5] = {0, 2, 0, 1, 1}, pb[5] = {0, 0, 2, 1, 0};
#pragma unroll
    for (int m = 0; m < 5; ++m)
#pragma unroll
        for (int k = 0; k < 2; ++k)  // descriptors count 16 bytes
            tc_mma_bf16(tmem + (m ? S::N : 0), da + (pa[m] * S::A_PLANE + k * 2 * kLboA) / 16,
                        db + (pb[m] * S::B_PLANE + k * 2 * kLboB) / 16, tc_idesc(kTcPoints, m ? S::N : 2 * S::N),
                        k > 0 || m > 0);
    tc_commit(bar);
}

// This thread's row of A: the point's column weights as words of two columns.
template <int K>
struct TcRow {
    Bf3 s[K + 1];
    int word;  // first word

    // the 2K+1 weights from patch column col
    __device__ __forceinline__ void make(const float (&w)[2 * K + 1], int col) {
        word = col >> 1;
        const bool odd = col & 1;
#pragma unroll
        for (int j = 0; j <= K; ++j)
            s[j] = split_weight(odd ? (j ? w[2 * j - 1] : 0.f) : w[2 * j], odd ? w[2 * j] : (j < K ? w[2 * j + 1] : 0.f));
    }
    __device__ __forceinline__ static void put(unsigned char *p, int x, uint32_t h, uint32_t m, uint32_t l) {
        unsigned char *d = p + (x >> 2) * kLboA + (x & 3) * 4;
        *reinterpret_cast<uint32_t *>(d) = h;
        *reinterpret_cast<uint32_t *>(d + TcGeo<K>::A_PLANE) = m;
        *reinterpret_cast<uint32_t *>(d + 2 * TcGeo<K>::A_PLANE) = l;
    }
    // Of the row's last weights (from word old), those that the new ones leave
    // behind are cleared.  Rows 8 apart fall in the same banks, so every other
    // group of 8 stores its words in pairs the other way round.
    __device__ __forceinline__ void store(unsigned char *p, int old) const {
        if (__any_sync(0xffffffffu, word != old)) {
#pragma unroll
            for (int j = 0; j <= K; ++j) {
                const int x = old + j;
                if (x < word || x > word + K) put(p, x, 0u, 0u, 0u);
            }
        }
        const bool swap = threadIdx.x & 8;
#pragma unroll
        for (int j = 0; j <= K; j += 2) {
            if (j == K) {
                put(p, word + j, s[j].h, s[j].m, s[j].l);
            } else {
                const Bf3 &u = s[j], &v = s[j + 1];
                put(p, word + j + (swap ? 1 : 0), swap ? v.h : u.h, swap ? v.m : u.m, swap ? v.l : u.l);
                put(p, word + j + (swap ? 0 : 1), swap ? u.h : v.h, swap ? u.m : v.m, swap ? u.l : v.l);
            }
        }
    }
};

// sum_r w1[r] Y[r] of the thread's accumulator lane, rows of the warp's
// windows (lr within [lo, hi]) 8 at a time; wcol: the point's row weights by
// patch row.  Inside 8 rows the small products go first; the sum over the
// steps is compensated (Kahan: the lost part goes into the next).
template <int K, bool COMP>
__device__ __forceinline__ float2 tc_gather_finish(uint32_t tmem, const float *wcol, int lo, int hi) {
    using S = TcGeo<K>;
    const int steps = (hi - lo + S::W + 7) / 8;
    const int start = min(lo, S::NR - 8 * steps);
    float2 s[2], c[2];  // real, imaginary: sums over even and odd rows
    s[0] = s[1] = c[0] = c[1] = make_float2(0.f, 0.f);
    const float *wr = wcol + start * kTcPoints;
    uint32_t at = tmem + start;
    for (int q = 0; q < steps; ++q, at += 8, wr += 8 * kTcPoints) {
        float yh[2][8], yl[2][8], w[8];
        tmem_ld8(yl[0], at + S::N);
        tmem_ld8(yh[0], at);
        tmem_ld8(yl[1], at + S::N + S::NR);
        tmem_ld8(yh[1], at + S::NR);
#pragma unroll
        for (int k = 0; k < 8; ++k) w[k] = wr[k * kTcPoints];
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            tmem_ready(yl[e]);
            tmem_ready(yh[e]);
            float2 x = c[e];
#pragma unroll
            for (int k = 0; k < 8; k += 2)
                x = __ffma2_rn(make_float2(yl[e][k], yl[e][k + 1]), make_float2(w[k], w[k + 1]), x);
#pragma unroll
            for (int k = 0; k < 8; k += 2)
                x = __ffma2_rn(make_float2(yh[e][k], yh[e][k + 1]), make_float2(w[k], w[k + 1]), x);
            const float2 n = __fadd2_rn(s[e], x);
            if constexpr (COMP) c[e] = sub2(x, sub2(n, s[e]));
            s[e] = n;
        }
    }
    return make_float2((s[0].x + s[0].y) + (c[0].x + c[0].y), (s[1].x + s[1].y) + (c[1].x + c[1].y));
}

// The MMAs up to the last commit are done; false if the wait ran out (latched;
// the CTA leaves at its next barrier, after a second wait so that no MMA is in
// flight then).
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t phase, int *status) {
    if (mbar_wait_bounded(bar, phase)) return true;
    (void)mbar_wait_bounded(bar, phase);
    latch_error(status, kErrTimeout);
    return false;
}

// One gathering CTA: its operands, its tensor memory, and what it must
// remember between batches.
template <int K>
struct TcGather {
    unsigned char *A, *B, *arow;  // operands; this thread's row of A
    float *wcol;                  // this thread's column of the row weights
    uint64_t *bar;
    uint32_t tmem, phase;
    int old_word, old_row;        // places of the weights last stored
    bool failed;

    __device__ __forceinline__ void begin(unsigned char *smem, uint32_t *tmem_slot, uint64_t *barrier) {
        using S = TcGeo<K>;
        const int tid = threadIdx.x;
        A = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem) + 127) & ~uintptr_t(127));
        B = A + 3 * S::A_PLANE;
        wcol = reinterpret_cast<float *>(B + 3 * S::B_PLANE) + tid;
        arow = A + (tid >> 3) * (4 * kLboA) + (tid & 7) * 16;
        bar = barrier;
        phase = 0;
        old_word = old_row = 0;
        failed = false;
        // what no patch and no window reaches stays zero
        for (int i = tid; i < (S::SMEM - 128) / 16; i += kTcPoints)
            reinterpret_cast<float4 *>(A)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid < 32) tmem_alloc(tmem_slot, S::COLS);
        if (tid == 0) {
            mbar_init(bar, 1);
            fence_proxy_async_smem();
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        tmem = *tmem_slot;
    }

    __device__ __forceinline__ void end() const {
        tc_fence_before();
        __syncthreads();
        if (threadIdx.x < 32) tmem_free(tmem, TcGeo<K>::COLS);
    }

    // Gather every batch of `walk`, from the run of items at i0 on, from one
    // padded grid.  n_recs records exist.  A record outside its tile latches
    // kErrBounds and has no result.  False if a wait has run out.
    template <bool COMP>
    __device__ __forceinline__ bool run(TcWalk walk, int i0, const float2 *__restrict__ grid, const Geom &g,
                                        const Rec32 *__restrict__ recs, int n_recs, float2 *__restrict__ out,
                                        int binned_io, const WinPoly &wp, int *status) {
        using S = TcGeo<K>;
        const int tid = threadIdx.x;
        bool more = walk.open(i0);
        TcPatch<K> patch;
        if (more) {
            patch.load(grid, g, walk.r0, walk.c0);
            patch.store(B);
        }
        // the records of the batch after the one at hand are loaded ahead (they
        // follow on, except after the last item of a run)
        int4 ahead = make_int4(0, 0, 0, 0);
        int ahead_first = -1;
        while (more) {
            int4 raw = ahead;
            if (ahead_first != walk.first && walk.first + tid < n_recs)
                raw = __ldg(reinterpret_cast<const int4 *>(recs) + walk.first + tid);
            int lr = static_cast<int>(static_cast<unsigned>(raw.z) >> 16) - walk.r0, lc = (raw.z & 0xFFFF) - walk.c0;
            bool ok = tid < walk.count;
            if (ok && (static_cast<unsigned>(lr) >= static_cast<unsigned>(g.T) ||
                       static_cast<unsigned>(lc) >= static_cast<unsigned>(g.T))) {
                latch_error(status, kErrBounds);
                ok = false;
            }
            // rows of the warp's windows
            const int lo = __reduce_min_sync(0xffffffffu, ok ? lr : 31), hi = __reduce_max_sync(0xffffffffu, ok ? lr : -1);
            const size_t dst = binned_io ? static_cast<size_t>(walk.first + tid) : static_cast<size_t>(raw.w);
            if (hi >= 0) {
                if (!ok) lr = lc = 0;  // no result: any finite weights
                float w1[S::W], w2[S::W];
                weights_poly2<K>(__int_as_float(raw.x), __int_as_float(raw.y), w1, w2, wp);
#pragma unroll
                for (int a = 0; a < S::W; ++a) wcol[(old_row + a) * kTcPoints] = 0.f;
#pragma unroll
                for (int a = 0; a < S::W; ++a) wcol[(lr + a) * kTcPoints] = w1[a];
                old_row = lr;
                TcRow<K> row;
                row.make(w2, lc + S::KE - K);
                row.store(arow, old_word);
                old_word = row.word;
            }
            ahead_first = walk.first + walk.count;
            if (ahead_first + tid < n_recs) ahead = __ldg(reinterpret_cast<const int4 *>(recs) + ahead_first + tid);
            fence_proxy_async_smem();  // this thread's operand words, before the MMAs read them
            tc_fence_before();         // and its reads of the accumulator, before they overwrite it
            if (__syncthreads_or(failed)) return false;
            if (tid == 0) {
                tc_fence_after();
                tc_gather_mma<K>(tmem, A, B, bar);
            }
            const int tile = walk.tile;
            more = walk.advance();
            const bool tile_change = more && walk.tile != tile;
            if (tile_change) patch.load(grid, g, walk.r0, walk.c0);  // arrives during the MMAs
            failed = !tc_wait(bar, phase, status);
            phase ^= 1;
            tc_fence_after();
            if (hi >= 0 && !failed) {
                const float2 f = tc_gather_finish<K, COMP>(tmem + (static_cast<uint32_t>(tid & ~31) << 16), wcol, lo, hi);
                if (ok) out[dst] = f;
            }
            if (tile_change) patch.store(B);  // the MMAs are done with the last one
        }
        return true;
    }
};

// When the tensor-core gather takes over from the direct one (FP32, tiles of
// at most 16 x 16).  It costs the same at every width (its contraction is 32
// columns wide), the direct one grows with the taps.  Measured on GB300, us,
// direct and tensor cores, 2^22 / 2^20 / 400 k uniform points on 1024^2
// coefficients (256 / 64 / 24 points a tile): w 8: 356 and 232 / 143 and 96 /
// 81 and 83; w 7: 436 and 230 / 139 and 94 / 67 and 81; w 6: 270 and 214 / 114
// and 90 / 59 and 79; w 5: 202 and 201 at 2^22.  Clustered sets fill fewer of
// its batches: w 6, 2^20 / 2^21 / 3 2^20 points (64 / 128 / 192 a tile), 87 and
// 102 / 136 and 141 / 190 and 177; w 8, 64 a tile, 115 and 111.  So from 48
// points a tile at w 7 and 8, and for a regridder's raster (whose tiles have no
// strips), from 128 at w 6.  Small sets give its persistent CTAs too few
// batches: w 6, 2^18 points on 512^2, 32 and 35.
inline bool tc_gather_pays(int K, const Geom &g, long long M) {
    const long long per_tile = K > 6 || g.SW == g.T ? 48 : 128;
    return K >= 6 && g.T <= 16 && M >= (1LL << 19) && M >= per_tile * g.tiles1 * g.tiles2;
}

}  // namespace nfft2d
