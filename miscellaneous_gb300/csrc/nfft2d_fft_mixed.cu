// nfft2d_fft_mixed.cu -- the fused FFT passes (nfft2d_fft.cu) for sides that
// are products of 2, 3, 5, 7, 11 and 13, with at most one larger prime: FP32
// plans whose oversampled grid is not a power of two a side, which otherwise run
// pad, a 2D library plan (two kernels), halo fill -- fold, two, crop the other
// way.
//
// Same two passes a direction: P band columns a CTA with the pad or the crop,
// a row a CTA with the halo's fill or fold.  One Stockham stage per factor (16
// and 9 are taken whole); the first stage reads and the last writes global
// memory, those between go through two buffers of shared memory.  A thread
// takes butterflies one after another, so any side fits any block.
//
// Bound by latency on grids below 10^6 cells (250 x 378 coefficients: 6.4 us a
// pass, for 48 us of the library's four kernels and 10 us of pad, fill, fold
// and crop before), above by shared memory, 2 (stages - 1) accesses an element.
// With the loads and stores as passes of their own through shared memory it
// was 2 (stages + 1): 1000 x 1000 coefficients forward 115 -> 98 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "nfft2d_device.cuh"
#include "nfft2d_internal.h"

namespace nfft2d {
namespace {

constexpr int kMaxStages = 10;  // 4096 >= 3^7
constexpr int kMixedMaxSide = 4096, kMixedMaxPrime = 67;

struct MixedFft {
    int n, stages;
    int radix[kMaxStages], done[kMaxStages];  // factor; product of the factors before it
    unsigned inv[kMaxStages];                 // ceil(2^32 / done): i / done for i < 2^16
    unsigned inv_nb;                          // the same for n / radix[0]
};

struct MixedArgs {
    MixedFft f;  // along the pass's direction
    int N1, N2, n1, n2, H, C;
    int logP;
    float s;  // exponent sign
};

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 mul_si(float2 a, float s) { return make_float2(-s * a.y, s * a.x); }  // s i a
__host__ __device__ constexpr int padded(int i) { return i + (i >> 4); }

// cos and sin of 2 pi k / R, k = 1 .. R / 2 (k known at compile time)
template <int R>
__device__ __forceinline__ float2 root(int k) {
    if constexpr (R == 3) {
        constexpr float c[] = {-0.49999999999999978f};
        constexpr float s[] = {0.86602540378443871f};
        return make_float2(c[k - 1], s[k - 1]);
    } else if constexpr (R == 5) {
        constexpr float c[] = {0.30901699437494745f, -0.80901699437494734f};
        constexpr float s[] = {0.95105651629515353f, 0.58778525229247325f};
        return make_float2(c[k - 1], s[k - 1]);
    } else if constexpr (R == 7) {
        constexpr float c[] = {0.62348980185873359f, -0.22252093395631434f, -0.90096886790241903f};
        constexpr float s[] = {0.7818314824680298f, 0.97492791218182362f, 0.43388373911755823f};
        return make_float2(c[k - 1], s[k - 1]);
    } else if constexpr (R == 11) {
        constexpr float c[] = {0.84125353283118121f, 0.41541501300188644f, -0.142314838273285f, -0.65486073394528499f,
                               -0.95949297361449737f};
        constexpr float s[] = {0.54064081745559756f, 0.90963199535451833f, 0.9898214418809328f, 0.75574957435425827f,
                               0.28173255684142967f};
        return make_float2(c[k - 1], s[k - 1]);
    } else {
        constexpr float c[] = {0.88545602565320991f, 0.56806474673115592f, 0.12053668025532301f, -0.35460488704253545f,
                               -0.74851074817110119f, -0.97094181742605201f};
        constexpr float s[] = {0.46472317204376851f, 0.82298386589365635f, 0.99270887409805397f, 0.93501624268541483f,
                               0.66312265824079519f, 0.23931566428755768f};
        return make_float2(c[k - 1], s[k - 1]);
    }
}

// exp(s 2 pi i k / N) for N = 8, 9, 16 (k known at compile time, at most 9)
template <int N>
__device__ __forceinline__ float2 unit(int k, float s) {
    constexpr float c[3][10] = {
        {1.f, 0.70710678118654757f, 6.0000000000000001e-17f, -0.70710678118654746f,
         -1.f, -0.70710678118654768f, -1.7999999999999999e-16f,
         0.70710678118654735f, 1.f, 0.70710678118654768f},
        {1.f, 0.76604444311897801f, 0.17364817766693041f, -0.49999999999999978f,
         -0.93969262078590832f, -0.93969262078590843f, -0.50000000000000044f,
         0.17364817766692997f, 0.76604444311897779f, 1.f},
        {1.f, 0.92387953251128674f, 0.70710678118654757f, 0.38268343236508984f,
         6.0000000000000001e-17f, -0.38268343236508973f, -0.70710678118654746f,
         -0.92387953251128674f, -1.f, -0.92387953251128685f}};
    constexpr float d[3][10] = {
        {0.f, 0.70710678118654746f, 1.f, 0.70710678118654757f,
         1.2e-16f, -0.70710678118654746f, -1.f,
         -0.70710678118654768f, -2.4e-16f, 0.70710678118654735f},
        {0.f, 0.64278760968653925f, 0.98480775301220802f, 0.86602540378443871f,
         0.34202014332566888f, -0.34202014332566866f, -0.86602540378443837f,
         -0.98480775301220813f, -0.64278760968653958f, -2.4e-16f},
        {0.f, 0.38268343236508978f, 0.70710678118654746f, 0.92387953251128674f,
         1.f, 0.92387953251128674f, 0.70710678118654757f,
         0.38268343236508989f, 1.2e-16f, -0.38268343236508967f}};
    constexpr int i = N == 8 ? 0 : (N == 9 ? 1 : 2);
    return make_float2(c[i][k], s * d[i][k]);
}

template <int R>
__device__ __forceinline__ void dft(float2 (&x)[R], float s);

// A B points as A transforms of B points, turned, then B of A points.
template <int A, int B>
__device__ __forceinline__ void dft_product(float2 (&x)[A * B], float s) {
    float2 y[A][B];
#pragma unroll
    for (int a = 0; a < A; ++a) {
#pragma unroll
        for (int b = 0; b < B; ++b) y[a][b] = x[a + A * b];
        dft<B>(y[a], s);
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
        float2 z[A];
#pragma unroll
        for (int a = 0; a < A; ++a) z[a] = a * b ? cmul(y[a][b], unit<A * B>(a * b, s)) : y[a][b];
        dft<A>(z, s);
#pragma unroll
        for (int a = 0; a < A; ++a) x[b + B * a] = z[a];
    }
}

// X_q = sum_r x_r exp(s 2 pi i r q / R), in place and in order.
template <int R>
__device__ __forceinline__ void dft(float2 (&x)[R], float s) {
    if constexpr (R == 2) {
        const float2 a = x[0];
        x[0] = cadd(a, x[1]);
        x[1] = csub(a, x[1]);
    } else if constexpr (R == 4) {
        const float2 t0 = cadd(x[0], x[2]), t1 = csub(x[0], x[2]), t2 = cadd(x[1], x[3]);
        const float2 t3 = mul_si(csub(x[1], x[3]), s);
        x[0] = cadd(t0, t2);
        x[1] = cadd(t1, t3);
        x[2] = csub(t0, t2);
        x[3] = csub(t1, t3);
    } else if constexpr (R == 8) {
        dft_product<2, 4>(x, s);
    } else if constexpr (R == 9) {
        dft_product<3, 3>(x, s);
    } else if constexpr (R == 16) {
        dft_product<4, 4>(x, s);
    } else {  // odd: sums and differences of the pairs r, R - r
        constexpr int Q = R / 2;
        const float2 x0 = x[0];
        float2 a[Q], b[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            a[k] = cadd(x[k + 1], x[R - 1 - k]);
            b[k] = mul_si(csub(x[k + 1], x[R - 1 - k]), s);
            x[0] = cadd(x[0], a[k]);
        }
#pragma unroll
        for (int q = 1; q <= Q; ++q) {
            float2 u = x0, v = make_float2(0.f, 0.f);
#pragma unroll
            for (int k = 1; k <= Q; ++k) {
                const int m = q * k % R, i = m <= Q ? m : R - m;
                const float2 z = root<R>(i);
                const float c = z.x, d = m <= Q ? z.y : -z.y;
                u = make_float2(fmaf(c, a[k - 1].x, u.x), fmaf(c, a[k - 1].y, u.y));
                v = make_float2(fmaf(d, b[k - 1].x, v.x), fmaf(d, b[k - 1].y, v.y));
            }
            x[q] = cadd(u, v);
            x[R - q] = csub(u, v);
        }
    }
}

// One Stockham stage of radix R on P interleaved sequences: butterfly
// b = k L + j of a sequence takes the elements b + r n / R, turned by
// exp(s 2 pi i j r / (R L)), to k R L + j + q L.  in(i, q): element i of
// sequence q; out(i, q, value).  tw: exp(-2 pi i m / n).
template <int R, bool FIRST, typename In, typename Out>
__device__ __forceinline__ void stage(const MixedArgs &a, int L, unsigned inv, const float2 *__restrict__ tw, In &in,
                                      Out &out) {
    const int nb = a.f.n / R;
    const float s = a.s;
    for (int i = threadIdx.x; i < nb << a.logP; i += blockDim.x) {
        const int q = i & ((1 << a.logP) - 1), b = i >> a.logP;
        float2 x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = in(b + r * nb, q);
        int o = b * R;
        if constexpr (!FIRST) {
            const int k = static_cast<int>(__umulhi(static_cast<unsigned>(b), inv)), j = b - k * L;
            const int step = j * (nb / L);  // j n / (R L)
            o = k * R * L + j;
#pragma unroll
            for (int r = 1; r < R; ++r) {
                const float2 w = __ldg(tw + r * step);
                x[r] = cmul(x[r], make_float2(w.x, -s * w.y));
            }
        }
        dft<R>(x, s);
#pragma unroll
        for (int r = 0; r < R; ++r) out(o + r * L, q, x[r]);
    }
}

template <bool FIRST, typename In, typename Out>
__device__ __forceinline__ void any_stage(const MixedArgs &a, int i, const float2 *__restrict__ tw, In in, Out out) {
    const int L = a.f.done[i];
    const unsigned inv = a.f.inv[i];
    switch (a.f.radix[i]) {
        case 2: stage<2, FIRST>(a, L, inv, tw, in, out); break;
        case 3: stage<3, FIRST>(a, L, inv, tw, in, out); break;
        case 4: stage<4, FIRST>(a, L, inv, tw, in, out); break;
        case 5: stage<5, FIRST>(a, L, inv, tw, in, out); break;
        case 7: stage<7, FIRST>(a, L, inv, tw, in, out); break;
        case 8: stage<8, FIRST>(a, L, inv, tw, in, out); break;
        case 9: stage<9, FIRST>(a, L, inv, tw, in, out); break;
        case 11: stage<11, FIRST>(a, L, inv, tw, in, out); break;
        case 13: stage<13, FIRST>(a, L, inv, tw, in, out); break;
        default: stage<16, FIRST>(a, L, inv, tw, in, out); break;
    }
}

// The first stage (L = 1) of a prime radix p above 13, between the buffers: a
// thread computes output g and p - g of a butterfly from the sums and
// differences of its inputs r and p - r.
__device__ __forceinline__ void prime_stage(const MixedArgs &a, const float2 *__restrict__ tw, const float2 *u, float2 *v) {
    const int p = a.f.radix[0], nb = a.f.n / p, P = a.logP;
    const float s = a.s;
    for (int i = threadIdx.x; i < (p / 2 + 1) * nb << P; i += blockDim.x) {
        const int q = i & ((1 << P) - 1), e = i >> P;
        const int g = static_cast<int>(__umulhi(static_cast<unsigned>(e), a.f.inv_nb)), b = e - g * nb;
        float2 x = u[padded((b << P) + q)], y = make_float2(0.f, 0.f);
        int m = 0;  // r g mod p
#pragma unroll 4
        for (int r = 1; r <= p / 2; ++r) {
            m += g;
            m -= m >= p ? p : 0;
            const float2 w = __ldg(tw + m * nb);  // cos, -sin
            const float2 c = u[padded(((b + r * nb) << P) + q)], d = u[padded(((b + (p - r) * nb) << P) + q)];
            x = make_float2(fmaf(w.x, c.x + d.x, x.x), fmaf(w.x, c.y + d.y, x.y));
            y = make_float2(fmaf(w.y, c.x - d.x, y.x), fmaf(w.y, c.y - d.y, y.y));
        }
        const float2 z = mul_si(y, -s);
        v[padded(((b * p + g) << P) + q)] = cadd(x, z);
        if (g) v[padded(((b * p + p - g) << P) + q)] = csub(x, z);
    }
}

// The transform of P sequences from load(i, q) to store(i, q, value), between
// two buffers of shared memory (element i of sequence q at i P + q): the first
// stage reads and the last writes global memory (at least two stages).
template <typename Load, typename Store>
__device__ __forceinline__ void mixed_fft(float2 *u, const MixedArgs &a, const float2 *__restrict__ tw, Load load,
                                          Store store) {
    const int P = a.logP;
    float2 *v = u + padded(a.f.n << P);
    if (a.f.radix[0] > 16) {
#pragma unroll 4
        for (int e = threadIdx.x; e < a.f.n << P; e += blockDim.x) u[padded(e)] = load(e >> P, e & ((1 << P) - 1));
        __syncthreads();
        prime_stage(a, tw, u, v);
        float2 *t = u;
        u = v;
        v = t;
    } else {
        any_stage<true>(a, 0, tw, load, [=](int i, int q, float2 x) { u[padded((i << P) + q)] = x; });
    }
    __syncthreads();
#pragma unroll 1
    for (int st = 1; st + 1 < a.f.stages; ++st) {
        any_stage<false>(
            a, st, tw, [=](int i, int q) { return u[padded((i << P) + q)]; },
            [=](int i, int q, float2 x) { v[padded((i << P) + q)] = x; });
        __syncthreads();
        float2 *t = u;
        u = v;
        v = t;
    }
    any_stage<false>(a, a.f.stages - 1, tw, [=](int i, int q) { return u[padded((i << P) + q)]; }, store);
}

__device__ __forceinline__ int band_col(int bc, int N2, int n2) { return bc < N2 / 2 ? bc : n2 - N2 + bc; }
__device__ __forceinline__ int band_coef(int bc, int N2) { return bc < N2 / 2 ? bc + N2 / 2 : bc - N2 / 2; }

constexpr int kMixedThreads = 512;

// Type 2, pass 1: P band columns a CTA, padded and deapodized.  A column past
// the band's last repeats that and is not written.
__global__ void __launch_bounds__(kMixedThreads) k_mixed_cols_pad(const float2 *__restrict__ F, float2 *__restrict__ grid,
                                                                  const float *__restrict__ d1,
                                                                  const float *__restrict__ d2,
                                                                  const float2 *__restrict__ tw,
                                                                  const __grid_constant__ MixedArgs a) {
    extern __shared__ float2 sm[];
    start_next();
    const int n1 = a.n1, N1 = a.N1, N2 = a.N2, bc0 = blockIdx.x << a.logP;
    float2 *const cell = grid + static_cast<size_t>(a.H) * a.C + a.H;
    mixed_fft(
        sm, a, tw,
        [&](int r, int q) {
            // rows outside the band load the band's edge: no load waits behind a branch
            const int j = band_coef(min(bc0 + q, N2 - 1), N2);
            const int k1 = r < n1 / 2 ? r : r - n1, i = min(max(k1 + N1 / 2, 0), N1 - 1);
            const float sc = __ldg(d1 + i) * __ldg(d2 + j);
            const float2 f = __ldg(F + static_cast<size_t>(i) * N2 + j);
            return k1 >= -N1 / 2 && k1 < N1 / 2 ? make_float2(f.x * sc, f.y * sc) : make_float2(0.f, 0.f);
        },
        [&](int r, int q, float2 v) {
            if (bc0 + q < N2) cell[static_cast<size_t>(r) * a.C + band_col(bc0 + q, N2, a.n2)] = v;
        });
}

// Type 2, pass 2: a row a CTA, read in its band columns, written with its
// halo columns; the first and last H rows also to the halo rows.
__global__ void __launch_bounds__(kMixedThreads) k_mixed_rows_fill(float2 *__restrict__ grid, const float2 *__restrict__ tw,
                                                                   const __grid_constant__ MixedArgs a) {
    extern __shared__ float2 sm[];
    start_next();
    wait_previous();
    const int n2 = a.n2, N2 = a.N2, r = blockIdx.x, H = a.H;
    float2 *const row = grid + static_cast<size_t>(r + H) * a.C + H;
    const ptrdiff_t dr = static_cast<ptrdiff_t>(r < H ? a.n1 : (r >= a.n1 - H ? -a.n1 : 0)) * a.C;
    mixed_fft(
        sm, a, tw,
        [&](int c, int) {
            const int k2 = c < n2 / 2 ? c : c - n2;
            const float2 v = row[c];  // only the band is from this transform
            return k2 >= -N2 / 2 && k2 < N2 / 2 ? v : make_float2(0.f, 0.f);
        },
        [&](int c, int, float2 v) {
            const int dc = c < H ? n2 : (c >= n2 - H ? -n2 : 0);
            row[c] = v;
            if (dc) row[c + dc] = v;
            if (dr) {
                row[dr + c] = v;
                if (dc) row[dr + c + dc] = v;
            }
        });
}

// Type 1, pass 1: a row a CTA, the halo images of its cells added (no CTA
// writes a halo cell), its band columns written back.
__global__ void __launch_bounds__(kMixedThreads) k_mixed_rows_fold(float2 *__restrict__ grid, const float2 *__restrict__ tw,
                                                                   const __grid_constant__ MixedArgs a) {
    extern __shared__ float2 sm[];
    start_next();
    wait_previous();
    const int n2 = a.n2, N2 = a.N2, r = blockIdx.x, H = a.H;
    float2 *const row = grid + static_cast<size_t>(r + H) * a.C + H;
    const ptrdiff_t dr = static_cast<ptrdiff_t>(r < H ? a.n1 : (r >= a.n1 - H ? -a.n1 : 0)) * a.C;
    mixed_fft(
        sm, a, tw,
        [&](int c, int) {
            // a cell without a side image loads itself: no load waits behind a branch
            const int dc = c < H ? n2 : (c >= n2 - H ? -n2 : 0);
            float2 v = row[c];
            const float2 w = row[c + dc];
            if (dc) v = cadd(v, w);
            if (dr) {
                v = cadd(v, row[dr + c]);
                if (dc) v = cadd(v, row[dr + c + dc]);
            }
            return v;
        },
        [&](int c, int, float2 v) {
            const int k2 = c < n2 / 2 ? c : c - n2;
            if (k2 >= -N2 / 2 && k2 < N2 / 2) row[c] = v;
        });
}

// Type 1, pass 2: P band columns a CTA, cropped to the N1 band rows and
// deapodized into F.
__global__ void __launch_bounds__(kMixedThreads) k_mixed_cols_crop(const float2 *grid, float2 *F,
                                                                   const float *__restrict__ d1,
                                                                   const float *__restrict__ d2,
                                                                   const float2 *__restrict__ tw,
                                                                   const __grid_constant__ MixedArgs a) {
    extern __shared__ float2 sm[];
    wait_previous();
    const int n1 = a.n1, N1 = a.N1, N2 = a.N2, bc0 = blockIdx.x << a.logP;
    const float2 *const cell = grid + static_cast<size_t>(a.H) * a.C + a.H;
    mixed_fft(
        sm, a, tw,
        [&](int r, int q) {
            return __ldcg(cell + static_cast<size_t>(r) * a.C + band_col(min(bc0 + q, N2 - 1), N2, a.n2));
        },
        [&](int r, int q, float2 v) {
            const int k1 = r < n1 / 2 ? r : r - n1;
            if (bc0 + q >= N2 || k1 < -N1 / 2 || k1 >= N1 / 2) return;
            const int i = k1 + N1 / 2, j = band_coef(bc0 + q, N2);
            const float sc = __ldg(d1 + i) * __ldg(d2 + j);
            F[static_cast<size_t>(i) * N2 + j] = make_float2(v.x * sc, v.y * sc);
        });
}

// The factors of n, one prime from 17 to kMixedMaxPrime first, then largest
// first; false if n has others.
bool factor(int n, MixedFft *f) {
    *f = MixedFft{};
    f->n = n;
    int left = n, L = 1;
    auto take = [&](int r) {
        f->radix[f->stages] = r;
        f->done[f->stages] = L;
        f->inv[f->stages] = static_cast<unsigned>((0x100000000ull + L - 1) / L);
        ++f->stages;
        L *= r;
        left /= r;
    };
    int rest = n;
    for (const int r : {2, 3, 5, 7, 11, 13})
        while (rest % r == 0) rest /= r;
    if (rest > 1) {
        for (int d = 17; d * d <= rest; d += 2)
            if (rest % d == 0) return false;  // two of them
        if (rest > kMixedMaxPrime) return false;
        take(rest);
    }
    for (const int r : {16, 13, 11, 9, 8, 7, 5, 4, 3, 2})
        while (left % r == 0) {
            if (f->stages == kMaxStages) return false;
            take(r);
        }
    const int nb = n / f->radix[0];
    f->inv_nb = static_cast<unsigned>((0x100000000ull + nb - 1) / nb);
    return left == 1 && f->stages > 1;
}

MixedArgs mixed_args(const nfft2d_plan_s *p, int sign, int n) {
    const Geom &g = p->g;
    MixedArgs a{};
    factor(n, &a.f);
    a.N1 = p->N1, a.N2 = p->N2, a.n1 = g.n1, a.n2 = g.n2;
    a.H = g.H, a.C = g.C;
    a.s = sign < 0 ? -1.f : 1.f;
    return a;
}

// Columns a CTA: 4 (one sector of 32 bytes a row) while the two buffers leave
// an SM two CTAs, else 2; fewer where that leaves half the SMs without a CTA.
int cols_log(const nfft2d_plan_s *p) {
    int l = p->g.n1 <= 1536 ? 2 : 1;
    while (l > 0 && p->N2 >> l < p->num_sms / 2) --l;
    return l;
}

// Threads a CTA: 4 elements each while the grid is small (latency), else 8 (250
// x 378 coefficients adjoint: 37.1 us with 4, 39.4 with 8; 700 x 702: 94, 84).
int block_threads(const Geom &g, int elems) {
    const int per = 1LL * g.n1 * g.n2 < (1 << 19) ? 4 : 8;
    return std::min(kMixedThreads, std::max(64, (elems / per + 31) / 32 * 32));
}

template <typename Kernel, typename... Args>
cudaError_t launch(Kernel kernel, const nfft2d_plan_s *p, bool after, int blocks, int elems, Args... args) {
    const int smem = 2 * padded(elems) * static_cast<int>(sizeof(float2)) + 16;
    const cudaError_t e = allow_smem(kernel, smem);
    if (e != cudaSuccess) return e;
    if (after) return launch_after(kernel, dim3(blocks), block_threads(p->g, elems), smem, p->stream, args...);
    kernel<<<blocks, block_threads(p->g, elems), smem, p->stream>>>(args...);
    return cudaGetLastError();
}

}  // namespace

// Below 2048 x 2048 cells, and above where both sides have a prime factor of 5 or
// more (powers of 2 and 3 are what cuFFT is best at).  Measured on GB300, w 6, 50 k
// points, coefficients, us, cuFFT with its separate kernels -> here (forward |
// adjoint):
//     50 x 50    25.5 -> 18.9 | 41.3 -> 39.0      250 x 378   36.9 -> 27.1 | 45.2 -> 37.0
//    500 x 500   39.0 -> 34.9 | 53.4 -> 49.9      630 x 630   66.6 -> 53.3 | 81.7 -> 71.8
//   1100 x 900    136 -> 96   |  153 -> 116      1000 x 1000   120 -> 98   |  131 -> 124
//   1100 x 1300   222 -> 137  |  234 -> 165      1920 x 1920   366 -> 306  |  394 -> 384
//   1536 x 1536   241 -> 231  |  234 -> 254      1050 x 1024   111 -> 107  |  127 -> 134
//   1024 x 1024    94 -> 100  |  111 -> 126      2048 x 2048   274 -> 362  |  320 -> 462
// (the last four stay with cuFFT).  Errors fall, 2.5e-7 .. 3.7e-7 -> 2.0e-7.
//
// A prime above 13 costs its own length per element: up to 2^20 cells it beats
// cuFFT's chirp transforms.  Measured on GB300, w 6, 50 k points, coefficients
// (primes), us, cuFFT -> here (forward | adjoint):
//    106 x 134  (53, 67)  38.7 -> 26.7 | 54.6 -> 44.1    374 x 418   (17, 19)  52.0 -> 39.0 | 62.7 -> 51.5
//    244 x 248  (61, 31)  39.8 -> 26.7 | 51.5 -> 41.1    510 x 512   (17)      45.2 -> 39.0 | 60.8 -> 61.4
//    382 x 388  (191, 97) 60.0 -> 72.0 | 71.8 -> 83.5   1230 x 1230  (41)       207 -> 258  |  219 -> 279
bool mixed_fft_eligible(int precision, int n1, int n2) {
    auto side = [&](int n) {
        MixedFft f;
        return n >= 64 && n <= kMixedMaxSide && factor(n, &f) && (f.radix[0] <= 16 || 1LL * n1 * n2 <= 1 << 20);
    };
    auto rest = [](int n) {
        for (const int f : {2, 3})
            while (n % f == 0) n /= f;
        return n;
    };
    return precision == NFFT2D_F32 && side(n1) && side(n2) &&
           (1LL * n1 * n2 < 2048LL * 2048LL || (rest(n1) > 1 && rest(n2) > 1));
}

cudaError_t mixed_type2_cols(const nfft2d_plan_s *p, int sign, const void *F) {
    MixedArgs a = mixed_args(p, sign, p->g.n1);
    a.logP = cols_log(p);
    return launch(k_mixed_cols_pad, p, false, (p->N2 + (1 << a.logP) - 1) >> a.logP, a.n1 << a.logP,
                  static_cast<const float2 *>(F), static_cast<float2 *>(p->grid), static_cast<const float *>(p->deap1),
                  static_cast<const float *>(p->deap2), static_cast<const float2 *>(p->tw1), a);
}

cudaError_t mixed_type2_rows(const nfft2d_plan_s *p, int sign) {
    const MixedArgs a = mixed_args(p, sign, p->g.n2);
    return launch(k_mixed_rows_fill, p, true, a.n1, a.n2, static_cast<float2 *>(p->grid),
                  static_cast<const float2 *>(p->tw2), a);
}

cudaError_t mixed_type1_rows(const nfft2d_plan_s *p, int sign) {
    const MixedArgs a = mixed_args(p, sign, p->g.n2);
    return launch(k_mixed_rows_fold, p, true, a.n1, a.n2, static_cast<float2 *>(p->grid),
                  static_cast<const float2 *>(p->tw2), a);
}

cudaError_t mixed_type1_cols(const nfft2d_plan_s *p, int sign, void *F) {
    MixedArgs a = mixed_args(p, sign, p->g.n1);
    a.logP = cols_log(p);
    return launch(k_mixed_cols_crop, p, true, (p->N2 + (1 << a.logP) - 1) >> a.logP, a.n1 << a.logP,
                  static_cast<const float2 *>(p->grid), static_cast<float2 *>(F), static_cast<const float *>(p->deap1),
                  static_cast<const float *>(p->deap2), static_cast<const float2 *>(p->tw1), a);
}

}  // namespace nfft2d
