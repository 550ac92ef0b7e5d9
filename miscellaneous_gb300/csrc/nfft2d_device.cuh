// nfft2d_device.cuh -- device helpers: TMA / mbarrier / bulk-group inline PTX
// (sm_90+ forms, compiled for sm_103a) and the window pair in FP32 and FP64.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "nfft2d_internal.h"

namespace nfft2d {

// Spin bound for every device-side wait.  mbarrier.try_wait suspends for a
// hardware-defined time per call, so this bounds the wait to well under a
// second; on expiry the kernel latches kErrTimeout and returns.
constexpr uint32_t kSpinLimit = 1u << 22;

// ---------------------------------------------------------------------------
// shared-memory / async-proxy primitives
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Make mbarrier initialisation and prior generic-proxy shared-memory
// accesses visible to the async proxy (TMA).
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// One arrival on an mbarrier (no transaction bytes).
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, uint32_t limit = kSpinLimit) {
    for (uint32_t i = 0; i < limit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// 2D tiled TMA load global -> shared, completion signalled on an mbarrier.
// x is the innermost coordinate in elements of the tensor map (must make
// x * elemsize a multiple of 16 bytes), y the row.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// 2D tiled TMA reduction shared -> global: global[box] += shared[box] (f32 add).
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap *map, const void *src, int x, int y) {
    asm volatile(
        "cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group"
        " [%0, {%1, %2}], [%3];" ::"l"(reinterpret_cast<uint64_t>(map)),
        "r"(x), "r"(y), "r"(smem_u32(src))
        : "memory");
}

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Wait until at most one bulk group is still reading its shared-memory source.
__device__ __forceinline__ void bulk_wait_read_le1() {
    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}
// Wait until every committed bulk group has completed (writes performed).
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Programmatic dependent launch.  start_next: the next kernel of the stream, if
// launched with launch_after, may become resident once every CTA of this one
// has come here.  wait_previous: until the kernels before have completed and
// their writes are visible; returns at once in a kernel launched plainly.
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void latch_error(int *status, int bit) { atomicOr(status + 1, bit); }

// ---------------------------------------------------------------------------
// barrier of a cooperative grid of kGridCtas CTAs (all resident: one an SM)
// ---------------------------------------------------------------------------
constexpr int kGridCtas = 128;
// What any CTA wrote before it arrived at a barrier (1, 2, ...), every thread of
// the kernel sees after the wait.  False, latched, if the wait runs out: the CTA
// leaves, by grid_done as on every way out, and so do the others, by their own
// waits.  give_up: the barrier whose waits all run out at once (self-test), or 0.
__device__ __forceinline__ void grid_arrive(int *status) {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(status + kBarrierWord) : "memory");
}
__device__ __forceinline__ bool grid_wait(int *status, int barrier, int give_up) {
    __shared__ int ok;
    if (threadIdx.x == 0) {
        const int target = barrier * kGridCtas;
        int seen = 0;
        uint32_t spins = 0;
        do
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(status + kBarrierWord) : "memory");
        while (seen < target && ++spins < kSpinLimit && barrier != give_up);
        ok = seen >= target && barrier != give_up;
        if (!ok) latch_error(status, kErrTimeout);
    }
    __syncthreads();
    return ok != 0;
}
__device__ __forceinline__ bool grid_barrier(int *status, int barrier, int give_up) {
    grid_arrive(status);
    return grid_wait(status, barrier, give_up);
}
// The last CTA to come here leaves the barrier's words zero for the next launch,
// whether or not a wait has run out: every CTA ends with this, and none arrives
// at a barrier after it.  `failed`: a wait of this CTA has run out.  True in one
// thread of the last CTA, if any has; what a failed CTA wrote, and what others
// wrote before they arrived at a barrier, is in memory by then.
__device__ __forceinline__ bool grid_done(int *status, bool failed) {
    constexpr int kFailed = 1 << 16;
    __syncthreads();
    if (threadIdx.x != 0) return false;
    if (failed) __threadfence();
    const int sum = atomicAdd(status + kBarrierWord + 1, failed ? kFailed + 1 : 1) + (failed ? kFailed + 1 : 1);
    if ((sum & (kFailed - 1)) != kGridCtas) return false;
    status[kBarrierWord] = 0;
    status[kBarrierWord + 1] = 0;
    return sum >= kFailed;
}

// ---------------------------------------------------------------------------
// Window pair.  The reference window (NFFT1_2D.m:34-36, NFFT2_2D.cu:112-122)
//     phi_hat(u) = (1/pi) sinh(alpha s)/s,  s = sqrt(K^2 - u^2)
// (sin form for |u| > K) is used here normalised to 1 at u = 0:
//     w(u) = cn sinh(alpha s)/s,  cn = K / sinh(alpha K);
// the factor sinh(alpha K)/(pi K) moves into the deapodisation table.
// A tap of a point with offset t in [-1/2, 1/2] at grid offset m sits at
// u = t - m; K^2 - u^2 is formed as ((K+m) - t) * ((K-m) + t), a product of
// two well-conditioned factors, so its relative error stays near 1 ulp.
// ---------------------------------------------------------------------------

// Interior tap (|m| < K, so s >= sqrt(K - 1/4)): with cosh/sinh ~ e^{alpha s}/2
//     w = kp * exp(alpha (s - K)) / s,  s - K = -u^2 / (s + K),
// evaluated through the well-conditioned difference -u^2/(s+K); for K <= 3
// the dropped factor (1 - e^{-2 alpha s}) is restored.
template <int K>
__device__ __forceinline__ float win_interior_f32(float t, int m, float alpha, float kp) {
    const float pa = static_cast<float>(K + m) - t;
    const float pb = static_cast<float>(K - m) + t;
    const float P = pa * pb;
    const float r = rsqrtf(P);
    const float s = P * r;
    const float u = t - static_cast<float>(m);
    const float x = __fdividef(-alpha * (u * u), s + static_cast<float>(K));
    float w = kp * __expf(x) * r;
    if (K <= 3) w *= 1.0f - __expf(-2.0f * alpha * s);
    return w;
}

// Edge tap (m = -K or m = K): full formula, both branches.
template <int K>
__device__ __forceinline__ float win_edge_f32(float t, int m, float alpha, float cn) {
    const float pa = static_cast<float>(K + m) - t;
    const float pb = static_cast<float>(K - m) + t;
    const float P = pa * pb;
    const float s = sqrtf(fabsf(P));
    const float as = alpha * s;
    if (s == 0.0f) return cn * alpha;
    const float v = (P > 0.0f) ? sinhf(as) : __sinf(as);  // |as| < 13 here
    return cn * v / s;
}

template <int K>
__device__ __forceinline__ void weights_f32(float t, float (&w)[2 * K + 1], float alpha, float cn, float kp) {
#pragma unroll
    for (int a = 0; a <= 2 * K; ++a) {
        const int m = a - K;
        if (a == 0 || a == 2 * K)
            w[a] = win_edge_f32<K>(t, m, alpha, cn);
        else
            w[a] = win_interior_f32<K>(t, m, alpha, kp);
    }
}

// The taps of ND points (the two dimensions of one point, or one dimension).
// The window is even, so taps m and -m share one pair of half-degree
// polynomials in u = t^2 (coefficients read from kernel parameter space),
//     w(t - m) = c0 + t (O + t E),   w(t + m) = c0 - t (O - t E),
// and all share every coefficient read: for both dimensions 72 FMAs (64 of
// them packed) and 32 constant reads a point at K = 6, where a Horner run per
// tap and dimension took 126 of each.  Rounding as a Horner run's (rms 9.1e-9
// against 8.9e-9).
template <int K, int ND>
__device__ __forceinline__ void weights_even(const float (&ts)[ND], float (*const (&ws)[ND])[2 * K + 1],
                                             const WinPoly &P) {
    constexpr int D = poly_degree(K);
    constexpr int DE = D - (D & 1), DO = D - 1 + (D & 1);  // highest even and odd power
#pragma unroll
    for (int j = 0; j < K / 2; ++j) {  // taps (2j, 2j+1) and their mirror images
        float2 e[ND], o[ND], u[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            u[d] = make_float2(ts[d] * ts[d], ts[d] * ts[d]);
            e[d] = *reinterpret_cast<const float2 *>(&P.c[DE][2 * j]);
            o[d] = *reinterpret_cast<const float2 *>(&P.c[DO][2 * j]);
        }
#pragma unroll
        for (int k = DE - 2; k > 0; k -= 2)
#pragma unroll
            for (int d = 0; d < ND; ++d) e[d] = __ffma2_rn(e[d], u[d], *reinterpret_cast<const float2 *>(&P.c[k][2 * j]));
#pragma unroll
        for (int k = DO - 2; k > 0; k -= 2)
#pragma unroll
            for (int d = 0; d < ND; ++d) o[d] = __ffma2_rn(o[d], u[d], *reinterpret_cast<const float2 *>(&P.c[k][2 * j]));
        const float2 c0 = *reinterpret_cast<const float2 *>(&P.c[0][2 * j]);
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const float2 t = make_float2(ts[d], ts[d]), m = make_float2(-ts[d], -ts[d]);
            const float2 a = __ffma2_rn(t, __ffma2_rn(t, e[d], o[d]), c0);
            const float2 b = __ffma2_rn(m, __ffma2_rn(m, e[d], o[d]), c0);
            float(&w)[2 * K + 1] = *ws[d];
            w[2 * j] = a.x;
            w[2 * j + 1] = a.y;
            w[2 * K - 2 * j] = b.x;
            w[2 * K - 2 * j - 1] = b.y;
        }
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const float t = ts[d], u = t * t;
        float(&w)[2 * K + 1] = *ws[d];
        if constexpr (K & 1) {  // the pair next to the centre
            float e = P.c[DE][K - 1], o = P.c[DO][K - 1];
#pragma unroll
            for (int k = DE - 2; k > 0; k -= 2) e = fmaf(e, u, P.c[k][K - 1]);
#pragma unroll
            for (int k = DO - 2; k > 0; k -= 2) o = fmaf(o, u, P.c[k][K - 1]);
            w[K - 1] = fmaf(t, fmaf(t, e, o), P.c[0][K - 1]);
            w[K + 1] = fmaf(-t, fmaf(-t, e, o), P.c[0][K - 1]);
        }
        float e = P.c[DE][K];
#pragma unroll
        for (int k = DE - 2; k >= 0; k -= 2) e = fmaf(e, u, P.c[k][K]);
        w[K] = e;
    }
}

template <int K>
__device__ __forceinline__ void weights_poly2(float t1, float t2, float (&w1)[2 * K + 1], float (&w2)[2 * K + 1],
                                              const WinPoly &P) {
    const float ts[2] = {t1, t2};
    float(*const ws[2])[2 * K + 1] = {&w1, &w2};
    weights_even<K, 2>(ts, ws, P);
}

// The taps of one dimension, a Horner run a tap (two taps per packed FMA).  More
// FMAs than the half-degree form, but shorter chains: faster where a thread
// forms both dimensions' 15 or 17 weights at once from the registers of 24 warps
// an SM (the direct gather at w 7 and 8).
template <int K>
__device__ __forceinline__ void weights_poly(float t, float (&w)[2 * K + 1], const WinPoly &P) {
    constexpr int D = poly_degree(K);
    const float2 tt = make_float2(t, t);
    float2 acc[K];
    float last = P.c[D][2 * K];
#pragma unroll
    for (int j = 0; j < K; ++j) acc[j] = *reinterpret_cast<const float2 *>(&P.c[D][2 * j]);
#pragma unroll
    for (int d = D - 1; d >= 0; --d) {
#pragma unroll
        for (int j = 0; j < K; ++j) acc[j] = __ffma2_rn(acc[j], tt, *reinterpret_cast<const float2 *>(&P.c[d][2 * j]));
        last = fmaf(last, t, P.c[d][2 * K]);
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
        w[2 * j] = acc[j].x;
        w[2 * j + 1] = acc[j].y;
    }
    w[2 * K] = last;
}

// The taps and their derivatives d/dt from the same polynomials: Horner for
// value and slope together (slope = slope * t + value before each value
// step), two taps per packed FMA.  The slope of the fit differs from the
// closed form by less than 1e-7 of the window's peak slope.
template <int K>
__device__ __forceinline__ void weights_poly_d(float t, float (&w)[2 * K + 1], float (&dw)[2 * K + 1],
                                               const WinPoly &P) {
    constexpr int D = poly_degree(K);
    const float2 tt = make_float2(t, t);
    float2 acc[K], dacc[K];
    float last = P.c[D][2 * K], dlast = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        acc[j] = *reinterpret_cast<const float2 *>(&P.c[D][2 * j]);
        dacc[j] = make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int d = D - 1; d >= 0; --d) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
            dacc[j] = __ffma2_rn(dacc[j], tt, acc[j]);
            acc[j] = __ffma2_rn(acc[j], tt, *reinterpret_cast<const float2 *>(&P.c[d][2 * j]));
        }
        dlast = fmaf(dlast, t, last);
        last = fmaf(last, t, P.c[d][2 * K]);
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
        w[2 * j] = acc[j].x;
        w[2 * j + 1] = acc[j].y;
        dw[2 * j] = dacc[j].x;
        dw[2 * j + 1] = dacc[j].y;
    }
    w[2 * K] = last;
    dw[2 * K] = dlast;
}

// FP64 taps of both dimensions from the plan's polynomials (WinPoly64): taps
// K - m and K + m share one pair of half-degree polynomials, and both
// dimensions every coefficient read.
template <int K>
__device__ __forceinline__ void weights_f64(double t1, double t2, double (&w1)[2 * K + 1], double (&w2)[2 * K + 1],
                                            const WinPoly64 &P) {
    const double ts[2] = {t1, t2}, us[2] = {t1 * t1, t2 * t2};
    double *const ws[2] = {w1, w2};
#pragma unroll
    for (int a = 0; a <= K; ++a) {
        double e[2], o[2];
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            e[d] = P.e[kPoly64 - 1][a];
            o[d] = P.o[kPoly64 - 1][a];
        }
#pragma unroll
        for (int i = kPoly64 - 2; i >= 0; --i)
#pragma unroll
            for (int d = 0; d < 2; ++d) {
                if (i > 0 || a == K) e[d] = fma(e[d], us[d], P.e[i][a]);
                if (a < K) o[d] = fma(o[d], us[d], P.o[i][a]);
            }
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            if (a == K) {
                ws[d][K] = e[d];
            } else {
                ws[d][a] = fma(ts[d], fma(ts[d], e[d], o[d]), P.e[0][a]);
                ws[d][2 * K - a] = fma(-ts[d], fma(-ts[d], e[d], o[d]), P.e[0][a]);
            }
        }
    }
}

// Slopes of the FP64 taps, the reference formula's derivative directly.
template <int K>
__device__ __forceinline__ void dweights_f64(double t, double (&dw)[2 * K + 1], double alpha, double cn) {
#pragma unroll
    for (int a = 0; a <= 2 * K; ++a) {
        const int m = a - K;
        const double pa = static_cast<double>(K + m) - t;
        const double pb = static_cast<double>(K - m) + t;
        const double P = pa * pb;
        const double u = t - static_cast<double>(m);
        const double a2 = alpha * alpha;
        double gp;
        if (fabs(a2 * P) < 1.0) {
            double term = alpha * a2 / 6.0, acc = 0.0;
#pragma unroll 1
            for (int n = 1; n < 24; ++n) {
                acc += n * term;
                term *= a2 * P / ((2.0 * n + 2.0) * (2.0 * n + 3.0));
            }
            gp = acc;
        } else if (P > 0.0) {
            const double s = sqrt(P), as = alpha * s;
            gp = (as * cosh(as) - sinh(as)) / (2.0 * s * P);
        } else {
            const double s = sqrt(-P), as = alpha * s;
            gp = -(as * cos(as) - sin(as)) / (2.0 * s * (-P));
        }
        dw[a] = cn * gp * (-2.0 * u);
    }
}

// Error-free transformation (Knuth TwoSum): s + e == a + b exactly.  The
// _rn intrinsics keep the compiler from contracting or reassociating.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    const float bp = __fsub_rn(s, a);
    const float ap = __fsub_rn(s, bp);
    e = __fadd_rn(__fsub_rn(a, ap), __fsub_rn(b, bp));
}

}  // namespace nfft2d
