// The 11-tap Gaussian window (sigma 1.5) over shared-memory rows and columns, for the
// SSIM loss and the evaluation metrics.
//
// Each function computes RUN consecutive outputs in one thread: it walks the RUN + 10
// inputs in order and adds each to the outputs it belongs to, so every value is loaded
// once for all of them, and an output still adds its taps k = 0 .. 10 in order.
// Products and sums are rounded separately, as the reference's loops do (core/cpu/
// msplat_cpu.cpp:669-785, :1675-1712); pairs of values go through the packed FP32
// instructions, two IEEE operations each. A packed product is written as
// fma(a, b, -0), which rounds exactly as a * b does and cannot be fused with the
// addition that follows it (the compiler fuses packed mul and add, .rn or not, also
// where the -0 is a literal: it comes from constant memory).
#pragma once

#include "common.cuh"

namespace msplat {

constexpr int WIN_TAPS = 11;

// The window's weights (core/cpu/msplat_cpu.cpp:40-45); it is symmetric.
__device__ __forceinline__ constexpr float win_weight(int k) {
    return k == 0 || k == 10 ? 0.0010283801f
           : k == 1 || k == 9 ? 0.0075987581f
           : k == 2 || k == 8 ? 0.0360007721f
           : k == 3 || k == 7 ? 0.1093606895f
           : k == 4 || k == 6 ? 0.2130055377f
                              : 0.2660117249f;
}

__device__ __forceinline__ f32x2 pack2(float2 v) { return pack2(v.x, v.y); }
static __constant__ float kMinusZero = -0.f;
// a * b, each half rounded once
__device__ __forceinline__ f32x2 prod2(f32x2 a, f32x2 b) { return fma2(a, b, pack2(kMinusZero, kMinusZero)); }

// The five moment sums of (x, y) at one position: (x, y), (x^2, y^2) and xy.
template <int N>
struct Moments {
    float2 mu[N], sq[N];
    float xy[N];
};

// Weighted moment sums along a row: outputs o .. o + RUN - 1 of `out` from the inputs
// in[0 .. RUN + 9].
template <int RUN, int N>
__device__ __forceinline__ void window_moments_h(const float2 *in, Moments<N> &out, int o) {
    f32x2 mu[RUN], sq[RUN];
    float xy[RUN];
#pragma unroll
    for (int t = 0; t < RUN; t++) {
        mu[t] = sq[t] = pack2(0.f, 0.f);
        xy[t] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < RUN + WIN_TAPS - 1; i++) {
        const float2 v = in[i];
        const f32x2 v2 = pack2(v);
#pragma unroll
        for (int t = 0; t < RUN; t++) {
            const int k = i - t;
            if (k < 0 || k >= WIN_TAPS) continue;
            const f32x2 p = prod2(pack2(win_weight(k), win_weight(k)), v2);
            mu[t] = add2(mu[t], p);
            sq[t] = add2(sq[t], prod2(p, v2));
            xy[t] = xy[t] + unpack2(p).x * v.y;
        }
    }
#pragma unroll
    for (int t = 0; t < RUN; t++) {
        out.mu[o + t] = unpack2(mu[t]);
        out.sq[o + t] = unpack2(sq[t]);
        out.xy[o + t] = xy[t];
    }
}

// Weighted sums of a column of moments (rows of PITCH): RUN outputs from the rows
// starting at m[o].
template <int RUN, int PITCH, int N>
__device__ __forceinline__ void window_moments_v(const Moments<N> &m, int o, float2 mu[RUN], float2 sq[RUN],
                                                 float xy[RUN]) {
    f32x2 a[RUN], b[RUN];
#pragma unroll
    for (int t = 0; t < RUN; t++) {
        a[t] = b[t] = pack2(0.f, 0.f);
        xy[t] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < RUN + WIN_TAPS - 1; i++) {
        const f32x2 va = pack2(m.mu[o + i * PITCH]), vb = pack2(m.sq[o + i * PITCH]);
        const float vc = m.xy[o + i * PITCH];
#pragma unroll
        for (int t = 0; t < RUN; t++) {
            const int k = i - t;
            if (k < 0 || k >= WIN_TAPS) continue;
            const f32x2 wk = pack2(win_weight(k), win_weight(k));
            a[t] = add2(a[t], prod2(wk, va));
            b[t] = add2(b[t], prod2(wk, vb));
            xy[t] = xy[t] + win_weight(k) * vc;
        }
    }
#pragma unroll
    for (int t = 0; t < RUN; t++) {
        mu[t] = unpack2(a[t]);
        sq[t] = unpack2(b[t]);
    }
}

// Weighted sums of three values (v12, v3): RUN outputs from the entries o, o + STEP, ...
template <int RUN, int STEP>
__device__ __forceinline__ void window_sums(const float2 *v12, const float *v3, int o, float2 s12[RUN],
                                            float s3[RUN]) {
    f32x2 a[RUN];
#pragma unroll
    for (int t = 0; t < RUN; t++) {
        a[t] = pack2(0.f, 0.f);
        s3[t] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < RUN + WIN_TAPS - 1; i++) {
        const f32x2 va = pack2(v12[o + i * STEP]);
        const float vb = v3[o + i * STEP];
#pragma unroll
        for (int t = 0; t < RUN; t++) {
            const int k = i - t;
            if (k < 0 || k >= WIN_TAPS) continue;
            a[t] = add2(a[t], prod2(pack2(win_weight(k), win_weight(k)), va));
            s3[t] = s3[t] + win_weight(k) * vb;
        }
    }
#pragma unroll
    for (int t = 0; t < RUN; t++) s12[t] = unpack2(a[t]);
}

}  // namespace msplat
