// Image pipeline, evaluation metrics and display packing (the reference's
// bindings.h:158-180 group), one thread per output pixel unless said otherwise.
//
// Each kernel keeps the reference's float32 operation order (core/cpu/msplat_cpu.cpp:
// 1609-1745; -fmad=false), so resize, undistortion, packing and depth finalisation
// match it bit for bit. The metrics keep its summation order too: per-pixel terms in
// float, each row summed in double in (x, channel) order, then the rows in order.
#include <cmath>

#include "common.cuh"
#include "kernels.h"
#include "ordered_sums.cuh"
#include "ssim_window.cuh"

namespace msplat {

// Area (box) resample (msplat_cpu.cpp:1609-1639). src: (sh, sw, 4) RGBA8 when u8in,
// else (sh, sw, 3) float.
__global__ void resize_area_kernel(const void *src, int u8in, int sw, int sh, float *dst, int dw, int dh) {
    const int gx = blockIdx.x * blockDim.x + threadIdx.x, gy = blockIdx.y;
    if (gx >= dw || gy >= dh) return;
    const uint8_t *u8 = u8in ? static_cast<const uint8_t *>(src) : nullptr;
    const float *fs = u8in ? nullptr : static_cast<const float *>(src);
    const float sxs = (float)sw / (float)dw, sys = (float)sh / (float)dh;
    const float y0 = (float)gy * sys, y1 = (float)(gy + 1) * sys;
    const int iy0 = (int)y0, iy1 = min((int)ceilf(y1), sh);
    const float x0 = (float)gx * sxs, x1 = (float)(gx + 1) * sxs;
    const int ix0 = (int)x0, ix1 = min((int)ceilf(x1), sw);
    float sr = 0.f, sg = 0.f, sb = 0.f, area = 0.f;
    for (int iy = iy0; iy < iy1; iy++) {
        const float wy = fminf((float)(iy + 1), y1) - fmaxf((float)iy, y0);
        for (int ix = ix0; ix < ix1; ix++) {
            const float wx = fminf((float)(ix + 1), x1) - fmaxf((float)ix, x0);
            const size_t s = (size_t)iy * sw + ix;
            float r, g, b;
            if (u8) {
                r = (float)u8[4 * s] * (1.f / 255.f);
                g = (float)u8[4 * s + 1] * (1.f / 255.f);
                b = (float)u8[4 * s + 2] * (1.f / 255.f);
            } else {
                r = fs[3 * s];
                g = fs[3 * s + 1];
                b = fs[3 * s + 2];
            }
            const float w = wx * wy;
            sr = sr + w * r;
            sg = sg + w * g;
            sb = sb + w * b;
            area += w;
        }
    }
    float *o = dst + 3 * ((size_t)gy * dw + gx);
    o[0] = sr / area;
    o[1] = sg / area;
    o[2] = sb / area;
}

// Brown-Conrady undistortion with bilinear sampling (msplat_cpu.cpp:1641-1669).
__global__ void undistort_kernel(const float *in, int sw, int sh, float fx, float fy, float cx, float cy, float k1,
                                 float k2, float p1, float p2, float k3, int rx, int ry, float *out, int dw, int dh) {
    const int gx = blockIdx.x * blockDim.x + threadIdx.x, gy = blockIdx.y;
    if (gx >= dw || gy >= dh) return;
    const float x = ((float)(gx + rx) + 0.5f - cx) / fx;
    const float y = ((float)(gy + ry) + 0.5f - cy) / fy;
    const float r2 = x * x + y * y;
    const float rad = 1.f + k1 * r2 + k2 * r2 * r2 + k3 * r2 * r2 * r2;
    const float xd = x * rad + 2.f * p1 * x * y + p2 * (r2 + 2.f * x * x);
    const float yd = y * rad + p1 * (r2 + 2.f * y * y) + 2.f * p2 * x * y;
    const float sx = xd * fx + cx - 0.5f, sy = yd * fy + cy - 0.5f;
    const int x0 = (int)floorf(sx), y0 = (int)floorf(sy);
    const float ax = sx - floorf(sx), ay = sy - floorf(sy);
    const int xa = min(max(x0, 0), sw - 1), xb = min(max(x0 + 1, 0), sw - 1);
    const int ya = min(max(y0, 0), sh - 1), yb = min(max(y0 + 1, 0), sh - 1);
    const float *c00 = in + 3 * ((size_t)ya * sw + xa), *c10 = in + 3 * ((size_t)ya * sw + xb);
    const float *c01 = in + 3 * ((size_t)yb * sw + xa), *c11 = in + 3 * ((size_t)yb * sw + xb);
    float *o = out + 3 * ((size_t)gy * dw + gx);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float top = c00[c] * (1.f - ax) + c10[c] * ax;
        const float bot = c01[c] * (1.f - ax) + c11[c] * ax;
        o[c] = top * (1.f - ay) + bot * ay;
    }
}

// Metrics pass 1: the SSIM term of every (pixel, channel) (msplat_cpu.cpp:1675-1712), a
// 32x32 tile of one channel per block: inputs with a 5-pixel halo, clamped to the
// image's edge, and their horizontal moments in shared memory; each thread computes a
// run of consecutive outputs (ssim_window.cuh). 1297 x 840: 213 -> 54 us against two passes
// through a 60-byte-a-pixel buffer of moments, read eleven times.
constexpr int MT = 32, M_IN = MT + 10, M_PIN = M_IN + 1, M_PH = MT + 1;
constexpr int M_RUN_H = 8, M_RUN_V = 4, METRICS_THREADS = 256;
static_assert(MT * (MT / M_RUN_V) == METRICS_THREADS, "one vertical run a thread");

__global__ void __launch_bounds__(METRICS_THREADS) metrics_ssim_kernel(const float *a, const float *b, int h, int w,
                                                                        float *t_ssim) {
    __shared__ float2 in[M_IN * M_PIN];
    __shared__ Moments<M_IN * M_PH> hb;
    const float C1 = 0.0001f, C2 = 0.0009f;
    const int tile = blockIdx.x / 3, c = blockIdx.x - 3 * tile, nbx = (w + MT - 1) / MT;
    const int x0 = tile % nbx * MT, y0 = tile / nbx * MT;
    for (int i = threadIdx.x; i < M_IN * M_IN; i += METRICS_THREADS) {
        const int r = i / M_IN, q = i - r * M_IN;
        const int gy = min(max(y0 - 5 + r, 0), h - 1), gx = min(max(x0 - 5 + q, 0), w - 1);
        const size_t k = ((size_t)gy * w + gx) * 3 + c;
        in[r * M_PIN + q] = make_float2(a[k], b[k]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < M_IN * (MT / M_RUN_H); i += METRICS_THREADS) {
        const int seg = i / M_IN, r = i - seg * M_IN;
        window_moments_h<M_RUN_H>(in + r * M_PIN + seg * M_RUN_H, hb, r * M_PH + seg * M_RUN_H);
    }
    __syncthreads();
    const int q = threadIdx.x % MT, r0 = threadIdx.x / MT * M_RUN_V;
    float2 mu[M_RUN_V], sq[M_RUN_V];
    float xy[M_RUN_V];
    window_moments_v<M_RUN_V, M_PH>(hb, r0 * M_PH + q, mu, sq, xy);
#pragma unroll
    for (int t = 0; t < M_RUN_V; t++) {
        const int y = y0 + r0 + t, x = x0 + q;
        if (x >= w || y >= h) continue;
        const float m12 = mu[t].x * mu[t].y, m1 = mu[t].x * mu[t].x, m2 = mu[t].y * mu[t].y;
        const float num = (2.f * m12 + C1) * (2.f * (xy[t] - m12) + C2);
        const float den = (m1 + m2 + C1) * ((sq[t].x - m1) + (sq[t].y - m2) + C2);
        t_ssim[((size_t)y * w + x) * 3 + c] = num / den;
    }
}

// Metrics pass 2: each row's SSIM terms, |d| and d^2 summed in double in (x, channel)
// order. Bound by the chain of 3 w dependent additions: 42.9 us at 1297 x 840 against
// 951 with one thread a row, whose loads the chain waited for.
__global__ void __launch_bounds__(32 * ORD_WARPS) metrics_rows_kernel(const float *a, const float *b, int h, int w,
                                                                      const float *t_ssim, double *rows) {
    const int n = 3 * w;
    block_row_sums3(h, n, [&](int y, int i) {
        const size_t k = (size_t)y * n + i;
        return Raw3{{t_ssim[k], a[k], b[k]}};
    }, [](const Raw3 &r) {
        const float d = r.v[1] - r.v[2];
        return Terms3{{(double)r.v[0], (double)fabsf(d), (double)d * d}};
    }, rows);
}

// Metrics pass 3: the rows in order, then PSNR / SSIM / L1 (msplat_cpu.cpp:1713-1720).
__global__ void __launch_bounds__(32) metrics_final_kernel(int h, int w, const double *rows, double *out) {
    __shared__ double buf[3 * ORD_PITCH];
    const double s = warp_ordered_sums3(h, [&](int y) {
        return Terms3{{rows[3 * (size_t)y], rows[3 * (size_t)y + 1], rows[3 * (size_t)y + 2]}};
    }, [](const Terms3 &t) { return t; }, buf);
    const double l1 = __shfl_sync(0xffffffffu, s, 1), sq = __shfl_sync(0xffffffffu, s, 2);
    if (threadIdx.x != 0) return;
    const double cnt = (double)h * w * 3, mse = sq / cnt;
    out[0] = mse > 0 ? 10.0 * log10(1.0 / mse) : INFINITY;
    out[1] = s / cnt;
    out[2] = l1 / cnt;
}

// Float RGB to RGBA8 (msplat_cpu.cpp:1723-1734).
__global__ void pack_rgba8_kernel(const float *img, uint32_t n, uint8_t *out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uchar4 o;
    o.x = (uint8_t)(clamp01(img[3 * (size_t)i]) * 255.f);
    o.y = (uint8_t)(clamp01(img[3 * (size_t)i + 1]) * 255.f);
    o.z = (uint8_t)(clamp01(img[3 * (size_t)i + 2]) * 255.f);
    o.w = 255;
    reinterpret_cast<uchar4 *>(out)[i] = o;
}

// Expected depth and alpha from the aux render outputs (msplat_cpu.cpp:1736-1745).
__global__ void finalize_depth_kernel(const float *d, const float *t, uint32_t n, float inv_scale, float *od,
                                      float *oa) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float a = 1.f - t[i];
    oa[i] = a;
    od[i] = a > 1e-4f ? d[i] / a * inv_scale : 0.f;
}

void launch_resize_area(const void *src, int u8in, int sw, int sh, float *dst, int dw, int dh, cudaStream_t st) {
    if (dw <= 0 || dh <= 0) return;
    resize_area_kernel<<<dim3((dw + 127) / 128, dh), 128, 0, st>>>(src, u8in, sw, sh, dst, dw, dh);
}

void launch_undistort(const float *src, int sw, int sh, const float *intr, const float *dist, int rx, int ry,
                      float *dst, int dw, int dh, cudaStream_t st) {
    if (dw <= 0 || dh <= 0) return;
    undistort_kernel<<<dim3((dw + 127) / 128, dh), 128, 0, st>>>(src, sw, sh, intr[0], intr[1], intr[2], intr[3],
                                                                 dist[0], dist[1], dist[2], dist[3], dist[4], rx, ry,
                                                                 dst, dw, dh);
}

void launch_image_metrics(const float *a, const float *b, int h, int w, const MetricsScratch &s, double *out,
                          cudaStream_t st) {
    const int64_t tiles = (int64_t)((w + MT - 1) / MT) * ((h + MT - 1) / MT);
    metrics_ssim_kernel<<<(unsigned)(3 * tiles), METRICS_THREADS, 0, st>>>(a, b, h, w, s.t_ssim);
    metrics_rows_kernel<<<(h + ORD_WARPS - 1) / ORD_WARPS, 32 * ORD_WARPS, 0, st>>>(a, b, h, w, s.t_ssim, s.rows);
    metrics_final_kernel<<<1, 32, 0, st>>>(h, w, s.rows, out);
}

void launch_pack_rgba8(const float *img, uint32_t n, uint8_t *out, cudaStream_t st) {
    if (n == 0) return;
    pack_rgba8_kernel<<<(n + 255) / 256, 256, 0, st>>>(img, n, out);
}

void launch_finalize_depth(const float *d, const float *t, uint32_t n, float inv_scale, float *od, float *oa,
                           cudaStream_t st) {
    if (n == 0) return;
    finalize_depth_kernel<<<(n + 255) / 256, 256, 0, st>>>(d, t, n, inv_scale, od, oa);
}

}  // namespace msplat
