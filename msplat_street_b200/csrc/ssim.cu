// Fused L1 + SSIM loss, forward and backward, in one kernel.
//
// The reference runs three row passes with two (H, W, 15) float intermediates in
// memory (ssim_h_fwd, ssim_fused_v_fwd_h_bwd, ssim_v_bwd; core/cpu/msplat_cpu.cpp:
// 669-785). Here each CTA owns a 32x32 output tile of one channel and keeps every
// intermediate in shared memory: inputs with a 10-pixel halo, the horizontal moment
// sums, the SSIM derivative fields on the 5-pixel halo, and their horizontal
// back-convolution. HBM traffic is the minimum: read render + target once (plus halo),
// write v_rendered once.
//
// Semantics kept exactly: zero-padded 11-tap Gaussian window (sigma 1.5), C1 = 1e-4,
// C2 = 9e-4; loss per pixel w * (1 - SSIM/3) + (1 - w) * L1/3 summed in double;
// v_rendered = inv_n * (-w * dSSIM + (1 - w) * sign(render - target)). Each output's
// taps are added in the reference's order, every product and sum rounded separately
// (ssim_window.cuh), so the derivative fields equal the reference's bit for bit; the
// loss differs only in its double-precision sum (SSIM and L1 summed per channel, each
// float term widened first). Per-block partial sums are reduced in a fixed order.
#include "common.cuh"
#include "kernels.h"
#include "ssim_window.cuh"

namespace msplat {

constexpr int ST = 32;          // output tile edge
constexpr int SH_IN = ST + 20;  // input rows / cols with the 10-pixel halo
constexpr int SH_F = ST + 10;   // derivative-field rows / cols (5-pixel halo)
// A thread computes a run of consecutive outputs of one row or column, each value it
// reads from shared memory serving every output of the run: 7 of a row's (column's) 42
// horizontal moments (derivative fields), 8 of 32 back-convolutions, 4 of 32 pixels.
// 320 threads cover the first pass's 52 x 6 runs at once.
constexpr int RUN_H = 7, RUN_V = 7, RUN_B = 8, RUN_O = 4;
constexpr int SSIM_THREADS = 320;
static_assert(SH_F % RUN_H == 0 && SH_F % RUN_V == 0 && ST % RUN_B == 0 && ST % RUN_O == 0, "whole runs");
static_assert(ST * (ST / RUN_O) <= SSIM_THREADS, "one run of output pixels a thread, at most");

// Row pitches are odd in float2 units: lanes along a column or a row both touch 32
// different banks. Two arrays share the place of two that are read no more.
constexpr int P_IN = SH_IN + 1, P_F = SH_F + 1, P_D = ST + 1;
struct SsimSmem {
    union {
        float2 in[SH_IN * P_IN];  // (target, render): rows y0-10.., cols x0-10..
        struct {
            float2 f12[SH_F * P_F];  // derivative fields: rows y0-5.., cols x0-5..
            float f3[SH_F * P_F];
        };
    };
    union {
        Moments<SH_IN * P_F> hb;  // horizontal moments: rows y0-10.., cols x0-5..
        struct {
            float2 d12[SH_F * P_D];  // horizontal back-convolution: rows y0-5.., cols x0..
            float d3[SH_F * P_D];
        };
    };
    double red[SSIM_THREADS / 32];
};

// One 32x32 output tile (bx, by) of channel c of one image; its share of the loss goes
// to a.partials[pidx]. Every thread of the block calls it.
__device__ __forceinline__ void ssim_block(const SsimArgs &a, int bx, int by, int c, int pidx, SsimSmem &s) {
    const int W = a.W, H = a.H;
    const int x0 = bx * ST, y0 = by * ST;
    const float w = a.ssim_weight;
    // 1. inputs, zero outside the image
    constexpr int PER = (SH_IN * SH_IN + SSIM_THREADS - 1) / SSIM_THREADS;
    float2 v[PER];  // all loads before the first store
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int i = threadIdx.x + k * SSIM_THREADS, r = i / SH_IN, q = i - r * SH_IN;
        const int gy = y0 - 10 + r, gx = x0 - 10 + q;
        v[k] = make_float2(0.f, 0.f);
        if (i < SH_IN * SH_IN && gy >= 0 && gy < H && gx >= 0 && gx < W) {
            const size_t idx = ((size_t)gy * W + gx) * 3 + c;
            v[k] = make_float2(a.gt[idx], a.img[idx]);
        }
    }
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int i = threadIdx.x + k * SSIM_THREADS, r = i / SH_IN, q = i - r * SH_IN;
        if (i < SH_IN * SH_IN) s.in[r * P_IN + q] = v[k];
    }
    __syncthreads();
    // this thread's output pixels (pass 5): column ox, rows oy .. oy + RUN_O - 1
    const int ox = threadIdx.x % ST, oy = threadIdx.x / ST * RUN_O;
    const bool owner = threadIdx.x < ST * (ST / RUN_O);
    float2 own[RUN_O];
    double l1 = 0.0, ssim = 0.0;
    if (owner) {
#pragma unroll
        for (int t = 0; t < RUN_O; t++) {
            own[t] = s.in[(oy + t + 10) * P_IN + ox + 10];
            if (y0 + oy + t < H && x0 + ox < W) l1 += (double)fabsf(own[t].x - own[t].y);
        }
    }
    // 2. horizontal moments at cols x0-5 .. x0+ST+5 (core/cpu/msplat_cpu.cpp:669-696)
    for (int i = threadIdx.x; i < SH_IN * (SH_F / RUN_H); i += SSIM_THREADS) {
        const int seg = i / SH_IN, r = i - seg * SH_IN;
        window_moments_h<RUN_H>(s.in + r * P_IN + seg * RUN_H, s.hb, r * P_F + seg * RUN_H);
    }
    __syncthreads();
    // 3. vertical sums, SSIM terms and derivative fields (:698-736); rows outside the
    // image have zero moments, which change no sum
    for (int i = threadIdx.x; i < SH_F * (SH_F / RUN_V); i += SSIM_THREADS) {
        const int seg = i / SH_F, q = i - seg * SH_F, r0 = seg * RUN_V;
        float2 mu[RUN_V], sq[RUN_V];
        float xy[RUN_V];
        window_moments_v<RUN_V, P_F>(s.hb, r0 * P_F + q, mu, sq, xy);
        const int gx = x0 - 5 + q;
#pragma unroll
        for (int t = 0; t < RUN_V; t++) {
            const int r = r0 + t, gy = y0 - 5 + r;
            float f1 = 0.f, f2 = 0.f, f3 = 0.f;
            if (gy >= 0 && gy < H && gx >= 0 && gx < W) {
                const float mx = mu[t].x, my = mu[t].y;
                const float vx = sq[t].x - mx * mx, vy = sq[t].y - my * my, cv = xy[t] - mx * my;
                const float A = 2.0f * mx * my + 0.0001f, B = 2.0f * cv + 0.0009f;
                const float Cd = mx * mx + my * my + 0.0001f, D = vx + vy + 0.0009f;
                const float iCD = 1.0f / (Cd * D);
                const float dmu = 2.0f * B * (mx * Cd - A * my) / (Cd * Cd * D);
                const float dsyq = -A * B * iCD / D, dsxy = 2.0f * A * iCD;
                f1 = dmu - 2.0f * my * dsyq - mx * dsxy;
                f2 = 2.0f * dsyq;
                f3 = dsxy;
                if (r >= 5 && r < 5 + ST && q >= 5 && q < 5 + ST) ssim += (double)((A * B) / (Cd * D));
            }
            s.f12[r * P_F + q] = make_float2(f1, f2);
            s.f3[r * P_F + q] = f3;
        }
    }
    __syncthreads();
    // 4. horizontal back-convolution at rows y0-5 .. y0+ST+5, cols x0 .. (:737-747)
    for (int i = threadIdx.x; i < SH_F * (ST / RUN_B); i += SSIM_THREADS) {
        const int seg = i / SH_F, r = i - seg * SH_F, q0 = seg * RUN_B;
        float2 a12[RUN_B];
        float a3[RUN_B];
        window_sums<RUN_B, 1>(s.f12, s.f3, r * P_F + q0, a12, a3);
#pragma unroll
        for (int t = 0; t < RUN_B; t++) {
            s.d12[r * P_D + q0 + t] = a12[t];
            s.d3[r * P_D + q0 + t] = a3[t];
        }
    }
    __syncthreads();
    // 5. vertical back-convolution and the pixel gradient (:760-785)
    if (owner) {
        float2 a12[RUN_O];
        float a3[RUN_O];
        window_sums<RUN_O, P_D>(s.d12, s.d3, oy * P_D + ox, a12, a3);
#pragma unroll
        for (int t = 0; t < RUN_O; t++) {
            const int gy = y0 + oy + t, gx = x0 + ox;
            if (gy >= H || gx >= W) continue;
            const float gv = own[t].x, rv = own[t].y;
            const float vs = a12[t].x + rv * a12[t].y + gv * a3[t];
            const float vl = (gv > rv) ? -1.0f : ((gv < rv) ? 1.0f : 0.0f);
            a.v_out[((size_t)gy * W + gx) * 3 + c] = a.inv_n * (-w * vs + (1.0f - w) * vl);
        }
    }
    // this channel's third of the tile's loss, summed in double in a fixed order; the
    // constant w / 3 of every pixel enters once, from thread 0
    double sum = ((double)(1.0f - w) * l1 - (double)w * ssim) / 3.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) s.red[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = (double)w * ((double)min(ST, W - x0) * min(ST, H - y0)) / 3.0;
        for (int i = 0; i < SSIM_THREADS / 32; i++) t += s.red[i];
        a.partials[pidx] = t;
    }
}

// Block b of an image: tile b / 3, channel b % 3.
//
// Bound by FP32 issue: about 640 separately rounded operations a pixel and channel,
// halo included. 1024 x 512: 92 -> 55 us, 256 x 256: 33 -> 14 us against the form that
// computed one output a thread and step (two shared loads a tap) with a tile's channels
// one after another; the channels as blocks of their own triple the blocks of a small
// frame, and the inputs' loads all start before the first is stored (58 and 15.5 us where
// they did not). A packed instruction holds the FMA pipe as long as its two scalars:
// packing the window sums' third value as well left the time where it was.
__global__ void __launch_bounds__(SSIM_THREADS, 3) ssim_loss_kernel(SsimArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SsimSmem &s = *reinterpret_cast<SsimSmem *>(smem_raw);
    const int b = blockIdx.x, tile = b / 3, nbx = (a.W + ST - 1) / ST;
    ssim_block(a, tile % nbx, tile / nbx, b - 3 * tile, b, s);
}

// Persistent loss over the blocks of a batch of images (each with its own size,
// target and gradient output), pulling global block ids from a counter. Block b of
// view v writes partial boff[v] + (its index within the view), so each view's
// partials sit in the order the single-image kernel writes them.
__global__ void __launch_bounds__(SSIM_THREADS, 3) ssim_loss_batch_kernel(const SsimArgs *views, const int *boff,
                                                                       int n_views, int *counter) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SsimSmem &s = *reinterpret_cast<SsimSmem *>(smem_raw);
    __shared__ int s_blk;
    const int total = boff[n_views];
    for (;;) {
        if (threadIdx.x == 0) s_blk = atomicAdd(counter, 1);
        __syncthreads();
        const int b = s_blk;
        __syncthreads();
        if (b >= total) break;
        const int v = find_view(boff, n_views, b);
        const SsimArgs a = views[v];
        const int lb = b - boff[v], tile = lb / 3, nbx = (a.W + ST - 1) / ST;
        ssim_block(a, tile % nbx, tile / nbx, lb - 3 * tile, b, s);
        __syncthreads();
    }
}

__device__ __forceinline__ void loss_finalize_block(const double *partials, int nb, double npix, float *loss) {
    __shared__ double red[32];
    double s = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) s += partials[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += red[i];
        *loss = (float)(t / npix);
    }
}

__global__ void loss_finalize_kernel(const double *partials, int nb, double npix, float *loss) {
    loss_finalize_block(partials, nb, npix, loss);
}

// One 1024-thread block per view: the same reduction as loss_finalize_kernel over
// that view's partials, so each view's loss equals its single-image loss.
__global__ void loss_finalize_batch_kernel(const SsimArgs *views, const int *boff) {
    const int v = blockIdx.x;
    const SsimArgs &a = views[v];
    loss_finalize_block(a.partials + boff[v], boff[v + 1] - boff[v], (double)a.W * a.H, a.loss);
}

int ssim_blocks(int W, int H) { return 3 * ((W + ST - 1) / ST) * ((H + ST - 1) / ST); }

static void ssim_set_smem_attr() {
    static const bool done = [] {
        cudaFuncSetAttribute(ssim_loss_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SsimSmem));
        cudaFuncSetAttribute(ssim_loss_batch_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(SsimSmem));
        return true;
    }();
    (void)done;
}

// views[v].partials must all be the same batch-wide array (indexed by global block).
void launch_ssim_loss_batch(const SsimArgs *d_views, const int *d_boff, int n_views, int *d_counter, cudaStream_t st) {
    if (n_views <= 0) return;
    ssim_set_smem_attr();
    static const int grid = [] {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ssim_loss_batch_kernel, SSIM_THREADS,
                                                      sizeof(SsimSmem));
        return sms * (per_sm > 0 ? per_sm : 1);
    }();
    cudaMemsetAsync(d_counter, 0, sizeof(int), st);
    ssim_loss_batch_kernel<<<grid, SSIM_THREADS, sizeof(SsimSmem), st>>>(d_views, d_boff, n_views, d_counter);
    loss_finalize_batch_kernel<<<n_views, 1024, 0, st>>>(d_views, d_boff);
}

void launch_ssim_loss(const SsimArgs &a, cudaStream_t st) {
    if (a.W <= 0 || a.H <= 0) return;
    const size_t smem = sizeof(SsimSmem);
    ssim_set_smem_attr();
    const int blocks = ssim_blocks(a.W, a.H);
    ssim_loss_kernel<<<blocks, SSIM_THREADS, smem, st>>>(a);
    loss_finalize_kernel<<<1, 1024, 0, st>>>(a.partials, blocks, (double)a.W * a.H, a.loss);
}

}  // namespace msplat
