// Densification: classify, split, duplicate, cull and stream compaction; opacity reset.
//
// Follows msplat_densify (core/cpu/msplat_cpu.cpp:1330-1465) step by step:
//  1. classify (:1354-1369): a Gaussian seen in at least one view with mean screen
//     gradient (gn / vc) * half_max_dim above the threshold is split when its largest
//     scale exceeds size_thresh (or its screen size split_screen_size), and cloned
//     when it is small;
//  2. ordinals by exclusive scans (the reference counts serially, :1370-1375);
//  3. split children at N + 2*ord + k, offset by a parent-rotated N(0, s) sample
//     from the PCG/Box-Muller counter RNG, scales minus log(1.6); the parent's scales
//     shrink too (:1387-1415); then clones at N + 2*n_split + ord (:1417-1430), after
//     every split (a Gaussian may be both, and the clone copies the shrunk parent).
//     These per-parent kernels write only positions and scales and record each new
//     row's parent; one row-parallel pass per parameter group then copies the
//     quaternion, colour and opacity rows and zeroes the moments, coalesced;
//  4. cull (:1432-1448) over the N_new rows and order-preserving compaction of all 18
//     buffers (6 parameters, 6 first moments, 6 second moments) through a scratch
//     buffer (:1449-1464): the 15 narrow ones together, then the SH rest and its moments
//     one at a time.
// A Gaussian can be both split (large on screen) and cloned (small in the world), so
// the rows after step 3 number up to 4N, not 3N as the reference's capacity check
// assumes (its CPU port would then write past its buffers). Here every kernel from
// step 3 on first checks N + 2 splits + clones against the capacity; when it does not
// fit, nothing is written and the overflow flag is set (the host reports it).
// Child and clone moments are zeroed. Counts live on the device; the host reads the
// final count once (the reference's Metal backend also syncs there,
// core/metal/msplat_metal.mm:1998-2001).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace msplat {

__global__ void densify_classify_kernel(DensifyArgs a, int32_t *split, int32_t *dup) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    int s = 0, d = 0;
    const float vc = a.vis_counts[i];
    if (vc > 0.0f) {
        const bool high = (a.grad_norm[i] / vc) * a.half_max_dim > a.grad_thresh;
        const float *sc = a.buf[1] + 3 * (size_t)i;
        const float mx = fmaxf(fmaxf(exp_ref(sc[0]), exp_ref(sc[1])), exp_ref(sc[2]));
        const bool large = mx > a.size_thresh;
        bool sp = large;
        if (a.check_screen && a.max_2d[i] > a.screen_thresh) sp = true;
        s = (sp && high) ? 1 : 0;
        d = (!large && high) ? 1 : 0;
    }
    split[i] = s;
    dup[i] = d;
}

// Box-Muller on the PCG counter RNG (core/cpu/msplat_cpu.cpp:315-323)
__device__ __forceinline__ V3 rand_normal3(uint32_t seed, uint32_t stream) {
    const uint32_t c = stream * 4u;
    const float u0 = rand_unif(seed, c), u1 = rand_unif(seed, c + 1u);
    const float u2 = rand_unif(seed, c + 2u), u3 = rand_unif(seed, c + 3u);
    const float r0 = sqrtf(-2.0f * (float)log((double)u0)), r1 = sqrtf(-2.0f * (float)log((double)u2));
    const float tau = 6.28318530717958647692f;
    const float t0 = tau * u1, t1 = tau * u3;
    return V3{r0 * (float)cos((double)t0), r0 * (float)sin((double)t0), r1 * (float)cos((double)t1)};
}

// rows after splits and clones, and whether they fit the buffers
__device__ __forceinline__ bool rows_fit(const DensifyArgs &a, const int32_t *n_split, const int32_t *n_dup,
                                         int64_t &total) {
    total = (int64_t)a.n + 2 * (int64_t)(*n_split) + *n_dup;
    return total <= a.cap;
}

__global__ void densify_split_kernel(DensifyArgs a, const int32_t *split, const int32_t *split_ord,
                                     const int32_t *n_split, const int32_t *n_dup, int32_t *overflow,
                                     int32_t *row_parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int64_t total;
    if (!rows_fit(a, n_split, n_dup, total)) {
        if (i == 0) *overflow = 1;
        return;
    }
    if (i >= a.n || !split[i]) return;
    const int ord = split_ord[i];
    float *means = a.buf[0], *scales = a.buf[1];
    const float *q = a.buf[2] + 4 * (size_t)i;
    float qw = q[0], qx = q[1], qy = q[2], qz = q[3];
    const float ql = sqrtf(qw * qw + qx * qx + qy * qy + qz * qz);
    qw /= ql;
    qx /= ql;
    qy /= ql;
    qz /= ql;
    const float sx = exp_ref(scales[3 * i]), sy = exp_ref(scales[3 * i + 1]), sz = exp_ref(scales[3 * i + 2]);
    for (int k = 0; k < 2; k++) {
        const int64_t c = (int64_t)a.n + 2 * ord + k;
        const V3 nr = rand_normal3(a.seed, (uint32_t)(ord * 2 + k));
        const float r0 = nr.x * sx, r1 = nr.y * sy, r2 = nr.z * sz;
        const float v0 = (1.f - 2.f * (qy * qy + qz * qz)) * r0 + 2.f * (qx * qy - qw * qz) * r1 +
                         2.f * (qx * qz + qw * qy) * r2;
        const float v1 = 2.f * (qx * qy + qw * qz) * r0 + (1.f - 2.f * (qx * qx + qz * qz)) * r1 +
                         2.f * (qy * qz - qw * qx) * r2;
        const float v2 = 2.f * (qx * qz - qw * qy) * r0 + 2.f * (qy * qz + qw * qx) * r1 +
                         (1.f - 2.f * (qx * qx + qy * qy)) * r2;
        means[3 * c] = means[3 * i] + v0;
        means[3 * c + 1] = means[3 * i + 1] + v1;
        means[3 * c + 2] = means[3 * i + 2] + v2;
        for (int j = 0; j < 3; j++) scales[3 * c + j] = scales[3 * i + j] - a.log_size_fac;
        row_parent[2 * ord + k] = i;  // the other groups are copied row-parallel (densify_rows_kernel)
    }
    for (int j = 0; j < 3; j++) scales[3 * i + j] -= a.log_size_fac;
}

__global__ void densify_dup_kernel(DensifyArgs a, const int32_t *dup, const int32_t *dup_ord, const int32_t *n_split,
                                   const int32_t *n_dup, int32_t *row_parent) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int64_t total;
    if (!rows_fit(a, n_split, n_dup, total)) return;
    if (i >= a.n || !dup[i]) return;
    const int64_t r = 2 * (int64_t)(*n_split) + dup_ord[i];  // new-row index; row a.n + r
    const int64_t d = (int64_t)a.n + r;
    for (int j = 0; j < 3; j++) a.buf[0][3 * d + j] = a.buf[0][3 * i + j];
    for (int j = 0; j < 3; j++) a.buf[1][3 * d + j] = a.buf[1][3 * i + j];  // a split parent's shrunk scales
    row_parent[r] = i;
}

// The new rows a.n .. total - 1 (split children, then clones): quaternion, DC, SH rest
// and opacity copied from the row's parent, every moment zeroed. blockIdx.y: the group;
// a block takes ROWS new rows at a time as one flat range, consecutive threads
// consecutive floats, with the rows' parents in shared memory. 84 -> 41 us for 137 k new
// rows, against one launch a group with a 64-bit division a float.
constexpr int ROWS = 256, ROW_THREADS = 256;

__global__ void __launch_bounds__(ROW_THREADS) densify_rows_kernel(DensifyArgs a, const int32_t *n_split,
                                                                   const int32_t *n_dup, const int32_t *row_parent) {
    __shared__ int32_t parent[ROWS];
    int64_t total;
    if (!rows_fit(a, n_split, n_dup, total)) return;
    const int g = blockIdx.y, st = a.stride[g];
    if (st <= 0) return;
    const int64_t rows = total - a.n;
    for (int64_t r0 = (int64_t)blockIdx.x * ROWS; r0 < rows; r0 += (int64_t)gridDim.x * ROWS) {  // block-uniform
        const int here = (int)min((int64_t)ROWS, rows - r0);
        __syncthreads();
        for (int i = threadIdx.x; i < here; i += ROW_THREADS) parent[i] = row_parent[r0 + i];
        __syncthreads();
        const int64_t dst = ((int64_t)a.n + r0) * st;
        for (int j = threadIdx.x; j < here * st; j += ROW_THREADS) {
            const int row = j / st;
            if (g >= 2) a.buf[g][dst + j] = a.buf[g][(int64_t)parent[row] * st + j - row * st];
            a.m1[g][dst + j] = 0.f;
            a.m2[g][dst + j] = 0.f;
        }
    }
}

__global__ void densify_cull_kernel(DensifyArgs a, const int32_t *split, const int32_t *n_split,
                                    const int32_t *n_dup, int32_t *keep, int32_t *n_new) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t total;
    const bool fit = rows_fit(a, n_split, n_dup, total);
    if (i == 0) *n_new = fit ? (int32_t)total : 0;  // no rows to compact when they did not fit
    if (i >= 4 * (int64_t)a.n) return;
    if (!fit || i >= total) {
        keep[i] = 0;
        return;
    }
    const float o = 1.0f / (1.0f + exp_ref(-a.buf[5][i]));
    bool cull = o < a.cull_alpha;
    if (i < a.n && split[i]) cull = true;
    if (a.check_huge) {
        const float *sc = a.buf[1] + 3 * i;
        const float mx = fmaxf(fmaxf(exp_ref(sc[0]), exp_ref(sc[1])), exp_ref(sc[2]));
        if (mx > a.cull_scale) cull = true;
        if (a.check_screen && i < a.n && a.max_2d[i] > a.cull_screen) cull = true;
    }
    keep[i] = cull ? 0 : 1;
}

// Compaction of several buffers at once (blockIdx.y): kept rows to scratch at their
// ordinal, then back. A block takes ROWS source rows as one flat range, four floats a
// thread and load, with the rows' destinations in shared memory; the rows kept lie side
// by side in the scratch, so the stores of neighbouring threads do too. The copy back
// moves float4s when both arrays are 16-byte aligned. 300 k Gaussians at SH degree 3 (437 k
// rows before, 357 k after): gather 343 -> 207 us and copy 152 -> 112 us against one
// thread a float with a 64-bit division and two look-ups each, a launch pair per buffer.
constexpr int MAX_COMPACT = 15;
struct CompactArgs {
    float *buf[MAX_COMPACT];
    int64_t at[MAX_COMPACT];  // its place in the scratch, floats
    int stride[MAX_COMPACT];
};

__global__ void __launch_bounds__(ROW_THREADS) compact_gather_kernel(const CompactArgs c, float *scratch,
                                                                     const int32_t *keep, const int32_t *keep_ord,
                                                                     const int32_t *n_new) {
    __shared__ int32_t to[ROWS];
    const int64_t rows = *n_new;
    const int st = c.stride[blockIdx.y];
    const float *src = c.buf[blockIdx.y];
    float *dst = scratch + c.at[blockIdx.y];
    const bool vec4 = (reinterpret_cast<uintptr_t>(src) & 15) == 0;  // a block's first float is a multiple of 256
    for (int64_t r0 = (int64_t)blockIdx.x * ROWS; r0 < rows; r0 += (int64_t)gridDim.x * ROWS) {  // block-uniform
        const int here = (int)min((int64_t)ROWS, rows - r0);
        __syncthreads();
        for (int i = threadIdx.x; i < here; i += ROW_THREADS) to[i] = keep[r0 + i] ? keep_ord[r0 + i] : -1;
        __syncthreads();
        const float *from = src + r0 * st;
        const int floats = here * st, n4 = vec4 ? floats / 4 : 0;
        constexpr int AHEAD = 4;  // loads before the first store
        for (int q0 = threadIdx.x; q0 < n4; q0 += AHEAD * ROW_THREADS) {
            float4 v[AHEAD];
#pragma unroll
            for (int h = 0; h < AHEAD; h++) {
                const int q = q0 + h * ROW_THREADS;
                if (q < n4) v[h] = reinterpret_cast<const float4 *>(from)[q];
            }
#pragma unroll
            for (int h = 0; h < AHEAD; h++) {
                const int q = q0 + h * ROW_THREADS;
                if (q >= n4) break;
                const float f[4] = {v[h].x, v[h].y, v[h].z, v[h].w};
                int row = 4 * q / st, col = 4 * q - row * st;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int o = to[row];
                    if (o >= 0) dst[(int64_t)o * st + col] = f[u];
                    if (++col == st) {
                        col = 0;
                        if (++row == here) break;  // past the last float
                    }
                }
            }
        }
        for (int j = 4 * n4 + threadIdx.x; j < floats; j += ROW_THREADS) {
            const int row = j / st, o = to[row];
            if (o >= 0) dst[(int64_t)o * st + j - row * st] = from[j];
        }
    }
}

__global__ void compact_copy_back_kernel(const CompactArgs c, const float *scratch, const int32_t *new_count,
                                         const int32_t *overflow) {
    if (*overflow) return;
    float *dst = c.buf[blockIdx.y];
    const float *src = scratch + c.at[blockIdx.y];
    const int64_t elems = (int64_t)(*new_count) * c.stride[blockIdx.y];
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool vec4 = ((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15) == 0;
    const int64_t n4 = vec4 ? elems / 4 : 0;
    float4 *d4 = reinterpret_cast<float4 *>(dst);
    const float4 *s4 = reinterpret_cast<const float4 *>(src);
    for (int64_t t = t0; t < n4; t += step) d4[t] = s4[t];
    for (int64_t t = 4 * n4 + t0; t < elems; t += step) dst[t] = src[t];
}

__global__ void opacity_reset_kernel(float *o, float *m1, float *m2, int n, float reset_logit) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    o[i] = fminf(o[i], reset_logit);
    m1[i] = 0.f;
    m2[i] = 0.f;
}

// A buffer's place in the scratch: each starts on 16 bytes.
static int64_t align4(int64_t floats) { return (floats + 3) / 4 * 4; }

// Room for the widest buffer's rows, as compacting one buffer at a time needs, and for
// all 15 narrow ones at once (a launch pair instead of 15) where those take no more than
// NARROW_FLOATS: at SH degree 3 the two are the same size, at degree 0 ten times apart,
// and a large model's buffers are long enough to be compacted a few at a time. 2 M
// Gaussians at degree 0: 874 us with 512 MB, 831 with the 1.3 GB of all at once, 943 with
// 256 MB.
constexpr int64_t NARROW_FLOATS = 1 << 27;  // 512 MB
int64_t densify_scratch_floats(int64_t rows, int max_stride) {
    const int64_t narrow = 3 * (3 * align4(3 * rows) + align4(4 * rows) + align4(rows));
    return std::max(align4(rows * max_stride), std::min(narrow, NARROW_FLOATS));
}

void launch_densify(const DensifyArgs &a, DensifyScratch &s, cudaStream_t st) {
    const int n = a.n;
    if (n <= 0) {
        cudaMemsetAsync(s.new_count, 0, sizeof(int32_t), st);
        return;
    }
    const int bs = 256;
    const int gb = (n + bs - 1) / bs;
    densify_classify_kernel<<<gb, bs, 0, st>>>(a, s.split, s.dup);
    scan_exclusive<int32_t>(s.split, s.split_ord, n, s.n_split, s.scan_part, st);
    scan_exclusive<int32_t>(s.dup, s.dup_ord, n, s.n_dup, s.scan_part, st);
    cudaMemsetAsync(s.overflow, 0, sizeof(int32_t), st);
    densify_split_kernel<<<gb, bs, 0, st>>>(a, s.split, s.split_ord, s.n_split, s.n_dup, s.overflow, s.row_parent);
    densify_dup_kernel<<<gb, bs, 0, st>>>(a, s.dup, s.dup_ord, s.n_split, s.n_dup, s.row_parent);
    const int64_t rows = 4 * (int64_t)n;  // at most N + 2 N splits + N clones
    const unsigned row_blocks = (unsigned)std::min<int64_t>((rows + ROWS - 1) / ROWS, 148 * 16);
    densify_rows_kernel<<<dim3(row_blocks, 6), ROW_THREADS, 0, st>>>(a, s.n_split, s.n_dup, s.row_parent);
    densify_cull_kernel<<<(unsigned)((rows + bs - 1) / bs), bs, 0, st>>>(a, s.split, s.n_split, s.n_dup, s.keep,
                                                                       s.n_new);
    scan_exclusive<int32_t>(s.keep, s.keep_ord, (int)rows, s.new_count, s.scan_part, st);
    // the narrow groups' 15 buffers side by side in the scratch, as many at a time as it
    // holds, then each SH-rest buffer
    CompactArgs c;
    int k = 0;
    int64_t at = 0;
    auto flush = [&] {
        if (k > 0) {
            compact_gather_kernel<<<dim3(row_blocks, (unsigned)k), ROW_THREADS, 0, st>>>(c, s.scratch, s.keep,
                                                                                         s.keep_ord, s.n_new);
            compact_copy_back_kernel<<<dim3(148 * 4, (unsigned)k), bs, 0, st>>>(c, s.scratch, s.new_count, s.overflow);
        }
        k = 0;
        at = 0;
    };
    auto add = [&](float *buf, int stride) {
        if (stride <= 0) return;  // e.g. no SH rest at degree 0
        const int64_t size = align4(rows * stride);
        if (at + size > s.scratch_floats) flush();
        c.buf[k] = buf;
        c.at[k] = at;
        c.stride[k++] = stride;
        at += size;
    };
    for (int g = 0; g < 6; g++) {
        if (g == 4) continue;
        for (float *buf : {a.buf[g], a.m1[g], a.m2[g]}) add(buf, a.stride[g]);
    }
    flush();
    for (float *buf : {a.buf[4], a.m1[4], a.m2[4]}) {
        add(buf, a.stride[4]);
        flush();
    }
}

void launch_opacity_reset(float *o, float *m1, float *m2, int n, float reset_logit, cudaStream_t st) {
    if (n <= 0) return;
    opacity_reset_kernel<<<(n + 255) / 256, 256, 0, st>>>(o, m1, m2, n, reset_logit);
}

}  // namespace msplat
