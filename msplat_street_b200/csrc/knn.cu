// Exact 3-nearest-neighbour mean distance and Gaussian initialisation.
//
// msplat_knn3_mean_dist (core/cpu/msplat_cpu.cpp:1498-1580 builds a k-d tree; the
// Metal backend sorts by Morton code and culls by box distance) returns, for every
// point, the mean distance to its 3 nearest OTHER points (fewer if n < 4, 1.0 if
// none). Here points are sorted by a 30-bit Morton code with the device radix sort and
// cut into boxes of 32 consecutive points, groups of 32 boxes and supergroups of 32
// groups, each with its bounds. One warp answers one box's 32 queries: it searches its
// own box, the rest of its own group, then every other group, descending from the
// supergroups; its lanes test 32 nodes of a level at a time against the query box's
// bounds, and a node survives only if its lower-bound squared distance is below the
// warp's worst third-best so far. A surviving box is tested once more by every query
// for itself before its 32 points are read. The lower bounds use the same float
// subtractions and squares as the point distances, and float rounding is monotonic, so
// a pruned node can hold no point that would enter a lane's best three: the result is
// exact, whatever the order of the search.
//
// msplat_init_gaussians (:1582-1605): isotropic log-scale log(max(d, 1e-7)), a
// uniformly random rotation from three PCG uniforms (Shoemake), DC colour from RGB
// and a constant opacity logit.
#include "common.cuh"
#include "kernels.h"

namespace msplat {

constexpr int KNN_BOX = 32;

__device__ __forceinline__ unsigned int ordered_bits(float f) {
    unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered(unsigned int u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

constexpr int KNN_BOUNDS_THREADS = 512;

// One atomic per block and bound: with one per warp, the 57 k atomics of a 400 k-point
// cloud on six addresses took 38 us.
__global__ void __launch_bounds__(KNN_BOUNDS_THREADS) knn_bounds_kernel(const float *pts, int n, unsigned int *bb) {
    __shared__ unsigned int part[6][KNN_BOUNDS_THREADS / 32];
    unsigned int mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        for (int a = 0; a < 3; a++) {
            const float v = pts[3 * (size_t)i + a];
            if (!isfinite(v)) continue;
            const unsigned int o = ordered_bits(v);
            mn[a] = min(mn[a], o);
            mx[a] = max(mx[a], o);
        }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const unsigned int lo = __reduce_min_sync(0xffffffffu, mn[a]), hi = __reduce_max_sync(0xffffffffu, mx[a]);
        if (lane == 0) {
            part[a][warp] = lo;
            part[3 + a][warp] = hi;
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const int a = threadIdx.x;
        unsigned int r = part[a][0];
        for (int w = 1; w < KNN_BOUNDS_THREADS / 32; w++) r = a < 3 ? min(r, part[a][w]) : max(r, part[a][w]);
        if (a < 3) atomicMin(&bb[a], r);
        else atomicMax(&bb[a], r);
    }
}

__device__ __forceinline__ uint32_t spread10(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__global__ void knn_morton_kernel(const float *pts, int n, const unsigned int *bb, uint32_t *keys, uint32_t *vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t q[3];
    for (int a = 0; a < 3; a++) {
        const float lo = from_ordered(bb[a]), hi = from_ordered(bb[3 + a]);
        const float ext = hi - lo;
        const float v = pts[3 * (size_t)i + a];
        float t = (isfinite(v) && ext > 0.f) ? (v - lo) / ext : 0.f;
        t = fminf(fmaxf(t, 0.f), 1.f);
        q[a] = (uint32_t)(t * 1023.f);
    }
    keys[i] = spread10(q[0]) | (spread10(q[1]) << 1) | (spread10(q[2]) << 2);
    vals[i] = (uint32_t)i;
}

__global__ void knn_gather_kernel(const float *pts, int n, const uint32_t *order, float4 *sp) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t i = order[j];
    sp[j] = make_float4(pts[3 * (size_t)i], pts[3 * (size_t)i + 1], pts[3 * (size_t)i + 2], __uint_as_float(i));
}

// Bounds over a warp's lanes, on every lane.
struct Bounds {
    float lo[3], hi[3];
};
__device__ __forceinline__ void warp_bounds(Bounds &b) {
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            b.lo[a] = fminf(b.lo[a], __shfl_xor_sync(0xffffffffu, b.lo[a], o));
            b.hi[a] = fmaxf(b.hi[a], __shfl_xor_sync(0xffffffffu, b.hi[a], o));
        }
}
__device__ __forceinline__ void store_bounds(float4 *mn, float4 *mx, int i, const Bounds &b) {
    mn[i] = make_float4(b.lo[0], b.lo[1], b.lo[2], 0.f);
    mx[i] = make_float4(b.hi[0], b.hi[1], b.hi[2], 0.f);
}

// One block per group: each warp takes one of its boxes, a lane per point, and warp 0
// the group's bounds from the warps'. Non-finite coordinates bound nothing.
__global__ void __launch_bounds__(KNN_BOX * KNN_BOX) knn_boxes_kernel(const float4 *sp, int n, int nboxes,
                                                                      float4 *bmin, float4 *bmax, float4 *gmin,
                                                                      float4 *gmax) {
    __shared__ Bounds s[KNN_BOX];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int box = blockIdx.x * KNN_BOX + warp, j = box * KNN_BOX + lane;
    Bounds b{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
    if (box < nboxes && j < n) {
        const float4 p = sp[j];
        const float c[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int a = 0; a < 3; a++)
            if (isfinite(c[a])) b.lo[a] = b.hi[a] = c[a];
    }
    warp_bounds(b);
    if (lane == 0) {
        if (box < nboxes) store_bounds(bmin, bmax, box, b);
        s[warp] = b;
    }
    __syncthreads();
    if (warp == 0) {
        b = s[lane];
        warp_bounds(b);
        if (lane == 0) store_bounds(gmin, gmax, blockIdx.x, b);
    }
}

// The supergroups' bounds, a warp each.
__global__ void knn_super_kernel(const float4 *gmin, const float4 *gmax, int ngroups, int nsuper, float4 *smin,
                                 float4 *smax) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= nsuper) return;  // warp-uniform
    const int g = i * KNN_BOX + lane;
    Bounds b{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
    if (g < ngroups) {
        const float4 lo = gmin[g], hi = gmax[g];
        b = Bounds{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}};
    }
    warp_bounds(b);
    if (lane == 0) store_bounds(smin, smax, i, b);
}

// best[0] <= best[1] <= best[2] (core/cpu/msplat_cpu.cpp:1522-1531); a NaN distance
// (a candidate with non-finite coordinates) is no neighbour
__device__ __forceinline__ void keep3(float d, float &b0, float &b1, float &b2) {
    if (!(d < b2)) return;
    if (d < b1) {
        b2 = b1;
        if (d < b0) {
            b1 = b0;
            b0 = d;
        } else {
            b1 = d;
        }
    } else {
        b2 = d;
    }
}

// Lower bound of the squared distance between a point of [qlo, qhi] and one of [lo, hi].
__device__ __forceinline__ float gap(float qlo, float qhi, float blo, float bhi) {
    return fmaxf(fmaxf(blo - qhi, qlo - bhi), 0.f);
}
__device__ __forceinline__ float gap2(const Bounds &q, const float4 lo, const float4 hi) {
    const float gx = gap(q.lo[0], q.hi[0], lo.x, hi.x), gy = gap(q.lo[1], q.hi[1], lo.y, hi.y),
                gz = gap(q.lo[2], q.hi[2], lo.z, hi.z);
    return gx * gx + gy * gy + gz * gz;
}

// A warp's search state: its 32 queries (one per lane) and their three best distances.
struct KnnSearch {
    const float4 *sp;
    float4 *pts;  // shared memory of this warp: the points of the box being scanned
    int n;
    float4 q;
    uint32_t self;
    bool fin;      // this lane has a query with finite coordinates
    Bounds qb;     // bounds of the warp's finite queries
    float b0, b1, b2;
    unsigned boxes;  // boxes whose points were read

    // the warp's largest third-best: no node at or beyond it matters
    __device__ __forceinline__ float threshold() const {
        return from_ordered(__reduce_max_sync(0xffffffffu, ordered_bits(fin ? b2 : -INFINITY)));
    }
    // whether node i (< count) may hold a neighbour of one of the warp's queries
    __device__ __forceinline__ bool near(const float4 *mn, const float4 *mx, int i, int count, float thr) const {
        if (i >= count) return false;
        const float4 lo = mn[i], hi = mx[i];
        return lo.x <= hi.x && gap2(qb, lo, hi) < thr;
    }
    // the lane's point of box c (none: a distance that is no number)
    __device__ __forceinline__ float4 load_box(int c) const {
        const int j = c * KNN_BOX + (threadIdx.x & 31);
        return j < n ? sp[j] : make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
    }
    // a box's points, a lane's each, against every query
    __device__ __forceinline__ void scan_box(const float4 mine) {
        boxes++;
        __syncwarp();  // the box before is read
        pts[threadIdx.x & 31] = mine;
        __syncwarp();
#pragma unroll 8
        for (int k = 0; k < KNN_BOX; k++) {
            const float4 p = pts[k];
            const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
            const float d = dx * dx + dy * dy + dz * dz;
            if (d < b2 && fin && __float_as_uint(p.w) != self) keep3(d, b0, b1, b2);
        }
    }
    // the 32 boxes of group g, except box `skip`
    __device__ __forceinline__ void scan_group(int g, int skip, const float4 *bmin, const float4 *bmax, int nboxes) {
        const int lane = threadIdx.x & 31, c = g * KNN_BOX + lane;
        const float thr = threshold();  // every lane takes part
        unsigned m = __ballot_sync(0xffffffffu, c != skip && near(bmin, bmax, c, nboxes, thr));
        while (m) {  // warp-uniform
            const int cb = g * KNN_BOX + __ffs(m) - 1;
            m &= m - 1;
            const float4 lo = bmin[cb], hi = bmax[cb];
            const Bounds me{{q.x, q.y, q.z}, {q.x, q.y, q.z}};
            if (__ballot_sync(0xffffffffu, fin && gap2(me, lo, hi) < b2)) scan_box(load_box(cb));
        }
    }
};

// evals (may be null): adds the point distances the warp computes (32 per query per
// box it reads) -- the search's work, for throughput reports.
//
// Bound by instruction issue: about 12 instructions a point of a box that is read. A
// 400 k-point cloud: 4.34 -> 0.39 ms against the form in which every warp tested all
// 12.5 k boxes, 32 at a time, and read all that passed the first test; the descent
// through groups and supergroups leaves a few dozen node tests a warp. A box comes in one
// load, a point a lane, and is read from shared memory: with a load a point, the same on
// every lane, each box cost four cache misses one after another (0.56 ms; one outlier far
// from 20 k points, which puts them all into one Morton cell, 2.46 against 1.01, and 1.41
// in the form before). Loading the next box ahead reads many that the second test drops:
// 0.58.
__global__ void __launch_bounds__(128) knn_query_kernel(const float4 *sp, int n, int nboxes, const float4 *bmin,
                                                        const float4 *bmax, int ngroups, const float4 *gmin,
                                                        const float4 *gmax, int nsuper, const float4 *smin,
                                                        const float4 *smax, float *out, unsigned long long *evals) {
    const int lane = threadIdx.x & 31;
    const int own = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
    if (own >= nboxes) return;  // warp-uniform
    const int j = own * KNN_BOX + lane;
    const bool valid = j < n;
    KnnSearch s;
    __shared__ float4 pts[128 / 32][KNN_BOX];
    s.sp = sp;
    s.pts = pts[threadIdx.x >> 5];
    s.n = n;
    s.q = valid ? sp[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    s.self = __float_as_uint(s.q.w);
    s.fin = valid && isfinite(s.q.x) && isfinite(s.q.y) && isfinite(s.q.z);
    const float c[3] = {s.q.x, s.q.y, s.q.z};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        s.qb.lo[a] = s.fin ? c[a] : INFINITY;
        s.qb.hi[a] = s.fin ? c[a] : -INFINITY;
    }
    warp_bounds(s.qb);
    s.b0 = s.b1 = s.b2 = INFINITY;
    s.boxes = 0;
    const unsigned nq = __popc(__ballot_sync(0xffffffffu, s.fin));
    if (nq) {  // warp-uniform
        const int og = own / KNN_BOX, os = og / KNN_BOX;
        s.scan_box(s.load_box(own));
        s.scan_group(og, own, bmin, bmax, nboxes);
        // supergroup 0 of the walk is the warp's own, then the others in order
        for (int i0 = 0; i0 < nsuper; i0 += 32) {
            const int i = i0 + lane, sg = i == 0 ? os : (i <= os ? i - 1 : i);
            const float thr = s.threshold();
            unsigned ms = __ballot_sync(0xffffffffu, i < nsuper && s.near(smin, smax, sg, nsuper, thr));
            while (ms) {
                const int sgi = __shfl_sync(0xffffffffu, sg, __ffs(ms) - 1);
                ms &= ms - 1;
                const int g = sgi * KNN_BOX + lane;
                const float thrg = s.threshold();
                unsigned mg = __ballot_sync(0xffffffffu, g != og && s.near(gmin, gmax, g, ngroups, thrg));
                while (mg) {
                    const int gi = sgi * KNN_BOX + __ffs(mg) - 1;
                    mg &= mg - 1;
                    s.scan_group(gi, -1, bmin, bmax, nboxes);
                }
            }
        }
        if (evals && lane == 0) atomicAdd(evals, (unsigned long long)s.boxes * nq * KNN_BOX);
    }
    if (!valid) return;
    float sum = 0.f, cnt = 0.f;
    if (isfinite(s.b0)) { sum += sqrtf(s.b0); cnt += 1.f; }
    if (isfinite(s.b1)) { sum += sqrtf(s.b1); cnt += 1.f; }
    if (isfinite(s.b2)) { sum += sqrtf(s.b2); cnt += 1.f; }
    out[s.self] = cnt > 0.f ? sum / cnt : 1.f;
}

int knn_boxes(int n) { return (n + KNN_BOX - 1) / KNN_BOX; }
int knn_nodes(int n) {
    const int nb = knn_boxes(n), ng = knn_boxes(nb);
    return nb + ng + knn_boxes(ng);
}

int launch_knn3(const float *pts, int n, float *out, KnnScratch &s, cudaStream_t st) {
    if (n <= 0) return 0;
    const unsigned int init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
    cudaMemcpyAsync(s.bounds, init, sizeof init, cudaMemcpyHostToDevice, st);
    if (s.evals) cudaMemsetAsync(s.evals, 0, sizeof(unsigned long long), st);
    knn_bounds_kernel<<<std::min((n + KNN_BOUNDS_THREADS - 1) / KNN_BOUNDS_THREADS, 2 * 148), KNN_BOUNDS_THREADS, 0,
                        st>>>(pts, n, s.bounds);
    knn_morton_kernel<<<(n + 255) / 256, 256, 0, st>>>(pts, n, s.bounds, s.keys[0], s.vals[0]);
    const int cur = radix_sort_pairs32(s.keys, s.vals, n, 30, s.radix_scratch, st);
    knn_gather_kernel<<<(n + 255) / 256, 256, 0, st>>>(pts, n, s.vals[cur], s.sorted);
    const int nb = knn_boxes(n), ng = knn_boxes(nb), ns = knn_boxes(ng);
    float4 *gmin = s.bmin + nb, *gmax = s.bmax + nb, *smin = gmin + ng, *smax = gmax + ng;
    knn_boxes_kernel<<<ng, KNN_BOX * KNN_BOX, 0, st>>>(s.sorted, n, nb, s.bmin, s.bmax, gmin, gmax);
    knn_super_kernel<<<(ns + 7) / 8, 256, 0, st>>>(gmin, gmax, ng, ns, smin, smax);
    knn_query_kernel<<<(int)(((int64_t)nb * 32 + 127) / 128), 128, 0, st>>>(
        s.sorted, n, nb, s.bmin, s.bmax, ng, gmin, gmax, ns, smin, smax, out, s.evals);
    return 0;
}

__global__ void init_gaussians_kernel(const float *md, const uint8_t *rgb, int n, uint32_t seed, float logit,
                                      float *scales, float *quats, float *dc, float *opac) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float ls = (float)log((double)fmaxf(md[i], 1e-7f));
    scales[3 * i] = scales[3 * i + 1] = scales[3 * i + 2] = ls;
    const uint32_t c = 3u * (uint32_t)i;
    const float u = rand_unif(seed, c), v = rand_unif(seed, c + 1u), w = rand_unif(seed, c + 2u);
    const float tau = 6.28318530717958647692f;
    const float a = sqrtf(1.f - u), b = sqrtf(u);
    const float tv = tau * v, tw = tau * w;
    quats[4 * i + 0] = a * (float)sin((double)tv);
    quats[4 * i + 1] = a * (float)cos((double)tv);
    quats[4 * i + 2] = b * (float)sin((double)tw);
    quats[4 * i + 3] = b * (float)cos((double)tw);
    for (int k = 0; k < 3; k++) dc[3 * i + k] = ((float)rgb[3 * i + k] * (1.f / 255.f) - 0.5f) / SH_C0;
    opac[i] = logit;
}

void launch_init_gaussians(const float *md, const uint8_t *rgb, int n, uint32_t seed, float logit, float *scales,
                           float *quats, float *dc, float *opac, cudaStream_t st) {
    if (n <= 0) return;
    init_gaussians_kernel<<<(n + 255) / 256, 256, 0, st>>>(md, rgb, n, seed, logit, scales, quats, dc, opac);
}

}  // namespace msplat
