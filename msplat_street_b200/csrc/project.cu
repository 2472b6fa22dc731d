// Projection with EWA 2D covariance and SH colour, one thread per Gaussian.
//
// Follows project_and_sh (core/cpu/msplat_cpu.cpp:452-500) and its helpers
// (:63-190). The output per visible Gaussian is one 48-byte Splat record (read by
// both rasterizer passes), its depth, radius, pixel AABB half-extent and the number
// of 16x16 tiles its AABB covers (what the binning deals out). Compiled with
// -fmad=false: tile rectangles and depth keys must equal the reference's bit for bit.
#include <algorithm>

#include "project_impl.cuh"

namespace msplat {

constexpr int PROJ_THREADS = 128;

// Key and value of the depth order at output slot o.
__device__ __forceinline__ void depth_key(const ProjectArgs &a, int o, bool kept, float depth) {
    a.depth_keys[o] = kept ? __float_as_uint(depth) : 0xffffffffu;
    a.depth_vals[o] = (uint32_t)o;
}

// With SH degree 3 in use the warp stages its SH-rest rows while the geometry runs
// (issue_rest_rows); no lane leaves before the wait that every lane of the warp takes.
// Bound by the 236 bytes a Gaussian reads and by double-precision issue: the general
// exp gave way to the table exponential, three of the skip extents' four divisions to one
// reciprocal, and 45 four-byte copies a lane to 12 of 16 bytes. 12 million Gaussians over
// eight views 826 -> 775 us.
__global__ void __launch_bounds__(PROJ_THREADS) project_kernel(ProjectArgs a) {
    __shared__ __align__(16) float rest_buf[PROJ_THREADS / 32][32 * PROJ_REST3];
    __shared__ double exp_t[EXP_TABLE];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < a.n;
    float *buf = rest_buf[threadIdx.x >> 5];
    bool staged = false;
    if (a.rest_stride == PROJ_REST3 && a.cam.degrees_to_use >= 3)  // grid-uniform
        staged = issue_rest_rows(a.features_rest + (size_t)PROJ_REST3 * (valid ? i : 0), valid, buf);
    exp_span_init_a(exp_t);
    __syncthreads();
    ProjState st;
    const bool kept = valid && project_geom(a, i, i, exp_t, st);
    if (valid) depth_key(a, i, kept, st.depth);
    if (staged) rest_rows_wait();
    if (kept) project_finish(a, i, i, st, staged ? buf + PROJ_REST3 * (threadIdx.x & 31) : nullptr);
}

void launch_project(const ProjectArgs &a, cudaStream_t st) {
    if (a.n <= 0) return;
    project_kernel<<<(a.n + PROJ_THREADS - 1) / PROJ_THREADS, PROJ_THREADS, 0, st>>>(a);
}

// Every (view, Gaussian) instance of a batch: the same per-Gaussian code, reading the
// view's scene and camera and writing at the instance's global slot.
__global__ void __launch_bounds__(PROJ_THREADS) project_batch_kernel(const BatchDesc d, int total) {
    __shared__ __align__(16) float rest_buf[PROJ_THREADS / 32][32 * PROJ_REST3];
    __shared__ double exp_t[EXP_TABLE];
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = g < total;
    const int v = valid ? find_view(d.inst_off, d.n_views, g) : 0;
    const int i = valid ? g - d.inst_off[v] : 0;
    float *buf = rest_buf[threadIdx.x >> 5];
    // lanes of one warp may belong to different views: the rows must be back to back
    const bool deg3 = valid && d.proj[v].rest_stride == PROJ_REST3 && d.proj[v].cam.degrees_to_use >= 3;
    const bool staged =
        issue_rest_rows(deg3 ? d.proj[v].features_rest + (size_t)PROJ_REST3 * i : nullptr, deg3, buf);
    exp_span_init_a(exp_t);
    __syncthreads();
    ProjState st;
    const bool kept = valid && project_geom(d.proj[v], i, g, exp_t, st);
    if (valid) depth_key(d.proj[v], g, kept, st.depth);
    if (staged) rest_rows_wait();
    if (kept) project_finish(d.proj[v], i, g, st, staged ? buf + PROJ_REST3 * (threadIdx.x & 31) : nullptr);
}

void launch_project_batch(const BatchDesc &d, int total, cudaStream_t st) {
    if (total <= 0) return;
    project_batch_kernel<<<(total + PROJ_THREADS - 1) / PROJ_THREADS, PROJ_THREADS, 0, st>>>(d, total);
}

// The scales' and opacities' exponential over n inputs (test hook).
__global__ void exp_wide_kernel(const float *x, int64_t n, float *out) {
    __shared__ double t[EXP_TABLE];
    exp_span_init_a(t);
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = exp_wide(x[i], t);
}

void launch_exp_wide(const float *x, int64_t n, float *out, cudaStream_t st) {
    if (n <= 0) return;
    exp_wide_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, st>>>(x, n, out);
}

}  // namespace msplat
