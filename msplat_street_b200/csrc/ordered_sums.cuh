// Sums of many terms in double, in a prescribed order: the reference adds a row's terms
// one after another and then the rows, and results must equal its. The additions form
// one dependent chain per sum; what can be done side by side is everything before them.
// So a warp takes a row, its lanes load and widen a chunk of terms (consecutive lanes,
// consecutive terms) into shared memory while the previous chunk is being added, and
// one lane per sum adds the chunk in order.
#pragma once

#include <cuda_runtime.h>

namespace msplat {

constexpr int ORD_CHUNK = 128;             // terms staged at a time
constexpr int ORD_PITCH = ORD_CHUNK + 1;   // the adding lanes read different banks
constexpr int ORD_WARPS = 4;               // rows per block

struct Terms3 {
    double v[3];
};
struct Raw3 {
    float v[3];
};

// The three sums of terms widen(load(0)) .. widen(load(n - 1)), each in order; lane k < 3
// returns sum k, the other lanes 0. load only reads memory: its result is kept through
// the addition of the chunk before and widened after it, so that nothing waits for the
// loads. buf: 3 * ORD_PITCH doubles of shared memory of this warp. Every lane of the warp
// must call it with the same n.
template <typename Load, typename Widen>
__device__ __forceinline__ double warp_ordered_sums3(int n, Load load, Widen widen, double *buf) {
    constexpr int PER = ORD_CHUNK / 32;
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    decltype(load(0)) next[PER];
#pragma unroll
    for (int u = 0; u < PER; u++) {
        const int i = u * 32 + lane;
        if (i < n) next[u] = load(i);
    }
    for (int i0 = 0; i0 < n; i0 += ORD_CHUNK) {  // warp-uniform
        __syncwarp();
#pragma unroll
        for (int u = 0; u < PER; u++) {
            if (i0 + u * 32 + lane >= n) continue;
            const Terms3 t = widen(next[u]);
#pragma unroll
            for (int k = 0; k < 3; k++) buf[k * ORD_PITCH + u * 32 + lane] = t.v[k];
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = i0 + ORD_CHUNK + u * 32 + lane;
            if (i < n) next[u] = load(i);
        }
        if (lane < 3) {
            const double *b = buf + lane * ORD_PITCH;
            const int cnt = min(ORD_CHUNK, n - i0);
#pragma unroll 16
            for (int j = 0; j < cnt; j++) s += b[j];
        }
    }
    __syncwarp();
    return s;
}

// sums[3 y + k] for every row y of `rows` rows: ORD_WARPS rows a block.
template <typename RowLoad, typename Widen>
__device__ __forceinline__ void block_row_sums3(int rows, int n, RowLoad load, Widen widen, double *sums) {
    __shared__ double buf[ORD_WARPS][3 * ORD_PITCH];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, y = blockIdx.x * ORD_WARPS + warp;
    if (y >= rows) return;  // warp-uniform
    const double s = warp_ordered_sums3(n, [&](int i) { return load(y, i); }, widen, buf[warp]);
    if (lane < 3) sums[3 * (size_t)y + lane] = s;
}

}  // namespace msplat
