// Tile binning: every tile's list of Gaussians in (depth, index) order.
//
// The reference emits one (tile, depth) key per intersection and sorts them
// (bin_and_sort, core/cpu/msplat_cpu.cpp:505-567). Here only the Gaussians are sorted,
// by depth (stable, ties in index order); what is left is to deal each one to its tiles
// in that order, which needs no sort of the intersections:
//  1. count: the depth order is cut into chunks of about equal numbers of intersections,
//     and each chunk counts its entries per tile in shared memory;
//  2. scan: per tile, the chunks' counts become prefixes, and the tiles' totals their
//     list starts (so a chunk's first entry of a tile has a known place in the list);
//  3. emit: each chunk walks its Gaussians in order and writes their ids to those
//     places, advancing one shared-memory cursor per tile.
// Every list is then exactly the reference's, whatever the chunks. The radix sort of
// (tile, Gaussian) pairs this replaces moved 12 bytes a pair to emit them and 20 more a
// pass; the lists are written once, 4 bytes an entry (8 with the backward's map).
//
// In a batch the instances' depth order is view-major, a chunk belongs to one view, and
// tiles are numbered over all views.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace msplat {

// Tiles whose counters a block holds: a window of the image's tile grid. 16 KB of counts,
// 32 KB with the emission's masks, so that six blocks fit an SM; a 1080p frame (8160
// tiles) is two windows, which different blocks take.
constexpr int BIN_MAX_TILES = 4096;
constexpr int BIN_THREADS = 256, BIN_WARPS = BIN_THREADS / 32;
// Rectangles of up to this many tiles (within the window, or a warp's band of it) are
// one lane's; larger ones the warp's.
constexpr int BIN_LANE_MAX = 64;
// A view is cut into as many chunks as give each this many intersections, up to its
// share of the launch's blocks.
constexpr int BIN_MIN_ENTRIES = 1024;

struct BinWindow {
    int x0, y0, x1, y1, w;  // tiles [x0, x1) x [y0, y1); w: counters per row
};
struct BinView {
    int n0, n1;  // positions in the depth order
    int chunks;  // chunks in use
    int64_t first, entries;
    int tiles_x, tiles_y, tile0;
    int64_t counts;  // its first chunk's row of per-tile counts
};
struct BinChunk {
    int k, first, last;         // index within the view, depth-order positions
    int wins_x, wins;           // windows across, and in all
    int win_w, win_h;
    int64_t counts;
};

template <bool BATCH>
__device__ __forceinline__ void bin_grid(const BinArgs &a, int v, BinView &b) {
    b.tiles_x = BATCH ? a.d.tiles_x[v] : a.tiles_x;
    b.tiles_y = BATCH ? a.d.tiles_y[v] : a.tiles_y;
    b.tile0 = BATCH ? a.d.tile_off[v] : 0;
    b.counts = BATCH ? a.d.count_off[v] : 0;
}

template <bool BATCH>
__device__ __forceinline__ BinView bin_view(const BinArgs &a, int v) {
    BinView b;
    bin_grid<BATCH>(a, v, b);
    b.n0 = BATCH ? a.d.inst_off[v] : 0;
    b.n1 = BATCH ? a.d.inst_off[v + 1] : a.n;
    const int slots = BATCH ? a.d.chunk_off[v + 1] - a.d.chunk_off[v] : a.chunks;
    const int64_t total = *a.total;
    b.first = b.n0 < a.n ? a.offsets_sorted[b.n0] : total;
    b.entries = (b.n1 < a.n ? a.offsets_sorted[b.n1] : total) - b.first;
    b.chunks = (int)min((int64_t)slots, (b.entries + BIN_MIN_ENTRIES - 1) / BIN_MIN_ENTRIES);
    return b;
}

// First position r of [lo, hi) with off[r] >= e, else hi. The whole warp searches: 32
// probes a step.
__device__ __forceinline__ int warp_lower_bound(const int64_t *off, int lo, int hi, int64_t e) {
    const int lane = threadIdx.x & 31;
    while (lo < hi) {  // warp-uniform
        const int step = (hi - lo + 31) / 32;
        const int64_t r = (int64_t)lo + (int64_t)(lane + 1) * step - 1;  // the last of the lane's part
        const unsigned below = __ballot_sync(0xffffffffu, r < hi && off[r] < e);
        const int parts = __popc(below);  // whole parts below e
        lo += parts * step;
        hi = min(hi, lo + step - 1);      // the next part's last is not below e (or is past the end)
        if (step == 1) break;
    }
    return lo;
}

// The counts' row and the windows of chunk c.k.
__device__ __forceinline__ void bin_windows(const BinArgs &a, const BinView &v, BinChunk &c) {
    c.counts = v.counts + (int64_t)c.k * v.tiles_x * v.tiles_y;
    c.win_w = min(v.tiles_x, BIN_MAX_TILES);
    c.win_h = max(1, min(BIN_MAX_TILES / c.win_w, a.win_rows));
    c.wins_x = (v.tiles_x + c.win_w - 1) / c.win_w;
    c.wins = c.wins_x * ((v.tiles_y + c.win_h - 1) / c.win_h);
}

// Chunk b of the launch; every thread of the block must call it. False (block-uniform)
// where the view has fewer chunks. s_bounds: two shared ints. The emission takes the
// bounds from a.bounds, where the count leaves them.
template <bool BATCH>
__device__ __forceinline__ bool bin_chunk(const BinArgs &a, int b, BinView &v, BinChunk &c, int *s_bounds) {
    const int view = BATCH ? find_view(a.d.chunk_off, a.d.n_views, b) : 0;
    v = bin_view<BATCH>(a, view);
    c.k = BATCH ? b - a.d.chunk_off[view] : b;
    if (c.k >= v.chunks) {
        if (threadIdx.x == 0 && blockIdx.y == 0) a.bounds[b] = make_int2(0, 0);
        return false;
    }
    const int warp = threadIdx.x >> 5;
    if (warp < 2) {
        const int64_t e = v.first + v.entries * (c.k + warp) / v.chunks;
        const int r = warp_lower_bound(a.offsets_sorted, v.n0, v.n1, e);
        if ((threadIdx.x & 31) == 0) s_bounds[warp] = r;
    }
    __syncthreads();
    c.first = s_bounds[0];
    c.last = s_bounds[1];
    if (threadIdx.x == 0 && blockIdx.y == 0) a.bounds[b] = make_int2(c.first, c.last);
    bin_windows(a, v, c);
    return true;
}

__device__ __forceinline__ BinWindow bin_window(const BinView &v, const BinChunk &c, int i) {
    const int wy = i / c.wins_x, wx = i - wy * c.wins_x;
    BinWindow w;
    w.x0 = wx * c.win_w;
    w.y0 = wy * c.win_h;
    w.x1 = min(v.tiles_x, w.x0 + c.win_w);
    w.y1 = min(v.tiles_y, w.y0 + c.win_h);
    w.w = w.x1 - w.x0;
    return w;
}

// The tiles of a visible Gaussian's 3-sigma box, as the projection counted them.
__device__ __forceinline__ int4 rect_of(const Splat &s, float ax, float ay, int tx, int ty) {
    const float ccx = s.x / (float)TILE, ccy = s.y / (float)TILE;
    const float rrx = ax / (float)TILE, rry = ay / (float)TILE;
    const int x0 = min(max(0, (int)(ccx - rrx)), tx), x1 = min(max(0, (int)(ccx + rrx + 1)), tx);
    const int y0 = min(max(0, (int)(ccy - rry)), ty), y1 = min(max(0, (int)(ccy + rry + 1)), ty);
    return make_int4(x0, y0, x1, y1);
}

// The Gaussians' rectangles and tile counts in depth order (none for the invisible ones,
// which come last).
template <bool BATCH>
__global__ void bin_rects_kernel(const BinArgs a) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.n) return;
    const uint32_t g = a.order[r];
    int4 q = make_int4(0, 0, 0, 0);
    if (a.n_tiles[g] > 0) {
        int tx = a.tiles_x, ty = a.tiles_y;
        if (BATCH) {
            const int v = find_view(a.d.inst_off, a.d.n_views, r);  // the order is view-major
            tx = a.d.tiles_x[v];
            ty = a.d.tiles_y[v];
        }
        q = rect_of(a.splats[g], a.aabb[2 * (size_t)g], a.aabb[2 * (size_t)g + 1], tx, ty);
    }
    a.rects[r] = q;
    a.rect_tiles[r] = (q.z - q.x) * (q.w - q.y);
}

// A lane's walk over the tiles of a rectangle within a window, row-major, as cursor
// indices; `skip` tiles in (the walk wraps around at the end).
struct TileWalk {
    int i, row_end, width, jump;  // index, index past the row's last, tiles per row, to the next row
    int first, end;               // first index, and the index past the last row's last
    __device__ __forceinline__ void begin(int x0, int y0, int x1, int y1, const BinWindow &w) {
        width = x1 - x0;
        jump = w.w - width;
        first = (y0 - w.y0) * w.w + x0 - w.x0;
        end = first + (y1 - y0 - 1) * w.w + width;
        i = first;
        row_end = first + width;
    }
    __device__ __forceinline__ void skip(int tiles) {
        const int row = tiles / width;
        row_end += row * (width + jump);
        i = row_end - width + tiles - row * width;
    }
    __device__ __forceinline__ bool next() {  // whether a new row began
        if (++i < row_end) return false;
        if (i == end) i = first;
        else i += jump;
        row_end = i + width;
        return true;
    }
};

// Per-tile counts of a chunk. With offsets set, also every Gaussian's first emission
// index by Gaussian (the backward finds its slots from it).
template <bool BATCH>
__global__ void __launch_bounds__(BIN_THREADS) bin_count_kernel(const BinArgs a, int64_t *offsets) {
    __shared__ int cnt[BIN_MAX_TILES];
    __shared__ int bounds[2];
    BinView v;
    BinChunk c;
    if (!bin_chunk<BATCH>(a, blockIdx.x, v, c, bounds)) return;  // block-uniform
    const int lane = threadIdx.x & 31;
    if (offsets && blockIdx.y == 0)
        for (int r = c.first + threadIdx.x; r < c.last; r += BIN_THREADS) offsets[a.order[r]] = a.offsets_sorted[r];
    for (int wi = blockIdx.y; wi < c.wins; wi += gridDim.y) {  // block-uniform
        const BinWindow w = bin_window(v, c, wi);
        const int tiles = w.w * (w.y1 - w.y0);
        for (int i = threadIdx.x; i < tiles; i += BIN_THREADS) cnt[i] = 0;
        __syncthreads();
        for (int r0 = c.first; r0 < c.last; r0 += BIN_THREADS) {  // block-uniform
            const int r = r0 + threadIdx.x;
            const int4 q = r < c.last ? a.rects[r] : make_int4(0, 0, 0, 0);
            const int x0 = max(q.x, w.x0), y0 = max(q.y, w.y0), x1 = min(q.z, w.x1), y1 = min(q.w, w.y1);
            const int n = x0 < x1 && y0 < y1 ? (x1 - x0) * (y1 - y0) : 0;
            if (n > 0 && n <= BIN_LANE_MAX) {
                TileWalk t;
                t.begin(x0, y0, x1, y1, w);
                for (int j = 0; j < n; j++, t.next()) atomicAdd(&cnt[t.i], 1);
            }
            unsigned big = __ballot_sync(0xffffffffu, n > BIN_LANE_MAX);
            while (big) {  // warp-uniform
                const int src = __ffs(big) - 1;
                big &= big - 1;
                const int sx = __shfl_sync(0xffffffffu, x0, src), sy = __shfl_sync(0xffffffffu, y0, src);
                const int ex = __shfl_sync(0xffffffffu, x1, src), ey = __shfl_sync(0xffffffffu, y1, src);
                for (int y = sy; y < ey; y++)
                    for (int x = sx + lane; x < ex; x += 32) atomicAdd(&cnt[(y - w.y0) * w.w + x - w.x0], 1);
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < tiles; i += BIN_THREADS) {
            const int y = i / w.w;
            a.counts[c.counts + (int64_t)(w.y0 + y) * v.tiles_x + w.x0 + i - y * w.w] = cnt[i];
        }
        __syncthreads();
    }
}

// Per tile: the chunks' counts become exclusive prefixes, their sum the list's length.
// A block takes 32 tiles (its lanes), each warp a range of the chunks: sums first, then
// the prefixes from the sums of the warps before.
template <bool BATCH>
__global__ void __launch_bounds__(BIN_THREADS) bin_prefix_kernel(const BinArgs a) {
    __shared__ int part[BIN_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.x * 32 + lane, T = BATCH ? a.d.tile_off[a.d.n_views] : a.tiles_x * a.tiles_y;
    int live = 0, stride = T, lt = t;
    int64_t off = 0;
    if (t < T) {
        const int v = BATCH ? find_view(a.d.tile_off, a.d.n_views, t) : 0;
        const BinView b = bin_view<BATCH>(a, v);
        live = b.chunks;
        lt = t - b.tile0;
        stride = b.tiles_x * b.tiles_y;
        off = b.counts;
    }
    const int per = (live + BIN_WARPS - 1) / BIN_WARPS;
    const int k0 = min(live, warp * per), k1 = min(live, k0 + per);
    int32_t *col = a.counts + off + lt;
    int sum = 0;
#pragma unroll 4
    for (int k = k0; k < k1; k++) sum += col[(int64_t)k * stride];
    part[warp][lane] = sum;
    __syncthreads();
    int run = 0;
    for (int w = 0; w < warp; w++) run += part[w][lane];
    for (int k = k0; k < k1; k += 4) {  // loads of a group before its stores
        int c[4];
#pragma unroll
        for (int u = 0; u < 4; u++) c[u] = k + u < k1 ? col[(int64_t)(k + u) * stride] : 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (k + u < k1) col[(int64_t)(k + u) * stride] = run;
            run += c[u];
        }
    }
    if (warp == BIN_WARPS - 1 && t < a.tile_cap) a.tile_end[t] = t < T ? run : 0;
}

// tile_end holds the lengths; exclusive scan into tile_start, and tile_end = start +
// length. One block: a 1080p frame's 8160 tiles are one round.
constexpr int SCAN_THREADS = 1024, SCAN_PER = 8;

// order (ORDER; T <= BIN_ORDER_MAX): the tiles for the rasterizers' blocks, by the
// length of their lists, the longest first, so that the last blocks to start are short
// ones (a tile of the frame's last rows may hold its longest list). A counting sort over
// eighths of each power of two; tiles of one step in no particular order, which changes
// no tile's result. It costs 2.5 to 5 us and pays where a list's length measures its
// tile's work, which it does while lists are walked to their ends: forward and backward
// of 50 k to 200 k Gaussians at 512 x 512 to 1920 x 1080 (220 to 440 entries a tile) gain 8
// to 60 us of 250 to 680, 500 k of a street at 1024 x 512 4 to 48 of 240 to 450, early
// street steps 4 % of the step, the render of 500 k faint ones (1090 a tile) 55 of 750.
// Where they are long and opaque, pixels are done before their ends and the tiles that
// take longest come late: 730 to 870 entries a tile gain 26 to -29 us, 1100 to 1750 20 to
// -67, 3800 -6 to -107 of 1700, the backward's most of it. The average length tells the two
// apart no better than that (ending at 1024 cost the faint render its 55 us). At 1600 x
// 1060, eight rounds of blocks, nothing either way. Frames of up to BIN_ORDER_MIN tiles
// start them all at once: ordering them made a 256 x 256 step 1.5 % slower.
constexpr int ORDER_STEPS = 256;
static_assert(BIN_ORDER_MAX <= SCAN_THREADS * SCAN_PER, "one round");

__device__ __forceinline__ int order_step(int len) {
    return len > 0 ? ORDER_STEPS - 2 - (int)((__float_as_uint((float)len) >> 20) - (127u << 3)) : ORDER_STEPS - 1;
}

template <bool ORDER>
__global__ void __launch_bounds__(SCAN_THREADS) bin_starts_kernel(int T, int32_t *tile_start, int32_t *tile_end,
                                                                  int32_t *order) {
    __shared__ long long ws[32];
    __shared__ int step[ORDER ? ORDER_STEPS : 1], wsum[ORDER_STEPS / 32];
    if (ORDER && threadIdx.x < ORDER_STEPS) step[threadIdx.x] = 0;  // read after the scan's barriers
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long carry = 0;
    for (int b0 = 0; b0 < T; b0 += SCAN_THREADS * SCAN_PER) {
        const int i0 = b0 + threadIdx.x * SCAN_PER;
        int v[SCAN_PER];
        long long s = 0;
        const bool whole = i0 + SCAN_PER <= T;  // the buffers are 16-byte aligned, i0 a multiple of 8
        if (whole) {
            const int4 a = reinterpret_cast<const int4 *>(tile_end + i0)[0], b = reinterpret_cast<const int4 *>(tile_end + i0)[1];
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
            v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
        } else {
#pragma unroll
            for (int j = 0; j < SCAN_PER; j++) v[j] = i0 + j < T ? tile_end[i0 + j] : 0;
        }
#pragma unroll
        for (int j = 0; j < SCAN_PER; j++) s += v[j];
        long long inc = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) ws[warp] = inc;
        __syncthreads();
        long long x = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += u;
        }
        const long long all = __shfl_sync(0xffffffffu, x, 31);
        const long long before = __shfl_sync(0xffffffffu, x, max(warp - 1, 0));
        long long p = carry + (warp > 0 ? before : 0) + inc - s;
        int first[SCAN_PER];
#pragma unroll
        for (int j = 0; j < SCAN_PER; j++) {
            first[j] = (int)p;
            p += v[j];
            v[j] = (int)p;
        }
        if (whole) {
            int4 *s4 = reinterpret_cast<int4 *>(tile_start + i0), *e4 = reinterpret_cast<int4 *>(tile_end + i0);
            s4[0] = make_int4(first[0], first[1], first[2], first[3]);
            s4[1] = make_int4(first[4], first[5], first[6], first[7]);
            e4[0] = make_int4(v[0], v[1], v[2], v[3]);
            e4[1] = make_int4(v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
            for (int j = 0; j < SCAN_PER; j++)
                if (i0 + j < T) {
                    tile_start[i0 + j] = first[j];
                    tile_end[i0 + j] = v[j];
                }
        }
        carry += all;
        __syncthreads();
        if constexpr (!ORDER) continue;
#pragma unroll
        for (int j = 0; j < SCAN_PER; j++) {
            v[j] = i0 + j < T ? order_step(v[j] - first[j]) : -1;
            const unsigned none = __ballot_sync(0xffffffffu, v[j] == ORDER_STEPS - 1);  // often most of a frame
            if (v[j] >= 0 && v[j] < ORDER_STEPS - 1) atomicAdd(&step[v[j]], 1);
            if (lane == 0 && none) atomicAdd(&step[ORDER_STEPS - 1], __popc(none));
        }
        __syncthreads();
        int c = 0, incl = 0;
        if (threadIdx.x < ORDER_STEPS) {  // whole warps
            c = incl = step[threadIdx.x];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            if (lane == 31) wsum[warp] = incl;
        }
        __syncthreads();
        if (threadIdx.x < ORDER_STEPS) {
            for (int w = 0; w < warp; w++) incl += wsum[w];
            step[threadIdx.x] = incl - c;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < SCAN_PER; j++) {
            const unsigned none = __ballot_sync(0xffffffffu, v[j] == ORDER_STEPS - 1);
            int at = 0;
            if (lane == 0 && none) at = atomicAdd(&step[ORDER_STEPS - 1], __popc(none));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(none & ((1u << lane) - 1u));
            if (v[j] >= 0 && v[j] < ORDER_STEPS - 1) at = atomicAdd(&step[v[j]], 1);
            if (v[j] >= 0) order[at] = i0 + j;
        }
    }
}

// Writes the lists. A warp owns a band of the window's tile rows and walks the whole
// chunk in order, collecting the Gaussians that reach its band until it has one for each
// lane. The 32 are then dealt at once, each lane walking its own Gaussian's tiles three
// times: it sets its bit in the tile's mask; its place is the tile's cursor plus the bits
// of the lanes before it; and the last lane of a mask advances the cursor and clears it.
// (Dealing them one after another, a lane a tile, took 6.6 warp instructions an entry:
// few tiles to a Gaussian in a band, and every step waits for the last.) A rectangle too
// large for a lane is dealt by the warp, after the ones collected before it. The warps of
// a block share no tile, so no order between them matters. MAP: also the inverse map,
// emission index -> list position, for the backward's per-Gaussian sums; a Gaussian's
// intersections are numbered from its offset in row-major tile order. Entries at or past
// cap are dropped.
struct BinShared {
    int cursor[BIN_MAX_TILES];
    unsigned mask[BIN_MAX_TILES];
    int queue[BIN_WARPS][64];
};

template <bool MAP>
__device__ __forceinline__ void bin_deal(const BinArgs &a, BinShared &s, const BinWindow &w, int by0, int by1, int r,
                                         int32_t *gids, int32_t *inv, unsigned cap) {
    const int lane = threadIdx.x & 31;
    const unsigned bit = 1u << lane;
    int n = 0, g = 0;
    unsigned e = 0, e_jump = 0;
    TileWalk t0;
    t0.begin(0, 0, 1, 1, w);
    if (r >= 0) {
        const int4 q = a.rects[r];
        const int x0 = max(q.x, w.x0), y0 = max(q.y, by0), x1 = min(q.z, w.x1), y1 = min(q.w, by1);
        n = (x1 - x0) * (y1 - y0);
        g = (int)a.order[r];
        if (MAP) {
            e = (unsigned)a.offsets_sorted[r] + (unsigned)((y0 - q.y) * (q.z - q.x) + x0 - q.x);
            e_jump = (unsigned)((q.z - q.x) - (x1 - x0));
        }
        t0.begin(x0, y0, x1, y1, w);
    }
    // from different tiles on, so that lanes with much the same rectangle do not all wait
    // for one mask
    TileWalk t = t0;
    if (n > 8) t.skip((n * lane) >> 5);
    for (int j = 0; j < n; j++, t.next()) atomicOr(&s.mask[t.i], bit);
    __syncwarp();
    t = t0;
    for (int j = 0; j < n; j++) {
        const unsigned pos = (unsigned)s.cursor[t.i] + __popc(s.mask[t.i] & (bit - 1u));
        if (pos < cap) {
            gids[pos] = g;
            if (MAP && e < cap) inv[e] = (int)pos;
        }
        e++;
        if (t.next()) e += e_jump;
    }
    __syncwarp();
    t = t0;
    for (int j = 0; j < n; j++, t.next()) {
        const unsigned m = s.mask[t.i];
        if (m >> lane == 1u) {  // the last lane (a mask already cleared is 0)
            s.cursor[t.i] += __popc(m);
            s.mask[t.i] = 0u;
        }
    }
    __syncwarp();
}

template <bool BATCH, bool MAP>
__global__ void __launch_bounds__(BIN_THREADS) bin_emit_kernel(const BinArgs a, int32_t *gids, int32_t *inv,
                                                               unsigned cap) {
    __shared__ BinShared s;
    BinView v;
    BinChunk c;
    const int2 bounds = a.bounds[blockIdx.x];
    c.first = bounds.x;
    c.last = bounds.y;
    if (c.first >= c.last) return;  // block-uniform: the view has fewer chunks
    const int view = BATCH ? find_view(a.d.chunk_off, a.d.n_views, blockIdx.x) : 0;
    bin_grid<BATCH>(a, view, v);
    c.k = BATCH ? (int)blockIdx.x - a.d.chunk_off[view] : blockIdx.x;
    bin_windows(a, v, c);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int *queue = s.queue[warp];
    for (int wi = blockIdx.y; wi < c.wins; wi += gridDim.y) {  // block-uniform
        const BinWindow w = bin_window(v, c, wi);
        const int rows = w.y1 - w.y0, tiles = w.w * rows;
        for (int i = threadIdx.x; i < tiles; i += BIN_THREADS) {
            const int y = i / w.w, t = (w.y0 + y) * v.tiles_x + w.x0 + i - y * w.w;
            s.cursor[i] = a.tile_start[v.tile0 + t] + a.counts[c.counts + t];
            s.mask[i] = 0u;
        }
        __syncthreads();
        const int band = (rows + BIN_WARPS - 1) / BIN_WARPS;
        const int by0 = min(w.y1, w.y0 + warp * band), by1 = min(w.y1, by0 + band);
        if (by0 < by1) {  // warp-uniform; no block barrier inside
            int head = 0, queued = 0;  // warp-uniform: positions queue[head & 63 ...]
            int4 q = c.first + lane < c.last ? a.rects[c.first + lane] : make_int4(0, 0, 0, 0);
            for (int r0 = c.first; r0 < c.last; r0 += 32) {  // warp-uniform
                const int x0 = max(q.x, w.x0), y0 = max(q.y, by0), x1 = min(q.z, w.x1), y1 = min(q.w, by1);
                const int n = x0 < x1 && y0 < y1 ? (x1 - x0) * (y1 - y0) : 0;
                // the next 32 rectangles' load, while these are dealt
                q = r0 + 32 + lane < c.last ? a.rects[r0 + 32 + lane] : make_int4(0, 0, 0, 0);
                unsigned small = __ballot_sync(0xffffffffu, n > 0 && n <= BIN_LANE_MAX);
                unsigned big = __ballot_sync(0xffffffffu, n > BIN_LANE_MAX);
                for (;;) {  // warp-uniform: the small ones before the next large one, then that one
                    const unsigned upto = big ? (big & (0u - big)) - 1u : 0xffffffffu;
                    const unsigned m = small & upto;
                    if ((m >> lane) & 1u) queue[(head + queued + __popc(m & ((1u << lane) - 1u))) & 63] = r0 + lane;
                    small &= ~upto;
                    queued += __popc(m);
                    __syncwarp();
                    while (queued >= 32 || (big && queued > 0)) {
                        bin_deal<MAP>(a, s, w, by0, by1, lane < queued ? queue[(head + lane) & 63] : -1, gids, inv,
                                      cap);
                        const int took = min(queued, 32);
                        head += took;
                        queued -= took;
                    }
                    if (!big) break;
                    const int src = __ffs(big) - 1;
                    big &= big - 1;
                    const int sx = __shfl_sync(0xffffffffu, x0, src), sy = __shfl_sync(0xffffffffu, y0, src);
                    const int ex = __shfl_sync(0xffffffffu, x1, src), ey = __shfl_sync(0xffffffffu, y1, src);
                    const int g = (int)a.order[r0 + src];
                    unsigned e = 0, pitch = 0;
                    if (MAP) {
                        const int4 full = a.rects[r0 + src];
                        pitch = (unsigned)(full.z - full.x);
                        e = (unsigned)a.offsets_sorted[r0 + src] + (unsigned)(sy - full.y) * pitch - (unsigned)full.x;
                    }
                    for (int y = sy; y < ey; y++, e += pitch)
                        for (int x = sx + lane; x < ex; x += 32) {
                            int *cur = &s.cursor[(y - w.y0) * w.w + x - w.x0];
                            const unsigned pos = (unsigned)*cur;
                            *cur = (int)pos + 1;
                            if (pos < cap) {
                                gids[pos] = g;
                                if (MAP && e + x < cap) inv[e + x] = (int)pos;
                            }
                        }
                    __syncwarp();
                }
            }
            if (queued > 0)
                bin_deal<MAP>(a, s, w, by0, by1, lane < queued ? queue[(head + lane) & 63] : -1, gids, inv, cap);
        }
        __syncthreads();
    }
}

// View of each instance, in the depth order of all: the key of the pass that makes the
// order view-major.
__global__ void bin_view_keys_kernel(int n, const uint32_t *order, const BatchDesc d, uint32_t *keys) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) keys[r] = (uint32_t)find_view(d.inst_off, d.n_views, (int)order[r]);
}

// Gaussians to a chunk on average, which sets the number of chunks (each then takes an
// equal share of the intersections, however many Gaussians that is): so many chunks that
// there are four blocks an SM, but 64 to 2048 Gaussians each. The upper end keeps the
// writes of the lists in L2: the blocks at work at a time (some 600) then fill one
// stretch of every list, about 60 MB in all, line after line; with all chunks of a 100
// M-entry batch at work at once half-filled lines went to memory (2.28 ms against 1.26).
// Above it only where the per-tile counts (a row of the frame's tiles per chunk) would
// take more than BIN_MAX_COUNTS. tiles: the view's, in a batch the largest view's. A view
// uses fewer chunks where they would hold less than BIN_MIN_ENTRIES intersections.
constexpr int64_t BIN_MAX_COUNTS = 1 << 26;
int bin_chunk_len(int64_t n, int64_t tiles) {
    const int64_t len = std::min<int64_t>(2048, std::max<int64_t>(64, (n + GPU_PLACES - 1) / GPU_PLACES));
    return (int)std::min<int64_t>(INT32_MAX, std::max(len, (n * tiles + BIN_MAX_COUNTS - 1) / BIN_MAX_COUNTS));
}
int bin_chunks(int n, int len) { return (int)(((int64_t)n + len - 1) / len); }

// Blocks per chunk, each taking windows of its own: two in a batch, whose views' sizes the
// host need not know; else one per window, and up to eight where the chunks alone would
// leave SMs idle, with windows of fewer rows (a row for every warp at least).
void bin_plan(BinArgs &a) {
    a.win_rows = BIN_MAX_TILES;
    a.grid_y = 2;
    if (a.d.n_views > 0) return;
    const int split = std::min(8, std::max(1, GPU_PLACES / std::max(1, a.chunks)));
    if (split > 1) a.win_rows = std::max(BIN_WARPS, (a.tiles_y + split - 1) / split);
    const int w = std::min(a.tiles_x, BIN_MAX_TILES), h = std::max(1, std::min(BIN_MAX_TILES / w, a.win_rows));
    a.grid_y = std::min(8, ((a.tiles_x + w - 1) / w) * ((a.tiles_y + h - 1) / h));
}

// The depth order of a.n instances from their keys (s.keys[0], s.vals[0]), view-major in
// a batch: a.order; their rectangles, and their first emission indices in that order with
// the total.
void launch_depth_order(BinArgs &a, DepthScratch &s, int64_t *scan_part, int64_t *total, cudaStream_t st) {
    a.order = s.vals[0];
    a.total = total;
    if (a.n <= 0) {
        cudaMemsetAsync(total, 0, sizeof(int64_t), st);
        return;
    }
    int cur = radix_sort_pairs32(s.keys, s.vals, a.n, 32, s.radix_scratch, st);
    const bool batch = a.d.n_views > 0;
    if (a.d.n_views > 1) {
        uint32_t *k[2] = {s.keys[cur], s.keys[cur ^ 1]}, *v[2] = {s.vals[cur], s.vals[cur ^ 1]};
        bin_view_keys_kernel<<<(a.n + 255) / 256, 256, 0, st>>>(a.n, v[0], a.d, k[0]);
        int bits = 1;
        while ((1 << bits) < a.d.n_views) bits++;
        cur ^= radix_sort_pairs32(k, v, a.n, bits, s.radix_scratch, st);
    }
    a.order = s.vals[cur];
    if (batch) bin_rects_kernel<true><<<(a.n + 255) / 256, 256, 0, st>>>(a);
    else bin_rects_kernel<false><<<(a.n + 255) / 256, 256, 0, st>>>(a);
    scan_exclusive<int64_t>(a.rect_tiles, a.offsets_sorted, a.n, total, scan_part, st);
}

// Counts, prefixes and list starts; offsets (may be null): the emission indices by
// Gaussian.
void launch_bin_count(const BinArgs &a, int64_t *offsets, cudaStream_t st) {
    const bool batch = a.d.n_views > 0;
    if (a.n > 0) {
        const dim3 grid((unsigned)a.chunks, (unsigned)a.grid_y);
        if (batch) bin_count_kernel<true><<<grid, BIN_THREADS, 0, st>>>(a, offsets);
        else bin_count_kernel<false><<<grid, BIN_THREADS, 0, st>>>(a, offsets);
    }
    const int blocks = (a.tile_cap + 31) / 32;
    if (batch) bin_prefix_kernel<true><<<blocks, BIN_THREADS, 0, st>>>(a);
    else bin_prefix_kernel<false><<<blocks, BIN_THREADS, 0, st>>>(a);
    if (a.tile_order) bin_starts_kernel<true><<<1, SCAN_THREADS, 0, st>>>(a.tile_cap, a.tile_start, a.tile_end, a.tile_order);
    else bin_starts_kernel<false><<<1, SCAN_THREADS, 0, st>>>(a.tile_cap, a.tile_start, a.tile_end, nullptr);
}

void launch_bin_emit(const BinArgs &a, int32_t *gids, int32_t *inv, int64_t cap, cudaStream_t st) {
    if (a.n <= 0 || cap <= 0) return;
    const dim3 grid((unsigned)a.chunks, (unsigned)a.grid_y);
    const unsigned c = (unsigned)std::min<int64_t>(cap, INT32_MAX);
    const bool batch = a.d.n_views > 0;
    if (batch && inv) bin_emit_kernel<true, true><<<grid, BIN_THREADS, 0, st>>>(a, gids, inv, c);
    else if (batch) bin_emit_kernel<true, false><<<grid, BIN_THREADS, 0, st>>>(a, gids, nullptr, c);
    else if (inv) bin_emit_kernel<false, true><<<grid, BIN_THREADS, 0, st>>>(a, gids, inv, c);
    else bin_emit_kernel<false, false><<<grid, BIN_THREADS, 0, st>>>(a, gids, nullptr, c);
}

// A capacity-bounded (graph-capturable) step whose lists exceed the buffers renders
// nothing and updates nothing: the lists are emptied and *overflow set; the host grows
// the buffers and repeats it.
__global__ void bin_clamp_kernel(const int64_t *total, int64_t cap, int T, int32_t *tile_start, int32_t *tile_end,
                                 int *d_n, int *overflow) {
    const int64_t n = *total;
    const bool over = n > cap;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (over && t < T) tile_start[t] = tile_end[t] = 0;
    if (t == 0) {
        *d_n = over ? 0 : (int)n;
        if (over) *overflow = 1;
    }
}

void launch_bin_clamp(const BinArgs &a, int64_t cap, int *d_n, int *overflow, cudaStream_t st) {
    bin_clamp_kernel<<<(a.tile_cap + 255) / 256, 256, 0, st>>>(a.total, cap, a.tile_cap, a.tile_start, a.tile_end, d_n,
                                                              overflow);
}

}  // namespace msplat
