// Exclusive scan and stable radix sort.
//
// The radix sort is reduce-then-scan per 8-bit digit: a histogram kernel, a device
// scan of the digit-major counts, and a scatter kernel that ranks keys stably inside
// each 2048-key block with warp ballots and popc, no block waiting on another; small
// sorts of 32-bit keys run in one cluster of eight blocks instead.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace msplat {

// ---------------------------------------------------------------------------------
// Exclusive scan (int32 in, TO out), 2048 elements per block, three kernels.

constexpr int SCAN_THREADS = 256, SCAN_ITEMS = 8, SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T *warp_sums, T &block_total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        T w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : T(0);
        T wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < (int)(blockDim.x >> 5)) warp_sums[lane] = wi - w;
        if (lane == 31) warp_sums[32] = wi;
    }
    __syncthreads();
    T r = warp_sums[warp] + inc - v;
    block_total = warp_sums[32];
    __syncthreads();
    return r;
}

template <typename TO>
__global__ void scan_reduce_kernel(const int32_t *in, int n, TO *partials) {
    __shared__ TO ws[33];
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    TO s = 0;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; j++)
        if (base + j < n) s += (TO)in[base + j];
    TO tot;
    block_exclusive_scan<TO>(s, ws, tot);
    if (threadIdx.x == 0) partials[blockIdx.x] = tot;
}

template <typename TO>
__global__ void scan_partials_kernel(TO *partials, int nb, TO *total) {
    __shared__ TO ws[33];
    TO carry = 0;
    for (int base = 0; base < nb; base += blockDim.x) {
        const int i = base + threadIdx.x;
        TO v = i < nb ? partials[i] : TO(0);
        TO tot;
        TO ex = block_exclusive_scan<TO>(v, ws, tot);
        if (i < nb) partials[i] = ex + carry;
        carry += tot;
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

template <typename TO>
__global__ void scan_apply_kernel(const int32_t *in, int n, const TO *partials, TO *out) {
    __shared__ TO ws[33];
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    TO v[SCAN_ITEMS];
    TO s = 0;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; j++) {
        v[j] = base + j < n ? (TO)in[base + j] : TO(0);
        s += v[j];
    }
    TO tot;
    TO ex = block_exclusive_scan<TO>(s, ws, tot) + partials[blockIdx.x];
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; j++) {
        if (base + j < n) out[base + j] = ex;
        ex += v[j];
    }
}

int scan_blocks(int n) { return (n + SCAN_TILE - 1) / SCAN_TILE; }

// Small inputs: one 1024-thread block, 16 consecutive elements a thread (one launch
// instead of three). Bound by latency: loads and stores of 16 bytes, one block-wide scan.
// 10 k elements into 64 bits: 9.1 -> 5.7 us against rounds of four elements a thread.
constexpr int SMALL_ITEMS = 16, SCAN_SMALL = 1024 * SMALL_ITEMS;

template <typename TO>
__global__ void __launch_bounds__(1024) scan_small_kernel(const int32_t *in, int n, TO *out, TO *total) {
    __shared__ TO ws[33];
    const int i0 = threadIdx.x * SMALL_ITEMS;
    // 16-byte accesses: the thread's first element lies on 64 bytes where the arrays do on 16
    const bool wide = i0 + SMALL_ITEMS <= n &&
                      ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    int32_t v[SMALL_ITEMS];
    if (wide) {
#pragma unroll
        for (int j = 0; j < SMALL_ITEMS; j += 4) {
            const int4 q = *reinterpret_cast<const int4 *>(in + i0 + j);
            v[j] = q.x, v[j + 1] = q.y, v[j + 2] = q.z, v[j + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < SMALL_ITEMS; j++) v[j] = i0 + j < n ? in[i0 + j] : 0;
    }
    TO s = 0, tot;
#pragma unroll
    for (int j = 0; j < SMALL_ITEMS; j++) s += (TO)v[j];
    TO ex = block_exclusive_scan<TO>(s, ws, tot);
    if (wide) {
        constexpr int PER = 16 / sizeof(TO);
        struct alignas(16) Pack {
            TO e[PER];
        };
#pragma unroll
        for (int j = 0; j < SMALL_ITEMS; j += PER) {
            Pack p;
#pragma unroll
            for (int u = 0; u < PER; u++) {
                p.e[u] = ex;
                ex += (TO)v[j + u];
            }
            *reinterpret_cast<Pack *>(out + i0 + j) = p;
        }
    } else {
#pragma unroll
        for (int j = 0; j < SMALL_ITEMS; j++) {
            if (i0 + j < n) out[i0 + j] = ex;
            ex += (TO)v[j];
        }
    }
    if (threadIdx.x == 0 && total) *total = tot;
}

template <typename TO>
void scan_exclusive(const int32_t *in, TO *out, int n, TO *d_total, TO *partials, cudaStream_t st) {
    if (n <= 0) {
        if (d_total) cudaMemsetAsync(d_total, 0, sizeof(TO), st);
        return;
    }
    if (n <= SCAN_SMALL) {
        scan_small_kernel<TO><<<1, 1024, 0, st>>>(in, n, out, d_total);
        return;
    }
    const int nb = scan_blocks(n);
    scan_reduce_kernel<TO><<<nb, SCAN_THREADS, 0, st>>>(in, n, partials);
    scan_partials_kernel<TO><<<1, 1024, 0, st>>>(partials, nb, d_total);
    scan_apply_kernel<TO><<<nb, SCAN_THREADS, 0, st>>>(in, n, partials, out);
}
template void scan_exclusive<int32_t>(const int32_t *, int32_t *, int, int32_t *, int32_t *, cudaStream_t);
template void scan_exclusive<int64_t>(const int32_t *, int64_t *, int, int64_t *, int64_t *, cudaStream_t);

// ---------------------------------------------------------------------------------
// Stable LSD radix sort of (key, u32 value) pairs by key bits [0, key_bits), for
// 32- and 64-bit keys.

constexpr int RADIX = 256;
// Keys per block: THREADS x ITEMS. Large sorts of 32-bit keys take 256 threads x 16
// items (4096 keys a block): each digit's run in a block then averages 16 entries, so
// the scatter's stores come in runs of 64 bytes or more, and the per-block digit counts
// (256 per block, scanned every pass) stay small next to the keys. The depth order of 12
// million instances (32 bits): histograms 70, scatters 414 and scans 138 us against 89,
// 420 and 155 in 2048-key blocks. Below LARGE_SORT keys, 256 x 8 (2048 keys a block) keeps
// enough blocks to fill the GPU; 64-bit keys take 2048-key blocks too (4096 would need 48
// KB of staging per block). The scatter is bound by its integer pipe: the ranking's
// ballots, not DRAM, set its pace.
constexpr int SORT_THREADS = 256;
constexpr int LARGE_SORT = 4 << 20;
constexpr int MAX_SORT_THREADS = 1024;

// Up to this many blocks (131,072 keys at 2048 a block, the depth order of a training
// view), each scatter block sums the per-block digit counts itself instead of a
// separate scan launch over them.
constexpr int DIRECT_SORT_BLOCKS = 64;

// The most blocks any sort of up to n keys uses (scratch sizing): 2048-key blocks,
// the smallest of every block shape below.
int radix_max_blocks(int n) { return (n + 2047) / 2048; }

// The lanes of the warp whose digit equals this lane's (d in 0..RADIX, RADIX marking
// a lane with no key): nine ballots, one per bit of d, each narrowing the set to the
// lanes that agree on that bit. Constant cost whatever the number of distinct digits
// in the warp (up to 32).
// Only the bits a pass's digits can hold take a ballot (mask, uniform), and the no-key
// bit only in a block that is not full (full: every lane holds a key).
__device__ __forceinline__ unsigned digit_peers(int d, uint32_t mask, bool full) {
    unsigned m = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 9; b++) {
        if (b < 8 ? !((mask >> b) & 1u) : full) continue;  // uniform
        const bool on = (d >> b) & 1;
        const unsigned bal = __ballot_sync(0xffffffffu, on);
        m &= on ? bal : ~bal;
    }
    return m;
}

// Counting needs no ranks: each warp adds its keys' digits to its own shared-memory
// histogram with one atomic per key (lanes of a warp that share a digit are resolved
// by the shared-memory atomic unit), and the block sums the warps' histograms.
// d_n (may be null): a device-side count that caps n (capacity-bounded launches).
template <typename K, int THREADS, int SORT_ITEMS>
__global__ void __launch_bounds__(THREADS) radix_hist_kernel(const K *keys, int n, const int *d_n, int shift,
                                                             uint32_t mask, uint32_t *counts, int nb) {
    constexpr int WARPS = THREADS / 32;
    __shared__ uint32_t h[WARPS][RADIX];
    if (d_n) n = min(n, *d_n);
    for (int i = threadIdx.x; i < WARPS * RADIX; i += THREADS) (&h[0][0])[i] = 0;
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    constexpr int SORT_TILE = THREADS * SORT_ITEMS;
    const int base = blockIdx.x * SORT_TILE;
    int dig[SORT_ITEMS];
#pragma unroll
    for (int j = 0; j < SORT_ITEMS; j++) {  // independent loads first
        const int k = base + j * THREADS + threadIdx.x;
        dig[j] = k < n ? (int)((keys[k] >> shift) & mask) : RADIX;
    }
#pragma unroll
    for (int j = 0; j < SORT_ITEMS; j++)
        if (dig[j] < RADIX) atomicAdd(&h[warp][dig[j]], 1u);
    __syncthreads();
    for (int i = threadIdx.x; i < RADIX; i += THREADS) {
        uint32_t s = 0;
#pragma unroll
        for (int w = 0; w < WARPS; w++) s += h[w][i];
        counts[(size_t)i * nb + blockIdx.x] = s;
    }
}

// offs: the exclusive digit-major scan of the per-block digit counts; or, with offs
// null (a sort of at most DIRECT_SORT_BLOCKS blocks), counts: the per-block digit counts
// themselves, from which each block forms its own digit starts (no scan launch).
// The 64-bit-key scatter is held to 64 registers, four resident blocks per SM (32 M
// pairs of 40 bits: 2.35 instead of 2.49 ms); the 32-bit ones to 128 (the depth order
// of a street view's 100 k Gaussians ran 10 % slower at 64).
template <typename K, int THREADS, int SORT_ITEMS>
__global__ void __launch_bounds__(THREADS, sizeof(K) == 8 ? 1024 / THREADS : 512 / THREADS) radix_scatter_kernel(const K *kin, const uint32_t *vin, K *kout,
                                                                uint32_t *vout, int n, const int *d_n, int shift,
                                                                uint32_t mask, const int32_t *offs,
                                                                const uint32_t *counts, int nb) {
    // The block's keys are first ranked and placed in shared memory in digit order
    // (a block-local stable multisplit), then written out so that consecutive threads
    // write consecutive entries of each digit's run: coalesced global stores.
    static_assert(THREADS >= RADIX && THREADS <= MAX_SORT_THREADS, "a thread per digit");
    constexpr int WARPS = THREADS / 32;
    __shared__ uint32_t wcnt[WARPS][RADIX];
    __shared__ uint32_t gbase[RADIX], bstart[RADIX + 1];
    constexpr int SORT_TILE = THREADS * SORT_ITEMS;  // keys per block
    constexpr int WARP_KEYS = SORT_TILE / WARPS;     // contiguous keys per warp
    __shared__ uint32_t ws[33];
    extern __shared__ __align__(16) unsigned char sort_smem[];  // radix_scatter_smem<K, SORT_ITEMS>()
    K *skey = reinterpret_cast<K *>(sort_smem);
    uint32_t *sval = reinterpret_cast<uint32_t *>(skey + SORT_TILE);
    if (d_n) n = min(n, *d_n);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < WARPS * RADIX; i += THREADS) (&wcnt[0][0])[i] = 0;
    if (offs) {
        for (int i = threadIdx.x; i < RADIX; i += THREADS) gbase[i] = (uint32_t)offs[(size_t)i * nb + blockIdx.x];
    } else {  // thread d: digit d's count over all blocks and over the blocks before this one
        uint32_t tot = 0u, before = 0u;
        if (threadIdx.x < RADIX) {
            const uint32_t *row = counts + (size_t)threadIdx.x * nb;
            for (int b = 0; b < nb; b++) {
                const uint32_t c = row[b];
                tot += c;
                if (b < (int)blockIdx.x) before += c;
            }
        }
        uint32_t all;
        const uint32_t ex = block_exclusive_scan<uint32_t>(tot, ws, all) + before;
        if (threadIdx.x < RADIX) gbase[threadIdx.x] = ex;
    }
    K key[SORT_ITEMS];
    uint32_t val[SORT_ITEMS], rank[SORT_ITEMS];
    int dig[SORT_ITEMS];
    const int base = blockIdx.x * SORT_TILE + warp * WARP_KEYS;
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; r++) {  // independent loads first
        const int k = base + r * 32 + lane;
        const bool ok = k < n;
        key[r] = ok ? kin[k] : K(0);
        val[r] = ok ? vin[k] : 0u;
        dig[r] = ok ? (int)((key[r] >> shift) & mask) : RADIX;
    }
    __syncthreads();
    const unsigned lt = (1u << lane) - 1u;
    const bool full = (int64_t)blockIdx.x * SORT_TILE + SORT_TILE <= (int64_t)n;
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; r++) {
        const int d = dig[r];
        const bool ok = d < RADIX;
        const unsigned peers = digit_peers(d, mask, full);
        const uint32_t before = ok ? wcnt[warp][d] : 0u;
        rank[r] = before + (uint32_t)__popc(peers & lt);
        __syncwarp();
        if (ok && lane == __ffs(peers) - 1) wcnt[warp][d] = before + (uint32_t)__popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit: exclusive prefix over warps, then over digits (block-local starts)
    uint32_t tot = 0;
    if (threadIdx.x < RADIX) {
        const int d = threadIdx.x;
#pragma unroll
        for (int w = 0; w < WARPS; w++) {
            const uint32_t t = wcnt[w][d];
            wcnt[w][d] = tot;
            tot += t;
        }
    }
    uint32_t btot;
    const uint32_t ex = block_exclusive_scan<uint32_t>(threadIdx.x < RADIX ? tot : 0u, ws, btot);
    if (threadIdx.x < RADIX) bstart[threadIdx.x] = ex;
    if (threadIdx.x == 0) bstart[RADIX] = btot;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; r++) {
        const int d = dig[r];
        if (d < RADIX) {
            const uint32_t lp = bstart[d] + wcnt[warp][d] + rank[r];
            skey[lp] = key[r];
            sval[lp] = val[r];
        }
    }
    __syncthreads();
    const int valid = (int)bstart[RADIX];
    for (int i = threadIdx.x; i < valid; i += THREADS) {
        const K kk = skey[i];
        const int d = (int)((kk >> shift) & mask);
        const uint32_t pos = gbase[d] + ((uint32_t)i - bstart[d]);
        kout[pos] = kk;
        vout[pos] = sval[i];
    }
}

// Sorts of at most CLUSTER_SORT 32-bit keys (the depth order of a small scene): one
// cluster of eight blocks keeps them in registers and distributed shared memory through
// all the passes. A block ranks its part as the scatter does, the blocks exchange their
// digit counts, and every key goes straight to its place in the shared memory of the
// block that holds it next. In place; one launch where the histogram and scatter kernels
// take two a pass, few blocks each. The cluster's time grows with the keys, theirs does
// not while their blocks find SMs free: 10 k keys of 32 bits 30 -> 20 us, 17 k 31 -> 28, 20 k
// 31 -> 30; but 24 k 31 -> 33, 40 k 33 -> 50 and 65 k 47 -> 69, so it ends at 20,480.
constexpr int CLUSTER_BLOCKS = 8, CLUSTER_THREADS = 1024;
constexpr int CLUSTER_SORT = CLUSTER_BLOCKS * CLUSTER_THREADS * 5 / 2;

// per: keys a block holds, a multiple of 32, at most CLUSTER_THREADS * KEYS.
template <int KEYS>
__global__ void __cluster_dims__(CLUSTER_BLOCKS, 1, 1) __launch_bounds__(CLUSTER_THREADS)
    radix_cluster_kernel(uint32_t *keys, uint32_t *vals, int n, int key_bits, int per) {
    namespace cg = cooperative_groups;
    constexpr int WARPS = CLUSTER_THREADS / 32;
    __shared__ uint32_t wcnt[WARPS][RADIX];
    __shared__ uint32_t counts[CLUSTER_BLOCKS][RADIX];  // every block's, by digit
    __shared__ uint32_t start[RADIX], ws[33];
    extern __shared__ __align__(16) unsigned char sort_smem[];  // per keys, per values
    uint32_t *skey = reinterpret_cast<uint32_t *>(sort_smem), *sval = skey + per;
    cg::cluster_group cluster = cg::this_cluster();
    const int me = (int)cluster.block_rank();
    const int lo = min(n, me * per), m = min(n, lo + per) - lo;  // this block's part
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int base = warp * KEYS * 32;  // the warp's keys lie side by side
    const unsigned lt = (1u << lane) - 1u;
    uint32_t key[KEYS], val[KEYS], rank[KEYS];
    cluster.sync();  // every block runs before its shared memory is written to
#pragma unroll
    for (int r = 0; r < KEYS; r++) {
        const int k = base + r * 32 + lane;
        if (k < m) {
            key[r] = keys[lo + k];
            val[r] = vals[lo + k];
        }
    }
    for (int shift = 0; shift < key_bits; shift += 8) {
        const uint32_t mask = key_bits - shift < 8 ? (1u << (key_bits - shift)) - 1u : 255u;
        for (int i = threadIdx.x; i < WARPS * RADIX; i += CLUSTER_THREADS) (&wcnt[0][0])[i] = 0;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < KEYS; r++) {
            const int k0 = base + r * 32;
            if (k0 >= m) continue;  // warp-uniform
            const bool ok = k0 + lane < m;
            const int d = ok ? (int)((key[r] >> shift) & mask) : RADIX;
            const unsigned peers = digit_peers(d, mask, k0 + 32 <= m);
            const uint32_t before = ok ? wcnt[warp][d] : 0u;
            rank[r] = before + (uint32_t)__popc(peers & lt);
            __syncwarp();
            if (ok && lane == __ffs(peers) - 1) wcnt[warp][d] = before + (uint32_t)__popc(peers);
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x < RADIX) {  // the warps' counts become prefixes; the sum goes to every block
            uint32_t c[WARPS], tot = 0;
#pragma unroll
            for (int w = 0; w < WARPS; w++) c[w] = wcnt[w][threadIdx.x];
#pragma unroll
            for (int w = 0; w < WARPS; w++) {
                wcnt[w][threadIdx.x] = tot;
                tot += c[w];
            }
            for (int q = 0; q < CLUSTER_BLOCKS; q++) *cluster.map_shared_rank(&counts[me][threadIdx.x], q) = tot;
        }
        cluster.sync();
        uint32_t all = 0, before = 0;
        if (threadIdx.x < RADIX)
            for (int q = 0; q < CLUSTER_BLOCKS; q++) {
                const uint32_t c = counts[q][threadIdx.x];
                all += c;
                if (q < me) before += c;
            }
        uint32_t total;
        const uint32_t ex = block_exclusive_scan<uint32_t>(all, ws, total) + before;
        if (threadIdx.x < RADIX) start[threadIdx.x] = ex;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < KEYS; r++) {
            if (base + r * 32 + lane >= m) continue;
            const int d = (int)((key[r] >> shift) & mask);
            const uint32_t p = start[d] + wcnt[warp][d] + rank[r];
            const uint32_t q = p / (uint32_t)per, i = p - q * (uint32_t)per;
            *cluster.map_shared_rank(skey + i, q) = key[r];
            *cluster.map_shared_rank(sval + i, q) = val[r];
        }
        cluster.sync();  // all keys have arrived; all blocks have read the counts
#pragma unroll
        for (int r = 0; r < KEYS; r++) {
            const int k = base + r * 32 + lane;
            if (k < m) {
                key[r] = skey[k];
                val[r] = sval[k];
            }
        }
    }
#pragma unroll
    for (int r = 0; r < KEYS; r++) {
        const int k = base + r * 32 + lane;
        if (k < m) {
            keys[lo + k] = key[r];
            vals[lo + k] = val[r];
        }
    }
}

template <int KEYS>
void radix_cluster_launch(uint32_t *keys, uint32_t *vals, int n, int key_bits, int per, cudaStream_t st) {
    static std::atomic<uint64_t> done{0};  // once per device: room for the largest part
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (!(done.load() & bit)) {
        cudaFuncSetAttribute(radix_cluster_kernel<KEYS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             CLUSTER_THREADS * KEYS * 8);
        done.fetch_or(bit);
    }
    radix_cluster_kernel<KEYS><<<CLUSTER_BLOCKS, CLUSTER_THREADS, (size_t)per * 8, st>>>(keys, vals, n, key_bits, per);
}

// Sorts (keys, vals) in place.
void radix_cluster_sort(uint32_t *keys, uint32_t *vals, int n, int key_bits, cudaStream_t st) {
    const int per = ((n + CLUSTER_BLOCKS - 1) / CLUSTER_BLOCKS + 31) / 32 * 32;
    if (per <= CLUSTER_THREADS * 2) radix_cluster_launch<2>(keys, vals, n, key_bits, per, st);
    else radix_cluster_launch<4>(keys, vals, n, key_bits, per, st);  // CLUSTER_SORT's at most
}

template <typename K, int THREADS, int ITEMS>
constexpr size_t radix_scatter_smem() {
    return (size_t)THREADS * ITEMS * (sizeof(K) + sizeof(uint32_t));
}

size_t radix_scratch_bytes(int n) {
    const int nb = radix_max_blocks(n > 1 ? n : 1);
    const size_t cnt = (size_t)RADIX * nb;
    return cnt * sizeof(int32_t) * 2 + (size_t)scan_blocks((int)cnt) * sizeof(int32_t) + 64;
}

// Sorts (k[0], v[0]) using (k[1], v[1]) as the ping-pong buffers; returns the index
// (0 or 1) of the buffer pair holding the result. With d_n, n is a capacity and the
// count is read on the device (no host round trip; every pass runs).
template <typename K, int THREADS, int ITEMS>
int radix_sort_impl(K *k[2], uint32_t *v[2], int n, int key_bits, void *scratch, cudaStream_t st, const int *d_n) {
    const int nb = (n + THREADS * ITEMS - 1) / (THREADS * ITEMS);
    const size_t cnt = (size_t)RADIX * nb;
    int32_t *counts = reinterpret_cast<int32_t *>(scratch);
    int32_t *offs = counts + cnt;
    int32_t *partials = offs + cnt;
    constexpr size_t smem = radix_scatter_smem<K, THREADS, ITEMS>();
    {  // once per device: the dynamic staging (with the static arrays it can pass the 48 KB
       // default)
        static std::atomic<uint64_t> done{0};
        int dev = 0;
        cudaGetDevice(&dev);
        const uint64_t bit = 1ull << (dev & 63);
        if (!(done.load() & bit)) {
            cudaFuncSetAttribute(radix_scatter_kernel<K, THREADS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
            done.fetch_or(bit);
        }
    }
    int cur = 0;
    for (int shift = 0; shift < key_bits; shift += 8) {
        const int bits = key_bits - shift < 8 ? key_bits - shift : 8;  // digits above key_bits are ignored
        const uint32_t mask = (1u << bits) - 1u;
        radix_hist_kernel<K, THREADS, ITEMS><<<nb, THREADS, 0, st>>>(k[cur], n, d_n, shift, mask,
                                                                     reinterpret_cast<uint32_t *>(counts), nb);
        const bool direct = nb <= DIRECT_SORT_BLOCKS;
        if (!direct) scan_exclusive<int32_t>(counts, offs, (int)cnt, nullptr, partials, st);
        radix_scatter_kernel<K, THREADS, ITEMS><<<nb, THREADS, smem, st>>>(
            k[cur], v[cur], k[cur ^ 1], v[cur ^ 1], n, d_n, shift, mask, direct ? nullptr : offs,
            reinterpret_cast<const uint32_t *>(counts), nb);
        cur ^= 1;
    }
    return cur;
}

template <typename K>
int radix_sort_dispatch(K *k[2], uint32_t *v[2], int n, int key_bits, void *scratch, cudaStream_t st, const int *d_n) {
    if ((!d_n && n <= 1) || n <= 0 || key_bits <= 0) return 0;
    if constexpr (sizeof(K) == 4) {
        if (!d_n && n <= CLUSTER_SORT) {
            radix_cluster_sort(k[0], v[0], n, key_bits, st);
            return 0;
        }
        if (n >= LARGE_SORT) return radix_sort_impl<K, 256, 16>(k, v, n, key_bits, scratch, st, d_n);
    }
    return radix_sort_impl<K, 256, 8>(k, v, n, key_bits, scratch, st, d_n);
}

int radix_sort_pairs(uint64_t *k[2], uint32_t *v[2], int n, int key_bits, void *scratch, cudaStream_t st,
                     const int *d_n) {
    return radix_sort_dispatch<uint64_t>(k, v, n, key_bits, scratch, st, d_n);
}

int radix_sort_pairs32(uint32_t *k[2], uint32_t *v[2], int n, int key_bits, void *scratch, cudaStream_t st,
                       const int *d_n) {
    return radix_sort_dispatch<uint32_t>(k, v, n, std::min(key_bits, 32), scratch, st, d_n);
}

}  // namespace msplat
