// radix_sort.cu -- onesweep LSD radix sort (see radix_sort.cuh).
#include "radix_sort.cuh"
#include "common.cuh"
#include "errors.h"

namespace sph {

namespace {

constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPfx = 2u << 30;
constexpr uint32_t kValMask = (1u << 30) - 1u;
constexpr int kWarps = kSortThreads / 32;
// Bounded look-back: about 0.1 s of polling with nanosleep back-off before a
// tile gives up (a predecessor that is resident never needs that long).
constexpr int kSpinLimit = 1 << 20;
constexpr int kSpinLimitForced = 64;
constexpr int kLookAhead = 8;

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Exclusive scans of two values per thread over a 256-thread block.
__device__ __forceinline__ uint2 block_exclusive_scan2(uint32_t v, uint32_t w, uint2* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v, z = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o), u = __shfl_up_sync(0xFFFFFFFFu, z, o);
        if (lane >= o) {
            x += y;
            z += u;
        }
    }
    if (lane == 31) s_warp[warp] = make_uint2(x, z);
    __syncthreads();
    uint32_t xp = 0, zp = 0;
#pragma unroll
    for (int k = 0; k < kWarps; ++k)
        if (k < warp) {
            xp += s_warp[k].x;
            zp += s_warp[k].y;
        }
    return make_uint2(xp + x - v, zp + z - w);
}

__global__ void __launch_bounds__(256) histogram_kernel(const uint32_t* __restrict__ keys,
                                                        uint32_t n, int passes,
                                                        uint32_t* __restrict__ hist) {
    __shared__ uint32_t sh[kSortMaxPasses][256];
    for (int i = threadIdx.x; i < kSortMaxPasses * 256; i += blockDim.x) (&sh[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        sort_hist_add(sh, keys[i], passes);
    __syncthreads();
    for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) {
        uint32_t c = (&sh[0][0])[i];
        if (c) atomicAdd(&hist[i], c);
    }
}

__global__ void __launch_bounds__(kSortThreads) onesweep_kernel(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
    uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n,
    const uint32_t* __restrict__ n_dev, uint32_t small_max, int items, int shift,
    const uint32_t* __restrict__ hist, uint32_t* status, uint32_t* tile_ctr,
    uint32_t* err, int force_timeout) {
    __shared__ uint32_t s_keys[kSortTile];
    __shared__ uint32_t s_vals[kSortTile];
    __shared__ uint32_t s_whist[kWarps][257];  // column 256 collects out-of-range items
    __shared__ uint32_t s_local_start[256];
    __shared__ uint32_t s_gbase[256];
    __shared__ uint2 s_warp[kWarps];
    __shared__ uint32_t s_tile;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    grid_wait();
    if (n_dev) n = min(*after_wait(n_dev), n);  // key count known on the device only: the grid covers n keys
    if (n == 0) return;
    const int ni = n_dev && n <= small_max ? kSortItemsSmall : items;  // keys per thread
    const uint32_t tile_keys = (uint32_t)ni * kSortThreads;
    if (tid == 0) s_tile = atomicAdd(tile_ctr, 1u);
    for (int i = tid; i < kWarps * 257; i += kSortThreads) (&s_whist[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t base = tile * tile_keys;
    if (base >= n) return;  // tiles are handed out in order: no later tile waits on this one
    const uint32_t seg = base + (uint32_t)warp * ((uint32_t)ni * 32);
    const uint32_t digit_total = after_wait(hist)[tid];

    uint32_t k[kSortItems], v[kSortItems], rank[kSortItems];
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        uint32_t idx = seg + i * 32 + lane;
        bool ok = i < ni && idx < n;
        k[i] = ok ? keys_in[idx] : 0xFFFFFFFFu;
        v[i] = ok ? (vals_in ? vals_in[idx] : idx) : 0u;
    }

    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        if (i >= ni) break;
        uint32_t idx = seg + i * 32 + lane;
        uint32_t d = idx < n ? ((k[i] >> shift) & 255u) : 256u;
        uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
        int leader = 31 - __clz(peers);
        uint32_t b = s_whist[warp][d];
        rank[i] = b + __popc(peers & lt);
        __syncwarp();
        if (lane == leader) s_whist[warp][d] = b + __popc(peers);
        __syncwarp();
    }
    __syncthreads();

    // Thread t owns digit t: exclusive offsets across warps and the tile total.
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        uint32_t c = s_whist[w][tid];
        s_whist[w][tid] = total;
        total += c;
    }
    uint32_t* my_status = status + (size_t)tile * 256 + tid;
    st_relaxed(my_status, (tile == 0 ? kFlagPfx : kFlagAgg) | total);

    // every tile scans the digit histogram itself, beside its own counts: a kernel
    // for it cost a launch of its own in the chain
    const uint2 start = block_exclusive_scan2(total, digit_total, s_warp);
    const uint32_t local_start = start.x;
    s_local_start[tid] = local_start;

    uint32_t prefix = 0;
    if (tile > 0) {
        // kLookAhead predecessors' words are loaded together: tiles that start at
        // the same time each walk back to the first, and one word after the other
        // that was most of a pass's time (94,608 keys in 24 tiles, three passes: 95.5
        // -> 94.1 us per step; 16 together load more than they save)
        int pred = (int)tile - 1;
        int spins = 0;
        const int limit = force_timeout ? kSpinLimitForced : kSpinLimit;
        bool done = false;
        while (!done && pred >= 0) {
            uint32_t sv[kLookAhead];
#pragma unroll
            for (int u = 0; u < kLookAhead; ++u)
                sv[u] = force_timeout ? 0u
                                      : ld_relaxed(status + (size_t)max(pred - u, 0) * 256 + tid);
            int used = 0;
#pragma unroll
            for (int u = 0; u < kLookAhead; ++u) {
                const uint32_t flag = sv[u] & ~kValMask;
                if (done || used != u || flag == 0u || pred - u < 0) continue;
                prefix += sv[u] & kValMask;
                done = flag == kFlagPfx;
                used = u + 1;
            }
            pred -= used;
            if (used == 0) {
                if (++spins > limit) {
                    atomicOr(err, 1u);
                    break;
                }
                __nanosleep(64);
            }
        }
        st_relaxed(my_status, kFlagPfx | ((prefix + total) & kValMask));
    }
    s_gbase[tid] = start.y + prefix - local_start;
    __syncthreads();

#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        uint32_t idx = seg + i * 32 + lane;
        if (i < ni && idx < n) {
            uint32_t d = (k[i] >> shift) & 255u;
            uint32_t pos = s_local_start[d] + s_whist[warp][d] + rank[i];
            s_keys[pos] = k[i];
            s_vals[pos] = v[i];
        }
    }
    __syncthreads();

    const uint32_t tile_n = (n - base) < tile_keys ? (n - base) : tile_keys;
    for (uint32_t i = tid; i < tile_n; i += kSortThreads) {
        uint32_t key = s_keys[i];
        uint32_t g = s_gbase[(key >> shift) & 255u] + i;
        if (g < n) {
            keys_out[g] = key;
            vals_out[g] = s_vals[i];
        }
    }
}

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

SortScratch sort_scratch_from(void* base, uint32_t max_n) {
    SortScratch s;
    uint32_t tiles = (max_n + kSortTile - 1) / kSortTile;
    if (tiles == 0) tiles = 1;
    char* p = (char*)base;
    s.hist = (uint32_t*)p;
    p += align256(kSortMaxPasses * 256 * 4);
    s.tile_ctr = (uint32_t*)p;
    p += align256(kSortMaxPasses * 4);
    s.status = (uint32_t*)p;
    p += align256((size_t)kSortMaxPasses * tiles * 256 * 4);
    s.zero_bytes = (size_t)(p - (char*)base);
    return s;
}

void sort_reset(const SortScratch& s, cudaStream_t st) {
    cudaMemsetAsync(s.hist, 0, s.zero_bytes, st);
}

void sort_histogram(const uint32_t* keys, uint32_t n, int passes, const SortScratch& s,
                    cudaStream_t st) {
    if (n == 0) return;
    uint32_t blocks = (n + 255) / 256;
    if (blocks > 152 * 4) blocks = 152 * 4;
    histogram_kernel<<<blocks, 256, 0, st>>>(keys, n, passes, s.hist);
}

void sort_pass(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
               uint32_t* vals_out, uint32_t n, int p, const SortScratch& s, uint32_t* err,
               int force_timeout, cudaStream_t st) {
    if (n == 0) return;
    uint32_t tiles = (n + kSortTile - 1) / kSortTile;
    onesweep_kernel<<<tiles, kSortThreads, 0, st>>>(
        keys_in, vals_in, keys_out, vals_out, n, nullptr, 0u, kSortItems, 8 * p, s.hist + p * 256,
        s.status + (size_t)p * tiles * 256, s.tile_ctr + p, err, force_timeout);
}

uint32_t sort_tiles(uint32_t n, uint32_t small_max) {
    const uint32_t tiles = (n + kSortTile - 1) / kSortTile;
    const uint32_t few = n < small_max ? n : small_max;
    const uint32_t small_tiles = (few + kSortTileSmall - 1) / kSortTileSmall;
    return small_tiles > tiles ? small_tiles : tiles;
}

namespace {

int passes_run(uint32_t* keys[2], uint32_t* vals[2], const uint32_t* first_vals, uint32_t n,
               const uint32_t* n_dev, uint32_t small_max, int items, uint32_t tiles, int passes,
               const SortScratch& s, uint32_t* err, int force_timeout, cudaStream_t st) {
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        const uint32_t* vin = (p == 0) ? first_vals : vals[cur];
        launch_after(onesweep_kernel, tiles, kSortThreads, st, keys[cur], vin, keys[cur ^ 1],
                     vals[cur ^ 1], n, n_dev, small_max, items, 8 * p, s.hist + p * 256,
                     s.status + (size_t)p * tiles * 256, s.tile_ctr + p, err, force_timeout);
        cur ^= 1;
    }
    return cur;
}

}  // namespace

int sort_passes_run_dev(uint32_t* keys[2], uint32_t* vals[2], const uint32_t* first_vals,
                        uint32_t n, const uint32_t* n_dev, uint32_t small_max, int passes,
                        const SortScratch& s, uint32_t* err, int force_timeout, cudaStream_t st) {
    if (n == 0) return 0;
    return passes_run(keys, vals, first_vals, n, n_dev, small_max, kSortItems,
                      sort_tiles(n, small_max), passes, s, err, force_timeout, st);
}

int sort_passes_run(uint32_t* keys[2], uint32_t* vals[2], const uint32_t* first_vals, uint32_t n,
                    int passes, const SortScratch& s, uint32_t* err, int force_timeout,
                    cudaStream_t st) {
    if (n == 0) return 0;
    return passes_run(keys, vals, first_vals, n, nullptr, 0u, kSortItems,
                      (n + kSortTile - 1) / kSortTile, passes, s, err, force_timeout, st);
}

int sort_step_run(uint32_t* keys[2], uint32_t* vals[2], uint32_t n, int passes,
                  const SortScratch& s, uint32_t* err, int force_timeout, cudaStream_t st) {
    if (n == 0) return 0;
    const int items = sort_step_items(n);
    const uint32_t tile = (uint32_t)(kSortThreads * items);
    return passes_run(keys, vals, nullptr, n, nullptr, 0u, items, (n + tile - 1) / tile, passes, s,
                      err, force_timeout, st);
}

int sort_pairs(uint32_t* keys[2], uint32_t* vals[2], uint32_t n, int key_bits,
               const SortScratch& s, uint32_t* err, int force_timeout, cudaStream_t st) {
    int passes = sort_passes(key_bits);
    sort_reset(s, st);
    sort_histogram(keys[0], n, passes, s, st);
    return sort_passes_run(keys, vals, vals[0], n, passes, s, err, force_timeout, st);
}

}  // namespace sph
