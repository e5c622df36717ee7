// Stable LSD radix sort for the sweep (sm_100a): onesweep passes with a
// decoupled look-back per digit.
//
// Keys are 32- or 64-bit, values optional 32-bit.  The item count and the
// number of key bits are read from device memory, and the buffer holding the
// result is recorded on the device (SortState::pass_info[kMaxPasses]), so a
// sort can be launched with host-side capacities only and captured in a CUDA
// graph.  Passes whose digit is the same for every key are skipped.
//
// Per pass and tile (kSortTile items): each warp ranks its items by the
// ballots of the digit's eight bits against a warp-private digit histogram in
// shared memory;
// thread d then publishes the tile's count of digit d, looks back over the
// preceding tiles' counts of d (status words stamped with a per-pass epoch,
// so the status area needs no clearing between sorts), and the tile is
// staged in shared memory in digit order before the coalesced scatter.
#pragma once

#include "pxr_common.cuh"

namespace pxr {

constexpr int kSortThreads = 256;
#ifndef PXR_SORT_ITEMS
#define PXR_SORT_ITEMS 16
#endif
constexpr int kSortItems = PXR_SORT_ITEMS;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kRadix = 256;
constexpr int kMaxPasses = 8;

// Tiles of `tile` items over count items.  Counts go up to 2^32 - 1 (both
// directions of 2^31 - 1 edges), where count + tile - 1 does not fit 32 bits.
__host__ __device__ constexpr uint32_t sort_tiles(uint32_t count, uint32_t tile) {
    return count / tile + (count % tile ? 1u : 0u);
}
static_assert(sort_tiles(0xFFFFFFFFu, 4096) == 1u << 20 && sort_tiles(0, 4096) == 0 && sort_tiles(4096, 4096) == 1 &&
                  sort_tiles(4097, 4096) == 2,
              "every item has a tile");

struct SortState {
    uint32_t* hist;       // [kMaxPasses][kRadix] digit counts (kept zero between sorts)
    uint32_t* bases;      // [kMaxPasses][kRadix] exclusive digit bases
    uint32_t* pass_info;  // [kMaxPasses + 1]: bit0 active, bit1 input buffer; [kMaxPasses]: result buffer
    uint32_t* tile_ctr;   // [kMaxPasses]
    uint32_t* epoch;      // [1]
    uint64_t* status;     // [max_tiles][kRadix]
    uint32_t max_tiles;
    unsigned long long* items_moved;  // optional: [0] += items x active passes, [1] += active passes
};

template <typename K>
struct SortBuffers {
    K* keys[2];
    uint32_t* vals[2];        // both null for keys-only sorts
    const uint32_t* count;    // device
    const uint32_t* end_bit;  // device: sort bits [0, end_bit)
    uint32_t capacity;        // host bound on *count
};

// ---------------------------------------------------------------------------

template <typename K>
__global__ void __launch_bounds__(kSortThreads) sort_histogram_kernel(SortBuffers<K> b, SortState s) {
    __shared__ uint32_t sh[kMaxPasses][kRadix];
    for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += blockDim.x) (&sh[0][0])[i] = 0;
    __syncthreads();
    const uint32_t count = *b.count;
    const uint32_t end_bit = *b.end_bit;
    const int npasses = (int)((end_bit + 7u) / 8u);
    const K* keys = b.keys[0];
    // 64-bit: within a stride of 2^32 a 32-bit index would start over and never end
    for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const K k = keys[i];
        for (int p = 0; p < npasses; ++p) atomicAdd(&sh[p][(uint32_t)(k >> (8 * p)) & 0xFFu], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npasses * kRadix; i += blockDim.x) {
        const uint32_t c = (&sh[0][0])[i];
        if (c) atomicAdd(&s.hist[i], c);
    }
}

// One block of kRadix threads: digit bases, pass activity, buffer parity,
// fresh epoch and tile counters; leaves the histogram zeroed.
template <typename K>
__global__ void __launch_bounds__(kRadix) sort_plan_kernel(SortBuffers<K> b, SortState s) {
    __shared__ uint64_t warp_tot[kRadix / 32];
    __shared__ uint32_t constant_digit;
    const uint32_t count = *b.count;
    const uint32_t end_bit = *b.end_bit;
    const int npasses = (int)((end_bit + 7u) / 8u);
    const uint32_t d = threadIdx.x;
    uint32_t parity = 0;
    for (int p = 0; p < kMaxPasses; ++p) {
        const uint32_t c = p < npasses ? s.hist[p * kRadix + d] : 0u;
        if (d == 0) constant_digit = 0;
        __syncthreads();
        if (c == count && count > 0) constant_digit = 1;
        uint64_t total;
        const uint64_t incl = block_inclusive<Add64>((uint64_t)c, warp_tot, &total);
        s.bases[p * kRadix + d] = (uint32_t)(incl - c);
        if (p < npasses) s.hist[p * kRadix + d] = 0;
        const bool active = p < npasses && count > 0 && !constant_digit;
        if (d == 0) s.pass_info[p] = (active ? 1u : 0u) | (parity << 1);
        if (active) parity ^= 1u;
        if (d == 0) s.tile_ctr[p] = 0;
        __syncthreads();
    }
    if (d == 0) {
        s.pass_info[kMaxPasses] = parity;
        *s.epoch = *s.epoch + kMaxPasses;
        uint32_t active = 0;
        for (int p = 0; p < kMaxPasses; ++p) active += s.pass_info[p] & 1u;
        if (s.items_moved) {
            s.items_moved[0] += (unsigned long long)count * active;
            s.items_moved[1] += active;
        }
    }
}

__device__ __forceinline__ uint64_t sort_status_word(uint32_t epoch, uint32_t flag, uint32_t cnt) {
    return ((uint64_t)((epoch << 2) | flag) << 32) | cnt;
}

// A predecessor tile's status word for this epoch, polled at most spin_limit
// times; when it never arrives the error bit is set and the stale word is
// returned.  Tile ids are taken in launch order, so a predecessor is always
// resident or done and the limit (about a second) is reached only if the
// protocol itself is broken; the host then reports PXR_DEVICE_FAULT.
__device__ __forceinline__ uint64_t wait_sort_status(const uint64_t* word, uint32_t epoch, uint32_t* err,
                                                     uint32_t spin_limit = kSpinLimit) {
    uint64_t w = ld_relaxed64(word);
    uint32_t spins = 0;
    while ((uint32_t)(w >> 34) != (epoch & 0x3FFFFFFFu) || ((w >> 32) & 3u) == 0u) {
        if (++spins > spin_limit) { atomicOr(err, kErrSortTiles); break; }
        __nanosleep(32);
        w = ld_relaxed64(word);
    }
    return w;
}

// 8-bit digit of a key at a bit position that is a multiple of 8.
__device__ __forceinline__ uint32_t sort_digit(uint32_t k, int shift) { return (k >> shift) & 0xFFu; }
__device__ __forceinline__ uint32_t sort_digit(uint64_t k, int shift) {
    const uint32_t w = shift < 32 ? (uint32_t)k : (uint32_t)(k >> 32);
    return (w >> (shift & 31)) & 0xFFu;
}

#ifndef PXR_SORT_MIN_BLOCKS
#define PXR_SORT_MIN_BLOCKS 2
#endif
// One digit pass.  ITEMS keys per thread (tile = 256 ITEMS) and the CTAs per
// SM the register budget is sized for (MINB) are the sort plan's two axes
// (pxr_sort_plan); every plan gives the same output, item for item.
template <typename K, int ITEMS = kSortItems, int MINB = PXR_SORT_MIN_BLOCKS>
__global__ void __launch_bounds__(kSortThreads, MINB) sort_pass_kernel(SortBuffers<K> b, SortState s, int pass,
                                                                       uint32_t* err) {
    constexpr int kSortItems = ITEMS;
    constexpr int kSortTile = kSortThreads * ITEMS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K* skeys = reinterpret_cast<K*>(smem_raw);
    uint32_t* svals = reinterpret_cast<uint32_t*>(skeys + kSortTile);
    uint32_t (*whist)[kRadix] = reinterpret_cast<uint32_t (*)[kRadix]>(svals + kSortTile);
    __shared__ uint32_t gbase[kRadix];
    __shared__ uint64_t warp_tot[kSortThreads / 32];
    __shared__ uint32_t s_tile;

    const uint32_t info = s.pass_info[pass];
    if (!(info & 1u)) return;
    const int in = (info >> 1) & 1;
    // selects, not indexing: a parameter array indexed at run time is copied to local memory
    const K* kin = in ? b.keys[1] : b.keys[0];
    K* kout = in ? b.keys[0] : b.keys[1];
    const uint32_t* vin = in ? b.vals[1] : b.vals[0];
    uint32_t* vout = in ? b.vals[0] : b.vals[1];
    const bool has_vals = vin != nullptr;
    const uint32_t count = *b.count;
    const uint32_t num_tiles = sort_tiles(count, kSortTile);
    const uint32_t epoch = *s.epoch + (uint32_t)pass;
    const int shift = 8 * pass;

    if (threadIdx.x == 0) s_tile = atomicAdd(&s.tile_ctr[pass], 1u);
    for (int i = threadIdx.x; i < (kSortThreads / 32) * kRadix; i += kSortThreads) (&whist[0][0])[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= num_tiles) return;

    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t in_warp = warp * (32 * kSortItems);   // the warp's first place in the tile
    const uint32_t base = tile * kSortTile + in_warp;
    const uint32_t tile_items = min((uint32_t)kSortTile, count - tile * kSortTile);
    const bool full = tile_items == (uint32_t)kSortTile;   // all but the last tile skip the bounds tests
    K key[kSortItems];
    uint32_t val[kSortItems];
    if (full) {
#pragma unroll
        for (int k = 0; k < kSortItems; ++k) key[k] = kin[base + k * 32 + lane];
#pragma unroll
        for (int k = 0; k < kSortItems; ++k) val[k] = has_vals ? vin[base + k * 32 + lane] : 0u;
    } else {
#pragma unroll
        for (int k = 0; k < kSortItems; ++k) {
            const uint32_t idx = base + k * 32 + lane;
            const bool valid = in_warp + k * 32 + lane < tile_items;
            key[k] = valid ? kin[idx] : (K)0;
            val[k] = (valid && has_vals) ? vin[idx] : 0u;
        }
    }
    // Lanes of the same digit, for every item at once: the ballots of
    // different items are independent, where one __match_any_sync per item,
    // each ahead of its shared-memory count, was a serial chain.  What bounds a
    // pass is latency (ranking about 6,000 of a tile's 27,000 cycles, the
    // look-back 7,500, the scatter 7,500), not bandwidth.  Whole sorts under
    // plans 0 / 1 / 2, before and after: 16.7 M pairs, four digits 958 / 892 /
    // 949 -> 830 / 806 / 862 us; 4.2 M 296 / 282 / 282 -> 257 / 255 / 259; 67 M
    // keys without values, six digits 4.86 / 4.49 / 5.05 -> 4.33 / 4.18 / 4.59 ms.
    // (Measured and not taken: looking back 4 or 8 tiles at once, a warp of its
    // own for the look-back, and counting in a kernel of its own instead of the
    // look-back: slower below 16 M items.)
    const uint32_t lt = lanemask_lt();
    uint32_t rank[kSortItems];   // the item's peers, then its place in the warp's digit run
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t d = sort_digit(key[k], shift);
        uint32_t peers = 0xFFFFFFFFu;
        if (!full) {
            const bool valid = in_warp + k * 32 + lane < tile_items;
            const uint32_t in_range = __ballot_sync(0xFFFFFFFFu, valid);
            peers = valid ? in_range : ~in_range;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t set = __ballot_sync(0xFFFFFFFFu, (d >> q) & 1u);
            peers &= (d >> q) & 1u ? set : ~set;
        }
        rank[k] = peers;
    }
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const bool valid = full || in_warp + k * 32 + lane < tile_items;
        const uint32_t d = sort_digit(key[k], shift);
        const uint32_t peers = rank[k];
        // every lane reads its digit's count (peers read one word), the first peer advances it
        const uint32_t before = valid ? whist[warp][d] : 0u;
        __syncwarp();
        if (valid && (peers & lt) == 0u) whist[warp][d] = before + __popc(peers);
        __syncwarp();
        rank[k] = before + __popc(peers & lt);
    }
    __syncthreads();

    // digit d = threadIdx.x: per-warp exclusive offsets, tile count, look-back
    const uint32_t d = threadIdx.x;
    uint32_t tile_cnt = 0;
#pragma unroll
    for (int w = 0; w < kSortThreads / 32; ++w) {
        const uint32_t c = whist[w][d];
        whist[w][d] = tile_cnt;
        tile_cnt += c;
    }
    // a status word carries its own count, so relaxed accesses suffice (no fences)
    uint64_t* st = s.status + (size_t)tile * kRadix + d;
    st_relaxed64(st, sort_status_word(epoch, 1u, tile_cnt));
    uint32_t excl = 0;
    for (int32_t t = (int32_t)tile - 1; t >= 0; --t) {
        const uint64_t w = wait_sort_status(s.status + (size_t)t * kRadix + d, epoch, err);
        excl += (uint32_t)w;
        if (((w >> 32) & 3u) == 2u) break;
    }
    st_relaxed64(st, sort_status_word(epoch, 2u, excl + tile_cnt));
    uint64_t total;
    const uint64_t incl = block_inclusive<Add64>((uint64_t)tile_cnt, warp_tot, &total);
    const uint32_t in_tile = (uint32_t)incl - tile_cnt;   // the digit's first place in the tile
    gbase[d] = s.bases[pass * kRadix + d] + excl - in_tile;
#pragma unroll
    for (int w = 0; w < kSortThreads / 32; ++w) whist[w][d] += in_tile;
    __syncthreads();

#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        if (full || in_warp + k * 32 + lane < tile_items) {
            const uint32_t pos = whist[warp][sort_digit(key[k], shift)] + rank[k];
            skeys[pos] = key[k];
            svals[pos] = val[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kSortItems; ++q) {
        const uint32_t j = threadIdx.x + q * kSortThreads;
        if (full || j < tile_items) {
            const K kk = skeys[j];
            const uint32_t out = gbase[sort_digit(kk, shift)] + j;
            kout[out] = kk;
            if (has_vals) vout[out] = svals[j];
        }
    }
}

template <typename K, int ITEMS = kSortItems>
constexpr size_t sort_pass_smem() {
    return (sizeof(K) + sizeof(uint32_t)) * kSortThreads * ITEMS + sizeof(uint32_t) * (kSortThreads / 32) * kRadix;
}

// Sort plans (items per thread, CTAs per SM) the tuner chooses from; plan 0
// is the default.  The smallest tile sets how many tile status words a sort
// may need (kSortMinTile).
struct SortPlanEntry { int items, ctas; };
constexpr SortPlanEntry kSortPlans[3] = {{16, 2}, {12, 3}, {8, 4}};
constexpr int kSortPlanCount = 3;
constexpr int kSortMinTile = kSortThreads * 8;

template <typename K, int ITEMS, int MINB>
inline void launch_sort_passes(const SortBuffers<K>& b, const SortState& s, uint32_t* err, cudaStream_t stream,
                               int npasses) {
    const uint32_t tiles = sort_tiles(b.capacity, kSortThreads * ITEMS);
    for (int p = 0; p < npasses; ++p)
        sort_pass_kernel<K, ITEMS, MINB><<<tiles, kSortThreads, sort_pass_smem<K, ITEMS>(), stream>>>(b, s, p, err);
}

// Launch a full sort on `stream` with sort plan `plan` (index into
// kSortPlans).  After it, s.pass_info[kMaxPasses] on the device names the
// buffer (0/1) holding the sorted keys and values.
template <typename K>
inline cudaError_t radix_sort(const SortBuffers<K>& b, const SortState& s, uint32_t* err, cudaStream_t stream,
                              int max_end_bit, int plan = 0) {
    if (b.capacity == 0) return cudaSuccess;
    const uint32_t tiles = sort_tiles(b.capacity, kSortTile);
    const uint32_t hgrid = min(tiles * 4u, 148u * 8u);
    sort_histogram_kernel<K><<<hgrid, kSortThreads, 0, stream>>>(b, s);
    sort_plan_kernel<K><<<1, kRadix, 0, stream>>>(b, s);
    const int npasses = (max_end_bit + 7) / 8;
    switch (plan) {
        case 1: launch_sort_passes<K, 12, 3>(b, s, err, stream, npasses); break;
        case 2: launch_sort_passes<K, 8, 4>(b, s, err, stream, npasses); break;
        default: launch_sort_passes<K, 16, PXR_SORT_MIN_BLOCKS>(b, s, err, stream, npasses); break;
    }
    return cudaGetLastError();
}

template <typename K>
inline cudaError_t radix_sort_prepare() {
    cudaError_t e = cudaFuncSetAttribute(sort_pass_kernel<K, 16, PXR_SORT_MIN_BLOCKS>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_pass_smem<K, 16>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sort_pass_kernel<K, 12, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sort_pass_smem<K, 12>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sort_pass_kernel<K, 8, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sort_pass_smem<K, 8>());
    return e;
}

}  // namespace pxr
