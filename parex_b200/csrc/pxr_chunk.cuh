// Chunked sweep sort (sm_100a): the sort of a round done CTA by CTA in
// shared memory, when every cluster of the previous round is small.
//
// The active list is in the previous round's sort order with deactivated
// vertices removed, so the vertices of each previous-round cluster (a
// "parent") form one contiguous run of it, and every cluster of this round
// lies inside one parent's run.  When every parent holds at most CAP
// vertices, chunk k takes the parents whose run starts in
// [k * ROWS, (k + 1) * ROWS) - at most ROWS + CAP - 1 items -
// sorts them stably by (label, potential) with an LSD radix sort in shared
// memory, and writes every cluster to its start position from the cluster
// tables.  The result is the global stable sort's, item for item: the same
// key, the same tie order (the active list's order), the same positions.
// Rounds with larger parents use the global onesweep sort.
#pragma once

#include "pxr_kernels.cuh"

namespace pxr {

// A chunk's shape: ROWS list positions whose parents it takes, CAP the longest
// parent, THREADS a CTA's threads.
template <uint32_t ROWS, uint32_t CAP, int THREADS>
struct ChunkShape {
    static constexpr uint32_t kRows = ROWS;
    static constexpr uint32_t kItems = ROWS + CAP;
    static constexpr int kThreads = THREADS;
    static constexpr int kIpt = (int)kItems / THREADS;      // items per thread
    static constexpr int kWarps = THREADS / 32;
    static constexpr uint32_t kSlots = 2 * kItems;          // label hash table (in the second key buffer)
    static constexpr size_t kSmem = 2 * kItems * sizeof(uint64_t) + 2 * kItems * sizeof(uint32_t) +
                                    kWarps * 256 * sizeof(uint32_t);
};
// One CTA per SM while clusters of thousands of vertices remain; then chunks of
// a quarter of the size, three CTAs per SM: what bounds a chunk is its own chain
// of gathers, scans and barriers (36 us whatever the list's length), so several
// per SM hide it (sorts of the 128^3 grid 5.6 -> 5.0 ms, its decomposition 20.6 ->
// 19.8; 64^3 7.1 -> 6.8; two or four CTAs per SM within 1 %).
using LargeChunk = ChunkShape<4096, kChunkCapRows, 512>;
using SmallChunk = ChunkShape<1024, kChunkCapSmall, 256>;
// Direct ranking (comparisons within a parent run) is used when no parent
// run of the chunk is longer than this.
constexpr uint32_t kCountRun = 512;

// first p >= p0 where a parent run starts (p == 0, or the parent changes), else n
template <class C>
__device__ __forceinline__ uint32_t chunk_boundary(const uint32_t* par, uint32_t p0, uint32_t n, uint32_t* s_min) {
    if (p0 == 0) return 0;
    if (p0 >= n) return n;
    for (uint32_t base = p0; base < n; base += C::kThreads) {
        if (threadIdx.x == 0) *s_min = n;
        __syncthreads();
        const uint32_t p = base + threadIdx.x;
        if (p < n && par[p] != par[p - 1]) atomicMin(s_min, p);
        __syncthreads();
        const uint32_t found = *s_min;
        __syncthreads();
        if (found < n) return found;
    }
    return n;
}

// One stable LSD pass over cnt items (8-bit digit at `shift`), src -> dst.
template <class C>
__device__ __forceinline__ void chunk_pass(const uint64_t* sk, const uint32_t* sv, uint64_t* dk, uint32_t* dv,
                                           uint32_t cnt, int shift, uint32_t (*whist)[256], uint32_t* tpre) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lt = lanemask_lt();
    for (int i = lane; i < 256; i += 32) whist[warp][i] = 0;
    __syncwarp();
    const uint32_t base = warp * (32 * C::kIpt);
    uint32_t dg[C::kIpt], rank[C::kIpt];
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) {
        const uint32_t j = base + k * 32 + lane;
        dg[k] = j < cnt ? ((uint32_t)(sk[j] >> shift) & 0xFFu) : 0x100u;
    }
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) {
        const bool valid = dg[k] < 0x100u;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, dg[k]);
        // the lowest lane of each digit reads and advances the warp's count
        const uint32_t leader = (uint32_t)__ffs(peers) - 1u;
        uint32_t before = 0;
        if (valid && lane == leader) {
            before = whist[warp][dg[k]];
            whist[warp][dg[k]] = before + __popc(peers);
        }
        before = __shfl_sync(0xFFFFFFFFu, before, leader);
        rank[k] = before + __popc(peers & lt);
        __syncwarp();
    }
    __syncthreads();
    // digit d: offsets of the warps, then the block's exclusive digit prefix
    if (threadIdx.x < 256) {
        const uint32_t d = threadIdx.x;
        uint32_t tot = 0;
#pragma unroll
        for (int w = 0; w < C::kWarps; ++w) {
            const uint32_t c = whist[w][d];
            whist[w][d] = tot;
            tot += c;
        }
        tpre[d] = tot;
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // exclusive scan of 256 digit totals by one warp (8 per lane)
        uint32_t v[8], sum = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) { v[q] = tpre[threadIdx.x * 8 + q]; sum += v[q]; }
        uint32_t inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (threadIdx.x >= (uint32_t)o) inc += u;
        }
        uint32_t run = inc - sum;
#pragma unroll
        for (int q = 0; q < 8; ++q) { tpre[threadIdx.x * 8 + q] = run; run += v[q]; }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) {
        const uint32_t j = base + k * 32 + lane;
        if (dg[k] < 0x100u) {
            const uint32_t pos = tpre[dg[k]] + whist[warp][dg[k]] + rank[k];
            dk[pos] = sk[j];
            dv[pos] = sv[j];
        }
    }
    __syncthreads();
}

template <class C, typename OffT>
__device__ __forceinline__ void chunk_one(const Dev<OffT>& d, const ClusterTables& t, const uint32_t* act,
                                          const uint32_t* par, uint64_t* keys_out, uint32_t* vals_out, uint32_t lo,
                                          uint32_t n, uint64_t* ka, uint64_t* kb, uint32_t* va, uint32_t* vb,
                                          uint32_t (*whist)[256], uint32_t* tpre, uint32_t* sh, uint32_t* s_min_p,
                                          uint32_t* s_and_p, uint32_t* s_or_p) {
    uint32_t& s_min = *s_min_p;
    uint32_t& s_and = *s_and_p;
    uint32_t& s_or = *s_or_p;
    uint32_t* table = reinterpret_cast<uint32_t*>(kb);   // label hash table until the first pass
    const uint32_t begin = chunk_boundary<C>(par, lo, n, &s_min);
    const uint32_t end = chunk_boundary<C>(par, lo + C::kRows, n, &s_min);
    if (begin >= end) return;
    const uint32_t cnt = end - begin;
    if (cnt > C::kItems) {   // a parent longer than the shape's cap: the path was chosen wrongly
        if (threadIdx.x == 0) atomicOr(&d.ctr->err, kErrLabelRange);
        return;
    }
    if (threadIdx.x == 0) { s_and = 0xFFFFFFFFu; s_or = 0u; }
    // gathers: every load of a thread in flight together
    uint32_t v[C::kIpt], L[C::kIpt], xo[C::kIpt];
#pragma unroll
    for (int r = 0; r < C::kIpt; ++r) {
        const uint32_t j = threadIdx.x + r * C::kThreads;
        v[r] = j < cnt ? act[begin + j] : 0u;
    }
#pragma unroll
    for (int r = 0; r < C::kIpt; ++r) {
        const uint32_t j = threadIdx.x + r * C::kThreads;
        L[r] = j < cnt ? (uint32_t)d.lab[v[r]] : 0u;
        xo[r] = j < cnt ? ordered_bits(d.x[v[r]]) : 0u;
    }
    // Short parent runs: rank every vertex directly among the vertices of its
    // run with the same label (earlier by potential, ties by list position),
    // which is its place in the stable sort.  Work: sum of squared run lengths.
#pragma unroll
    for (int r = 0; r < C::kIpt; ++r) {
        const uint32_t j = threadIdx.x + r * C::kThreads;
        if (j < cnt) {
            ka[j] = ((uint64_t)L[r] << 32) | xo[r];
            va[j] = v[r];
            vb[j] = par[begin + j];
        }
    }
    __syncthreads();
    // parent runs by block scans over a contiguous layout (16 items per thread):
    // run start = last head at or before i, run end = first head after i
    const uint32_t c0 = threadIdx.x * C::kIpt;
    uint32_t rs[C::kIpt], re[C::kIpt];
    uint32_t last = 0;
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) {
        const uint32_t i = c0 + k;
        if (i < cnt && (i == 0 || vb[i] != vb[i - 1])) last = i;
        rs[k] = last;
    }
    uint32_t first = cnt;   // first head after this thread's items, from the right
#pragma unroll
    for (int k = C::kIpt - 1; k >= 0; --k) {
        const uint32_t i = c0 + k;
        re[k] = first;
        if (i < cnt && (i == 0 || vb[i] != vb[i - 1])) first = i;
    }
    // carries: max of earlier threads' last heads, min of later threads' first heads
    uint32_t mx = last, mn = first;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, mx, o);
        const uint32_t w = __shfl_down_sync(0xFFFFFFFFu, mn, o);
        if ((threadIdx.x & 31u) >= (uint32_t)o) mx = max(mx, u);
        if ((threadIdx.x & 31u) + o < 32u) mn = min(mn, w);
    }
    __syncthreads();
    if ((threadIdx.x & 31u) == 31u) tpre[threadIdx.x >> 5] = mx;           // warp's max head
    if ((threadIdx.x & 31u) == 0u) tpre[32 + (threadIdx.x >> 5)] = mn;      // warp's min first head
    __syncthreads();
    uint32_t before_max = __shfl_up_sync(0xFFFFFFFFu, mx, 1);
    if ((threadIdx.x & 31u) == 0) before_max = 0;
    uint32_t after_min = __shfl_down_sync(0xFFFFFFFFu, mn, 1);
    if ((threadIdx.x & 31u) == 31u) after_min = cnt;
    for (uint32_t w = 0; w < (threadIdx.x >> 5); ++w) before_max = max(before_max, tpre[w]);
    for (uint32_t w = (threadIdx.x >> 5) + 1; w < (uint32_t)C::kWarps; ++w) after_min = min(after_min, tpre[32 + w]);
    uint32_t longest = 0;
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) {
        const uint32_t i = c0 + k;
        rs[k] = max(rs[k], before_max);
        if (i >= cnt) continue;
        re[k] = min(re[k], after_min);
        longest = max(longest, re[k] - rs[k]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(0xFFFFFFFFu, longest, o));
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) sh[threadIdx.x >> 5] = longest;
    __syncthreads();
    uint32_t run_max = 0;
    for (int w = 0; w < C::kWarps; ++w) run_max = max(run_max, sh[w]);
    __syncthreads();
    if (run_max <= kCountRun) {
        // run bounds to shared memory (the second key buffer is free on this
        // path), then neighbouring lanes rank neighbouring items: the lanes
        // of a warp read the same run, so the reads are broadcasts
        uint32_t* srs = reinterpret_cast<uint32_t*>(kb);
        uint32_t* sre = srs + C::kItems;
#pragma unroll
        for (int k = 0; k < C::kIpt; ++k)
            if (c0 + k < cnt) { srs[c0 + k] = rs[k]; sre[c0 + k] = re[k]; }
        __syncthreads();
#pragma unroll 1
        for (int k = 0; k < C::kIpt; ++k) {
            const uint32_t i = threadIdx.x + k * C::kThreads;
            if (i >= cnt) break;
            const uint64_t ki = ka[i];
            const uint32_t li = (uint32_t)(ki >> 32), xi = (uint32_t)ki;
            const uint32_t jb = srs[i], je = sre[i];
            uint32_t rank = 0;
            for (uint32_t j = jb; j < je; ++j) {
                const uint64_t kj = ka[j];
                const uint32_t xj = (uint32_t)kj;
                rank += ((uint32_t)(kj >> 32) == li && (xj < xi || (xj == xi && j < i))) ? 1u : 0u;
            }
            const uint32_t pos = t.start[li] + rank;
            keys_out[pos] = ki;
            vals_out[pos] = va[i];
        }
        return;
    }
    for (uint32_t q = threadIdx.x; q < C::kSlots; q += C::kThreads) table[q] = 0xFFFFFFFFu;
    __syncthreads();
    // local cluster slot: the label's place in a hash table (injective; the
    // order of clusters inside a chunk is irrelevant, positions come from
    // the cluster starts)
    uint32_t slot[C::kIpt];
    uint32_t a = 0xFFFFFFFFu, o = 0u;
#pragma unroll
    for (int r = 0; r < C::kIpt; ++r) {
        const uint32_t j = threadIdx.x + r * C::kThreads;
        const bool valid = j < cnt;
        if (valid) {
            a &= xo[r];
            o |= xo[r];
        }
        // one insertion per distinct label of the warp (the lanes of a
        // cluster would otherwise serialise on one slot)
        const uint32_t key = valid ? L[r] : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
        const int leader = __ffs(peers) - 1;
        uint32_t h = ((key * 2654435761u) >> 16) & (C::kSlots - 1);
        if (valid && (int)(threadIdx.x & 31u) == leader) {
            for (uint32_t probe = 0; probe < C::kSlots; ++probe) {
                const uint32_t prev = atomicCAS(&table[h], 0xFFFFFFFFu, key);
                if (prev == 0xFFFFFFFFu || prev == key) break;
                h = (h + 1) & (C::kSlots - 1);
            }
        }
        slot[r] = __shfl_sync(0xFFFFFFFFu, h, leader);
    }
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) {
        a &= __shfl_xor_sync(0xFFFFFFFFu, a, q);
        o |= __shfl_xor_sync(0xFFFFFFFFu, o, q);
    }
    if ((threadIdx.x & 31u) == 0) { atomicAnd(&s_and, a); atomicOr(&s_or, o); }
    __syncthreads();
    // dense local ids: rank of the occupied slots (32 slots per thread)
    uint32_t occ = 0, mine[C::kSlots / C::kThreads];
#pragma unroll
    for (int q = 0; q < (int)(C::kSlots / C::kThreads); ++q) {
        mine[q] = table[threadIdx.x * (C::kSlots / C::kThreads) + q] != 0xFFFFFFFFu ? 1u : 0u;
        occ += mine[q];
    }
    uint32_t inc = occ;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, q);
        if ((threadIdx.x & 31u) >= (uint32_t)q) inc += u;
    }
    if ((threadIdx.x & 31u) == 31u) sh[threadIdx.x >> 5] = inc;
    __syncthreads();
    uint32_t wbase = 0, distinct = 0;
    for (int w = 0; w < C::kWarps; ++w) {
        if (w < (int)(threadIdx.x >> 5)) wbase += sh[w];
        distinct += sh[w];
    }
    __syncthreads();
    uint32_t rk = wbase + inc - occ;
#pragma unroll
    for (int q = 0; q < (int)(C::kSlots / C::kThreads); ++q) {
        // the slot's dense id replaces its label (each thread rewrites only its own slots)
        const uint32_t idx = threadIdx.x * (C::kSlots / C::kThreads) + q;
        table[idx] = mine[q] ? rk : 0u;
        rk += mine[q];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < C::kIpt; ++r) {
        const uint32_t j = threadIdx.x + r * C::kThreads;
        if (j < cnt) {
            ka[j] = ((uint64_t)table[slot[r]] << 32) | xo[r];
            va[j] = v[r];
        }
    }
    __syncthreads();
    // passes: the potential digits that vary inside the chunk, then the local id's
    const uint32_t varying = s_and ^ s_or;
    const int id_bits = (int)bitlen(distinct > 0 ? distinct - 1 : 0);
    uint64_t *sk = ka, *dk = kb;
    uint32_t *sv = va, *dv = vb;
    for (int shift = 0; shift < 32 + id_bits; shift += 8) {
        if (shift < 32 && ((varying >> shift) & 0xFFu) == 0u) continue;
        chunk_pass<C>(sk, sv, dk, dv, cnt, shift, whist, tpre);
        uint64_t* tk = sk; sk = dk; dk = tk;
        uint32_t* tv = sv; sv = dv; dv = tv;
    }
    // write out: position = cluster start + index inside the cluster's run
    const uint32_t q0 = threadIdx.x * C::kIpt;
    uint32_t head = 0;   // last run start at or before this thread's items
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) {
        const uint32_t q = q0 + k;
        if (q < cnt && (q == 0 || (sk[q] >> 32) != (sk[q - 1] >> 32))) head = q;
    }
    uint32_t hinc = head;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, hinc, q);
        if ((threadIdx.x & 31u) >= (uint32_t)q) hinc = max(hinc, u);
    }
    if ((threadIdx.x & 31u) == 31u) sh[threadIdx.x >> 5] = hinc;
    __syncthreads();
    uint32_t carry = 0;
    for (uint32_t w = 0; w < (threadIdx.x >> 5); ++w) carry = max(carry, sh[w]);
    uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, hinc, 1);
    if ((threadIdx.x & 31u) == 0) prev = 0;
    uint32_t run = max(carry, prev);
    uint32_t vv[C::kIpt], LL[C::kIpt];
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) {
        const uint32_t q = q0 + k;
        vv[k] = q < cnt ? sv[q] : 0u;
    }
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) LL[k] = q0 + k < cnt ? (uint32_t)d.lab[vv[k]] : 0u;
#pragma unroll
    for (int k = 0; k < C::kIpt; ++k) {
        const uint32_t q = q0 + k;
        if (q >= cnt) break;
        const uint64_t key = sk[q];
        if (q == 0 || (key >> 32) != (sk[q - 1] >> 32)) run = q;
        const uint32_t pos = t.start[LL[k]] + (q - run);
        keys_out[pos] = ((uint64_t)LL[k] << 32) | (uint32_t)key;
        vals_out[pos] = vv[k];
    }
}

// path: the value of RoundCtr::chunk_path this shape serves
template <class C, int CTAS, typename OffT>
__global__ void __launch_bounds__(C::kThreads, CTAS) k_chunk_sort(Dev<OffT> d, ClusterTables t, const uint32_t* act,
                                                                  const uint32_t* par, uint64_t* keys_out,
                                                                  uint32_t* vals_out, uint32_t path) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* ka = reinterpret_cast<uint64_t*>(smem_raw);
    uint64_t* kb = ka + C::kItems;
    uint32_t* va = reinterpret_cast<uint32_t*>(kb + C::kItems);
    uint32_t* vb = va + C::kItems;
    uint32_t (*whist)[256] = reinterpret_cast<uint32_t (*)[256]>(vb + C::kItems);
    __shared__ uint32_t tpre[256];
    __shared__ uint32_t sh[C::kWarps];
    __shared__ uint32_t s_min, s_and, s_or;

    if (d.ctr->chunk_path != path) return;
    const uint32_t n = d.ctr->n_active;
    for (uint32_t chunk = blockIdx.x; chunk * C::kRows < n; chunk += gridDim.x) {
        chunk_one<C>(d, t, act, par, keys_out, vals_out, chunk * C::kRows, n, ka, kb, va, vb, whist, tpre, sh, &s_min,
                     &s_and, &s_or);
        __syncthreads();
    }
}

}  // namespace pxr
