// The plain rounds of a small active set in one kernel (sm_100a): whole
// decompositions of small graphs, and the last rounds of larger ones.
//
// A round of the general path is about 23 launches.  On a graph of a few
// thousand vertices each of them is one or a few busy blocks walking a chain
// of dependent L2 loads (4-24 us a launch, 170 us a round on the
// 2,048-vertex planted partition), so the round costs launches and idle SMs,
// not work.  Here one thread-block cluster (up to 16 CTAs of 1,024 threads)
// runs every round: the stages are the general path's, with the hardware's
// cluster barrier between them instead of launches, totals exchanged through
// distributed shared memory instead of look-backs, and the sweep's sort as a
// stable merge sort (warps rank 32 items by comparison, runs merge by binary
// search, in shared memory up to kSmallTile items and in global memory
// above).  What bounds it is the chain of dependent L2 loads inside a stage
// and the barriers between stages (0.5-0.8 us each, about 18 a round), so a
// stage keeps several loads in flight per thread and does in one pass what
// the general path spreads over kernels.  Every result (labels, potentials,
// certificates, disabled slots, tables of the last sweep) is the general
// path's bit for bit: sums are exact fixed point, the sort is the same stable
// sort, roots and ties follow the same rules.
#pragma once

#include "pxr_kernels.cuh"

namespace pxr {

constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr uint32_t kSmallTile = 2 * kSmallThreads;   // sorted items of a CTA, and list positions it owns in the scans
constexpr uint32_t kSmallMaxCtas = 16;               // the largest (opt-in) cluster
// Which active sets take this kernel: those whose vertices fit the tiles of the
// largest cluster, up to kSmallMaxSlots edge slots at the graph's mean degree (a
// cluster is 16 of 148 SMs, so long row passes go to the whole GPU).  Measured,
// whole decomposition on a B200, here / general path in a graph: planted
// partition 2,048 vertices 1.50 / 4.42 ms, 8,192 2.10 / 5.94, 16,384 2.77 / 6.98,
// 32,000 (0.67 M slots) 3.87 / 6.22; 16,000 vertices and 1.0 M slots 2.88 / 5.64;
// 3D grid 25^3 2.92 / 6.39; R-MAT 14 3.53 / 6.96, R-MAT 15 (0.88 M slots, long
// rows) 6.47 / 8.69; 2,000 vertices and 0.84 M slots 1.46 / 4.58 (the
// union-find walks through L1 came after: here 1.45, 2.56, 3.70, 2.85 ms at
// 2,048, 16,384, 32,000 and 16,000 vertices).  Handing the last rounds over:
// 3D grid 41^3 6.2 -> 5.6 ms, 8-regular 100,000 vertices 4.8 -> 4.3, batch of 8
// instances 6.0 -> 4.4, of 64 instances 85.9 -> 83.5.
constexpr uint32_t kSmallMaxSlots = 1u << 20;
// CTAs are added while each has more vertices or edge slots than this
// (2,048-vertex planted partition: 1, 2, 4, 8 CTAs take 2.20, 2.22, 1.97,
// 1.83 ms; 16 take 1.92; 2,000 vertices with 0.84 M slots: 4, 8, 16 CTAs
// 3.24, 2.42, 2.08 ms).
constexpr uint32_t kSmallVerticesPerCta = 256;
constexpr uint32_t kSmallSlotsPerCta = 8192;
constexpr uint32_t kSmallLongRows = 2048;   // rows above light_max of a larger graph
constexpr uint32_t kSmallHash = 2 * kSmallTile;      // cluster volumes of a CTA's rescanned rows

struct SmallShared {
    union {
        struct {
            uint64_t key[2][kSmallTile];
            uint32_t at[2][kSmallTile];   // place in the unsorted tile
            uint32_t vtx[kSmallTile];
        } sort;
        struct {
            uint32_t key[kSmallHash], val[kSmallHash];
        } hash;
    };
    uint64_t pub[4];                // totals the cluster's other CTAs read
    uint64_t warp_tot[kSmallWarps];
    int64_t row_sum[kSmallWarps];
    uint32_t row_cnt[kSmallWarps];
    uint32_t red[kSmallWarps];
    uint32_t lead_end, trail_start;
};

template <typename OffT>
struct SmallArgs {
    Dev<OffT> d;
    ClusterTables tab[2];
    uint32_t* act[2];
    uint32_t* ids[2];
    uint32_t* par[2];
    float* xt[2];
    uint64_t* keys[2];
    uint32_t* vals[2];
    uint32_t xcur, tcur, acur;      // parities at entry
    uint32_t max_rounds;
};

// Barrier over the cluster; writes before it are visible to every thread after it,
// CTA-scope reads through L1 (ld_near) included: parent is rewritten every round
// inside one launch, and it is this acquire before each union-find pass, not the
// kernel's start, that bounds how old a parent read there can be.
__device__ __forceinline__ void small_sync() {
    if (gridDim.x == 1) {
        __syncthreads();
        return;
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// The other CTAs' published totals combined: exclusive prefix for this CTA and
// the sum over all, in every thread (lane i of each warp reads CTA i's word).
template <class Op>
__device__ __forceinline__ uint64_t small_prefix(const uint64_t* word, uint64_t* total) {
    const uint32_t lane = threadIdx.x & 31u;
    uint64_t v = Op::identity();
    if (lane < gridDim.x) {
        uint32_t local = (uint32_t)__cvta_generic_to_shared(word), remote;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(lane));
        asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(remote) : "memory");
    }
    uint64_t before = lane < blockIdx.x ? v : Op::identity(), all = v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        before = Op::combine(before, __shfl_xor_sync(0xFFFFFFFFu, before, o));
        all = Op::combine(all, __shfl_xor_sync(0xFFFFFFFFu, all, o));
    }
    *total = all;
    return before;
}

// Items of key < k (or <= k) in the sorted run a[0, len).
template <bool OrEqual>
__device__ __forceinline__ uint32_t small_count_below(const uint64_t* a, uint32_t len, uint64_t k) {
    uint32_t lo = 0, hi = len;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        const uint64_t x = a[mid];
        if (OrEqual ? x <= k : x < k) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Place of item i of n when the sorted runs of length L merge in pairs, ties
// to the left run: a stable merge level.
__device__ __forceinline__ uint32_t small_merge_place(const uint64_t* a, uint32_t n, uint32_t L, uint32_t i,
                                                      uint64_t k) {
    const uint32_t run = i / L, start = run * L, in_run = i - start;
    if (run & 1u) return start - L + in_run + small_count_below<true>(a + (start - L), L, k);
    const uint32_t other = start + L;
    if (other >= n) return i;
    return i + small_count_below<false>(a + other, min(L, n - other), k);
}

// The CTA's tile of the active list, sorted in shared memory; returns the
// buffer of sm.sort that holds it.
template <typename OffT>
__device__ __forceinline__ uint32_t small_sort_tile(const Dev<OffT>& d, SmallShared& sm, const uint32_t* act,
                                                    uint32_t t0, uint32_t cnt) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t base = threadIdx.x & ~31u; base < cnt; base += kSmallThreads) {
        const uint32_t i = base + lane;
        uint64_t k = ~0ull;   // above every key: labels are below 2^31
        if (i < cnt) {
            const uint32_t v = act[t0 + i];
            sm.sort.vtx[i] = v;
            k = ((uint64_t)(uint32_t)d.lab[v] << 32) | ordered_bits(d.x[v]);
        }
        // 32 items ranked by comparison; the keys come from shared memory two at
        // a time (broadcast reads cost a quarter of the shuffles they replace)
        sm.sort.key[1][i] = k;
        __syncwarp();
        uint32_t rank = 0;
#pragma unroll 8
        for (uint32_t j = 0; j < 32; j += 2) {
            const ulonglong2 o = *reinterpret_cast<const ulonglong2*>(&sm.sort.key[1][base + j]);
            rank += (o.x < k || (o.x == k && j < lane)) ? 1u : 0u;
            rank += (o.y < k || (o.y == k && j + 1 < lane)) ? 1u : 0u;
        }
        if (i < cnt) {
            sm.sort.key[0][base + rank] = k;
            sm.sort.at[0][base + rank] = i;
        }
    }
    __syncthreads();
    uint32_t cur = 0;
    for (uint32_t L = 32; L < cnt; L <<= 1) {
        for (uint32_t i = threadIdx.x; i < cnt; i += kSmallThreads) {
            const uint64_t k = sm.sort.key[cur][i];
            const uint32_t p = small_merge_place(sm.sort.key[cur], cnt, L, i, k);
            sm.sort.key[cur ^ 1u][p] = k;
            sm.sort.at[cur ^ 1u][p] = sm.sort.at[cur][i];
        }
        cur ^= 1u;
        __syncthreads();
    }
    return cur;
}

// Components, hooking pass: the root of v's tree (the forest is
// flat) goes under the smallest root among v's same-label neighbours.  Every
// pointer still leads to a smaller vertex of the same component; an edge whose
// hook another one overwrote is joined by the last pass, which looks at every edge.
// A cluster's first-link trees (one per local minimum, a tenth of the
// vertices) mostly become one here, so that pass
// finds little left to join (joining them one by one took 24 us a round on the
// 16,384-vertex planted partition, 11 after this pass).
// Long rows are left out: their edges are seen from the other ends.
// W lanes a row; every lane of the warp calls it.
template <typename OffT>
__device__ __forceinline__ void hook_row(const Dev<OffT>& d, uint32_t k, uint32_t v, bool in, uint32_t gl, uint32_t W) {
    const int32_t lv = in ? d.lab[v] : -1;
    in = in && in_split(d, k, lv);
    const OffT beg = in ? d.off[v] : 0;
    OffT end = in ? d.off[v + 1] : 0;
    if ((uint64_t)(end - beg) > d.light_max) end = beg;
    const uint32_t r = in ? ld_relaxed(&d.parent[v]) : 0u;
    uint32_t m = r;
    for (OffT s = beg + gl; s < end; s += kSlotUnroll * W) {
        uint32_t nb[kSlotUnroll];
#pragma unroll
        for (int u = 0; u < kSlotUnroll; ++u) nb[u] = s + u * W < end ? d.cols[s + u * W] : kInvalidEdge;
#pragma unroll
        for (int u = 0; u < kSlotUnroll; ++u) {
            const bool ok = slot_valid(nb[u]);
            const int32_t ln = ok ? d.lab[nb[u]] : -1;
            const uint32_t q = ok ? ld_relaxed(&d.parent[nb[u]]) : 0xFFFFFFFFu;
            if (ln == lv) m = min(m, q);
        }
    }
    for (uint32_t o = W >> 1; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if (in && gl == 0 && m < r) atomicMin(&d.parent[r], m);
}

__device__ __forceinline__ uint32_t small_block_max(uint32_t v, uint32_t* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = sh[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    }
    return v;   // valid in warp 0
}

// Rows of the vertex-order list, W lanes each (W a power of two): body(v,
// label, in the list, lane of W), called by whole warps.
template <class Body>
__device__ __forceinline__ void small_rows(const uint32_t* ids, uint32_t count, uint32_t W, Body body) {
    const uint32_t groups = gridDim.x * kSmallThreads / W;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp0 = (blockIdx.x * kSmallThreads + (threadIdx.x & ~31u)) / W;
    for (uint32_t j0 = warp0; j0 < count; j0 += groups) {
        const uint32_t j = j0 + lane / W;
        const bool in = j < count;
        body(in ? ids[j] : 0u, in, lane & (W - 1u));
    }
}

template <typename OffT>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small_decompose(SmallArgs<OffT> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmallShared& sm = *reinterpret_cast<SmallShared*>(smem_raw);
    const Dev<OffT>& d = a.d;
    RoundCtr* ctr = d.ctr;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t nt = gridDim.x * kSmallThreads;
    const uint32_t gid = blockIdx.x * kSmallThreads + threadIdx.x;
    uint32_t na = ctr->n_active, k = ctr->n_clusters, full = ctr->full_components;
    int32_t smallest = ctr->smallest;
    const uint32_t first_round = ctr->rounds;
    uint32_t rounds = first_round, last_na = 0, last_k = 0;
    uint32_t max_parent = 0xFFFFFFFFu, max_csize = d.n;   // the list at entry has no known runs
    bool err = ctr->err != 0;
    unsigned long long st_v = 0, st_s = 0, st_g = 0, st_items = 0;
    small_sync();   // everyone has read the counters
    if (gid == 0) {
        ctr->xmax_walk_bits = 0;
        ctr->any_split = 0;
    }
    small_sync();

    while (na > 0 && k > 0 && !err) {
        const uint32_t done_rounds = rounds - first_round;
        // the general loop looks at the cap after every second round
        if (done_rounds >= a.max_rounds && done_rounds > 0 && !(done_rounds & 1u)) break;
        const uint32_t par = done_rounds & 1u;
        const ClusterTables& t = a.tab[a.tcur ^ par];
        const ClusterTables& nt_tab = a.tab[a.tcur ^ par ^ 1u];
        const uint32_t* act = a.act[a.acur ^ par];
        const uint32_t* ids = a.ids[a.acur ^ par];
        uint32_t* act_next = a.act[a.acur ^ par ^ 1u];
        uint32_t* ids_next = a.ids[a.acur ^ par ^ 1u];
        const float* xt_in = a.xt[a.xcur ^ par];
        float* xt_out = a.xt[a.xcur ^ par ^ 1u];
        uint32_t W = 1;
        while (W < 8u && na * W * 2u <= nt) W <<= 1;   // idle threads share rows

        // ---- walk; beside it the cluster volumes' prefix inside each CTA's share
        {
            const int e = fixed_exponent(ld_relaxed(&ctr->xmax_bits), d.nb_bits);
            const double scale = pow2(e), inv = pow2(-e);
            uint32_t vmax = 0;
            small_rows(ids, na, W, [&](uint32_t v, bool in, uint32_t gl) {
                OffT beg = in ? d.off[v] : 0;
                const OffT end = in ? d.off[v + 1] : 0;
                const bool light = in && (uint64_t)(end - beg) <= d.light_max;
                if (!light) beg = end;
                int64_t acc = 0;
                for (OffT s = beg + gl; s < end; s += kSlotUnroll * W) {
                    uint32_t nb[kSlotUnroll];
#pragma unroll
                    for (int u = 0; u < kSlotUnroll; ++u) nb[u] = s + u * W < end ? d.cols[s + u * W] : kInvalidEdge;
                    float xv[kSlotUnroll];
#pragma unroll
                    for (int u = 0; u < kSlotUnroll; ++u) xv[u] = slot_valid(nb[u]) ? xt_in[nb[u]] : 0.0f;
#pragma unroll
                    for (int u = 0; u < kSlotUnroll; ++u) {
                        st_s += s + u * W < end ? 1 : 0;
                        if (slot_valid(nb[u])) { acc += to_fixed(xv[u], scale); ++st_g; }
                    }
                }
                for (uint32_t o = W >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
                if (light && gl == 0) {
                    const uint32_t b = walk_finish(d, v, acc, inv, xt_out);
                    vmax = b > vmax ? b : vmax;
                    ++st_v;
                }
            });
            walk_long_rows<OffT, 32>(d, xt_in, xt_out, blockIdx.x, gridDim.x, scale, inv, sm.row_sum, vmax, st_v, st_s, st_g);
            walk_long_rows<OffT, kSmallThreads>(d, xt_in, xt_out, blockIdx.x, gridDim.x, scale, inv, sm.row_sum, vmax, st_v, st_s, st_g);
            vmax = small_block_max(vmax, sm.red);
            if (threadIdx.x == 0 && vmax) atomicMax(&ctr->xmax_walk_bits, vmax);
        }
        // cluster share of this CTA: [c0, c0 + cper), two consecutive clusters a thread
        const uint32_t cper = (k + gridDim.x - 1) / gridDim.x, c0 = blockIdx.x * cper;
        const uint32_t cend = min(k, c0 + cper), cfirst = c0 + 2u * threadIdx.x;
        uint32_t cvol[2] = {0, 0};
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j)
            if (cfirst + j < cend) {
                cvol[j] = t.vol[cfirst + j];
                t.best[cfirst + j] = ~0ull;
            }
        uint64_t cta_total, all;
        const uint64_t cincl = block_inclusive<Add64>((uint64_t)cvol[0] + cvol[1], sm.warp_tot, &cta_total);
        if (threadIdx.x == 0) sm.pub[0] = cta_total;
        small_sync();

        // ---- edge differences; start volumes
        {
            const uint64_t before = small_prefix<Add64>(&sm.pub[0], &all);
            uint32_t p = (uint32_t)(before + cincl) - cvol[0] - cvol[1];
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j)
                if (cfirst + j < cend) {
                    t.vol_start[cfirst + j] = p;
                    p += cvol[j];
                }
        }
        small_rows(ids, na, W, [&](uint32_t v, bool in, uint32_t gl) {
            const uint32_t mine = in ? ordered_bits(d.x[v]) : 0u;
            OffT beg = in ? d.off[v] : 0;
            const OffT end = in ? d.off[v + 1] : 0;
            const bool light = in && (uint64_t)(end - beg) <= d.light_max;
            if (!light) beg = end;
            int32_t c = 0;
            for (OffT s = beg + gl; s < end; s += kSlotUnroll * W) {
                uint32_t nb[kSlotUnroll];
#pragma unroll
                for (int u = 0; u < kSlotUnroll; ++u) nb[u] = s + u * W < end ? d.cols[s + u * W] : kInvalidEdge;
                float xn[kSlotUnroll];
#pragma unroll
                for (int u = 0; u < kSlotUnroll; ++u) xn[u] = slot_valid(nb[u]) ? d.x[nb[u]] : 0.0f;
#pragma unroll
                for (int u = 0; u < kSlotUnroll; ++u) {
                    if (!slot_valid(nb[u])) continue;
                    const uint32_t o = ordered_bits(xn[u]);
                    c += (o < mine || (o == mine && nb[u] < v)) ? -1 : 1;
                }
            }
            for (uint32_t o = W >> 1; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
            if (light && gl == 0) d.dv[v] = make_int2(c, (int)d.ideg[v]);
        });
        nodediff_long_rows<OffT, 32>(d, blockIdx.x, gridDim.x, reinterpret_cast<int32_t*>(sm.row_cnt));
        nodediff_long_rows<OffT, kSmallThreads>(d, blockIdx.x, gridDim.x, reinterpret_cast<int32_t*>(sm.row_cnt));
        // ---- the sort's tiles, one a CTA
        // While no previous cluster (a contiguous
        // run of the active list) is longer than a tile, a cluster's items lie in
        // two neighbouring tiles at most and every item is placed at its
        // cluster's start directly; else tiles merge level by level.
        uint32_t tile = max(256u, ((na + gridDim.x - 1) / gridDim.x + 31u) & ~31u);
        if (max_parent > tile) tile = max_parent < kSmallTile ? (max_parent + 31u) & ~31u : kSmallTile;
        const bool direct = na > tile && max_parent <= tile;
        uint32_t levels = 0;
        if (!direct)
            while ((tile << levels) < na) ++levels;
        const uint32_t out = direct ? 1u : levels & 1u;
        const uint32_t t0 = blockIdx.x * tile, tcnt = t0 < na ? min(tile, na - t0) : 0u;
        uint32_t cur = 0;
        __syncthreads();
        if (tcnt) {
            cur = small_sort_tile(d, sm, act, t0, tcnt);
            for (uint32_t i = threadIdx.x; i < tcnt; i += kSmallThreads) {
                a.keys[out][t0 + i] = sm.sort.key[cur][i];
                a.vals[out][t0 + i] = sm.sort.vtx[sm.sort.at[cur][i]];
            }
            if (direct) {   // the runs the tile's first and last items belong to
                const uint32_t* parr = a.par[a.acur ^ par];
                if (threadIdx.x == 0) { sm.lead_end = tcnt; sm.trail_start = 0; }
                __syncthreads();
                const uint32_t lead = parr[t0], trail = parr[t0 + tcnt - 1];
                uint32_t le = tcnt, ts = 0;
                for (uint32_t i = threadIdx.x; i < tcnt; i += kSmallThreads) {
                    const uint32_t q = parr[t0 + i];
                    if (q != lead) le = min(le, i);
                    if (q != trail) ts = max(ts, i + 1u);
                }
                le = __reduce_min_sync(0xFFFFFFFFu, le);
                ts = __reduce_max_sync(0xFFFFFFFFu, ts);
                if (lane == 0) {
                    atomicMin(&sm.lead_end, le);
                    atomicMax(&sm.trail_start, ts);
                }
                __syncthreads();
                if (threadIdx.x == 0) {   // no run across the boundary: nothing to look up there
                    if (t0 == 0 || parr[t0 - 1] != lead) sm.lead_end = 0;
                    if (t0 + tcnt >= na || parr[t0 + tcnt] != trail) sm.trail_start = tcnt;
                }
            }
        }
        small_sync();

        // ---- sort across tiles
        if (direct) {
            for (uint32_t i = threadIdx.x; i < tcnt; i += kSmallThreads) {
                const uint64_t key = sm.sort.key[cur][i], low = key & 0xFFFFFFFF00000000ull;
                const uint32_t c = (uint32_t)(key >> 32), at = sm.sort.at[cur][i];
                uint32_t p = t.start[c] + i - small_count_below<false>(sm.sort.key[cur], tcnt, low);
                if (at < sm.lead_end)
                    p += small_count_below<true>(a.keys[1] + (t0 - tile), tile, key) -
                         small_count_below<false>(a.keys[1] + (t0 - tile), tile, low);
                if (at >= sm.trail_start) {
                    const uint32_t len = min(tile, na - t0 - tile);
                    p += small_count_below<false>(a.keys[1] + t0 + tile, len, key) -
                         small_count_below<false>(a.keys[1] + t0 + tile, len, low);
                }
                a.keys[0][p] = key;
                a.vals[0][p] = sm.sort.vtx[at];
            }
            small_sync();
        }
        for (uint32_t lev = 0; lev < levels; ++lev) {
            const uint32_t src = (levels - lev) & 1u;
            for (uint32_t i = gid; i < na; i += nt) {
                const uint64_t key = a.keys[src][i];
                const uint32_t p = small_merge_place(a.keys[src], na, tile << lev, i, key);
                a.keys[src ^ 1u][p] = key;
                a.vals[src ^ 1u][p] = a.vals[src][i];
            }
            small_sync();
        }
        const uint64_t* keys = a.keys[0];   // sorted: the last step writes buffer 0
        const uint32_t* vals = a.vals[0];

        // ---- sweep scan: two consecutive sorted positions a thread
        const uint32_t iper = (na + gridDim.x - 1) / gridDim.x, i0 = blockIdx.x * iper;
        const uint32_t ipt = iper > (uint32_t)kSmallThreads ? 2u : 1u;   // consecutive items a thread holds
        const uint32_t iend = min(na, i0 + iper), ifirst = i0 + ipt * threadIdx.x;
        uint32_t lab[2], vtx[2];
        uint64_t pre[2], run = 0;
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {
            lab[j] = 0xFFFFFFFFu;
            vtx[j] = 0;
            uint64_t val = 0;
            if (j < ipt && ifirst + j < iend) {
                lab[j] = (uint32_t)(keys[ifirst + j] >> 32);
                vtx[j] = vals[ifirst + j];
                const int2 dv = d.dv[vtx[j]];
                val = ((uint64_t)(uint32_t)dv.y << 32) | (uint32_t)dv.x;
            }
            run = PairAdd::combine(run, val);
            pre[j] = run;
        }
        const uint64_t sincl = block_inclusive<PairAdd>(run, sm.warp_tot, &cta_total);
        if (threadIdx.x == 0) sm.pub[1] = cta_total;
        small_sync();
        {
            const uint64_t before = small_prefix<PairAdd>(&sm.pub[1], &all);
            const uint32_t lo = (uint32_t)sincl - (uint32_t)run;
            const uint32_t hi = (uint32_t)(sincl >> 32) - (uint32_t)(run >> 32);
            const uint64_t excl = PairAdd::combine(before, ((uint64_t)hi << 32) | lo);
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j) {
                if (j >= ipt) break;
                const uint32_t i = ifirst + j;
                const bool in = i < iend;
                uint64_t cand = ~0ull;
                if (in) {
                    const uint64_t p = PairAdd::combine(excl, pre[j]);
                    const int32_t ldif = (int32_t)(uint32_t)p;
                    const uint32_t lvol = (uint32_t)(p >> 32) - t.vol_start[lab[j]];
                    const uint32_t tot = t.vol[lab[j]];
                    const uint32_t denom = lvol >= tot ? 0u : (lvol < tot - lvol ? lvol : tot - lvol);
                    const float sp = denom > 0 ? sweep_ratio((uint32_t)ldif, denom, d.division) : 2.0f;
                    d.pdif[i] = ldif;
                    d.pvol[i] = lvol;
                    cand = ((uint64_t)__float_as_uint(sp) << 32) | (uint32_t)~i;
                }
                // runs of one label are contiguous over the lanes: minimum towards each run's first lane
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint64_t oc = __shfl_down_sync(0xFFFFFFFFu, cand, o);
                    const uint32_t ol = __shfl_down_sync(0xFFFFFFFFu, lab[j], o);
                    if (lane + o < 32u && ol == lab[j] && oc < cand) cand = oc;
                }
                const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, lab[j], 1);
                if (in && (lane == 0 || prev != lab[j]))
                    atomicMin(reinterpret_cast<unsigned long long*>(&t.best[lab[j]]), (unsigned long long)cand);
            }
        }
        small_sync();

        // ---- cut: the cluster's decision, and the labels of split clusters
        bool any_here = false;
        {
            pxr_sweep_cut* cuts = reinterpret_cast<pxr_sweep_cut*>(d.allcuts);
            for (uint32_t c = gid; c < k; c += nt) {
                const uint64_t b = t.best[c];
                const float sp = __uint_as_float((uint32_t)(b >> 32));
                const uint32_t off = ~(uint32_t)b - t.start[c] + 1u;
                cuts[c].label = (int32_t)c;
                cuts[c].sparsity = sp;
                cuts[c].offset = off;
                const bool cut = sp < d.sc_threshold;
                const bool split = cut || full;
                d.cut_off[c] = cut ? off : kNoCut;
                d.split[c] = split ? 1 : 0;
                any_here |= split;
                if (!split) {
                    const uint32_t r = t.root[c];
                    d.rootc[r] = (kOriginSwept << 30) | c;
                    d.acc_max[r] = 0u;
                    d.acc_min[r] = 0xFFFFFFFFu;
                    d.acc_sum[r] = 0;
                    d.acc_cnt[r] = 0u;
                }
            }
            if (__any_sync(0xFFFFFFFFu, any_here) && lane == 0) ctr->any_split = 1u;
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j) {
                if (j >= ipt || ifirst + j >= iend) continue;
                const uint64_t b = t.best[lab[j]];
                const bool cut = __uint_as_float((uint32_t)(b >> 32)) < d.sc_threshold;
                // best holds ~position of the chosen prefix's last item
                if (cut || full) d.lab[vtx[j]] = (cut && ifirst + j > ~(uint32_t)b) ? (int32_t)(k + lab[j]) : (int32_t)lab[j];
            }
        }
        small_sync();

        // ---- components of split clusters
        if (ld_relaxed(&ctr->any_split)) {
            small_rows(ids, na, W, [&](uint32_t v, bool in, uint32_t gl) { link_first_row(d, k, v, in, gl, W); });
            small_sync();
            // ---- compress
            for (uint32_t j = gid; j < na; j += nt) {
                const uint32_t v = ids[j];
                if (in_split(d, k, d.lab[v])) uf_find_flat(d.parent, v);
            }
            small_sync();
            // ---- hook
            small_rows(ids, na, W, [&](uint32_t v, bool in, uint32_t gl) { hook_row(d, k, v, in, gl, W); });
            small_sync();
            // ---- compress again
            for (uint32_t j = gid; j < na; j += nt) {
                const uint32_t v = ids[j];
                if (in_split(d, k, d.lab[v])) uf_find_flat(d.parent, v);
            }
            small_sync();
            // ---- union
            for (uint32_t j = gid / W; j < na; j += nt / W) union_light_row(d, k, ids[j], gid & (W - 1u), W);
            union_long_rows<OffT, 32>(d, k, blockIdx.x, gridDim.x);
            union_long_rows<OffT, kSmallThreads>(d, k, blockIdx.x, gridDim.x);
            small_sync();
        }
        // ---- per-cluster data
        {
            const double scale = pow2(fixed_exponent(ld_relaxed(&ctr->xmax_walk_bits), d.nb_bits));
            if (gid == 0) {
                ctr->xmax_bits = 0;
                ctr->max_csize_next = 0;
                ctr->smallest_next = 0;
            }
            const DataAgg agg{d.acc_max, d.acc_min, d.acc_sum, d.acc_cnt};
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j) {
                if (j >= ipt) break;
                const bool in = ifirst + j < iend;
                uint32_t r = 0xFFFFFFFFu;
                ClusterAcc cur = DataAgg::identity();
                if (in) {
                    const uint32_t c = lab[j], v = vtx[j];
                    if (d.split[c]) {
                        r = uf_find_flat(d.parent, v);
                        if (r == v) d.rootc[r] = (kOriginChild << 30) | c;
                    } else {
                        r = t.root[c];
                    }
                    const float xv = d.x[v];
                    const uint32_t ob = ordered_bits(xv);
                    cur = ClusterAcc{ob, ob, to_fixed(xv, scale), 1u};
                }
                // one add per run of equal roots among the lanes: segments end at the next head
                const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, r, 1);
                const bool head = lane == 0 || prev != r;
                const uint32_t heads = __ballot_sync(0xFFFFFFFFu, head);
                const uint32_t later = heads & ~((2u << lane) - 1u);
                const uint32_t seg_end = later ? (uint32_t)__ffs(later) - 1u : 32u;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    ClusterAcc u;
                    u.mx = __shfl_down_sync(0xFFFFFFFFu, cur.mx, o);
                    u.mn = __shfl_down_sync(0xFFFFFFFFu, cur.mn, o);
                    u.sum = __shfl_down_sync(0xFFFFFFFFu, cur.sum, o);
                    u.cnt = __shfl_down_sync(0xFFFFFFFFu, cur.cnt, o);
                    if (lane + o < seg_end) cur = DataAgg::combine(cur, u);
                }
                if (in && head) agg.emit(r, cur);
            }
        }
        small_sync();

        // ---- the active list in vertex order: every vertex's root, and the roots'
        // index, dense label and start
        uint32_t idv[2], idc[2], idr[2];
        uint32_t rcnt[2];   // kept cluster: its size; 0: dropped
        uint32_t rinfo[2], rvol[2];
        double rsum[2];
        bool root[2];
        uint64_t rrun = 0;  // roots | kept << 20 | kept vertices << 40
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {
            root[j] = false;
            rcnt[j] = 0;
            idv[j] = 0;
            if (j >= ipt || ifirst + j >= iend) continue;
            const uint32_t v = ids[ifirst + j];
            const uint32_t lv = (uint32_t)d.lab[v];
            idv[j] = v;
            idc[j] = lv >= k ? lv - k : lv;
            idr[j] = d.split[idc[j]] ? ld_relaxed(&d.parent[v]) : t.root[idc[j]];
            root[j] = idr[j] == v;
            if (root[j]) {
                const uint32_t cnt = d.acc_cnt[v];
                const float pot = __fsub_rn(from_ordered_bits(d.acc_max[v]), from_ordered_bits(d.acc_min[v]));
                if (pot >= d.rw_threshold && cnt >= 2) rcnt[j] = cnt;
                rsum[j] = __ll2double_rn(d.acc_sum[v]);
                rinfo[j] = d.rootc[v];
                rvol[j] = t.vol[rinfo[j] & kOriginLabelMask];
                rrun += 1ull + (rcnt[j] ? (1ull << 20) + ((uint64_t)cnt << 40) : 0ull);
            }
        }
        const uint64_t rincl = block_inclusive<Add64>(rrun, sm.warp_tot, &cta_total);
        if (threadIdx.x == 0) sm.pub[2] = cta_total;
        small_sync();
        const uint64_t roots_before = small_prefix<Add64>(&sm.pub[2], &all);
        const uint32_t n_keep = (uint32_t)(all >> 20) & 0xFFFFFu, na_next = (uint32_t)(all >> 40);
        {
            uint64_t p = roots_before + rincl - rrun;
            const double inv = pow2(-fixed_exponent(ld_relaxed(&ctr->xmax_walk_bits), d.nb_bits));
            int32_t lowest = 0;
            const uint32_t biggest = __reduce_max_sync(0xFFFFFFFFu, max(rcnt[0], rcnt[1]));
            if (lane == 0 && biggest) atomicMax(&ctr->max_csize_next, biggest);
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j) {
                const uint32_t r = idv[j];
                if (!root[j]) continue;
                if (rcnt[j]) {
                    const uint32_t nl = (uint32_t)(p >> 20) & 0xFFFFFu;
                    d.newlab[r] = (int32_t)nl;
                    d.avg[r] = __ddiv_rn(__dmul_rn(rsum[j], inv), (double)rcnt[j]);
                    nt_tab.size[nl] = rcnt[j];
                    nt_tab.start[nl] = (uint32_t)(p >> 40);
                    nt_tab.root[nl] = r;
                    const bool child = (rinfo[j] >> 30) == kOriginChild;
                    d.nflag[nl] = child ? kRowsScan : kRowsKept;
                    nt_tab.vol[nl] = child ? 0u : rvol[j];
                    p += 1ull + (1ull << 20) + ((uint64_t)rcnt[j] << 40);
                } else {
                    const int32_t nl = (int32_t)((uint32_t)smallest - (uint32_t)(p & 0xFFFFFu) - 1u);
                    d.newlab[r] = nl;
                    lowest = min(lowest, nl);
                    p += 1ull;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) lowest = min(lowest, __shfl_xor_sync(0xFFFFFFFFu, lowest, o));
            if (lane == 0 && lowest < 0) atomicMin(&ctr->smallest_next, lowest);
        }
        small_sync();

        // ---- new labels, recentring, certificates (vertex order); both lists' survivors counted
        uint32_t keep_a = 0, keep_b = 0;
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {
            if (j >= ipt || ifirst + j >= iend) continue;
            const uint32_t cs = lab[j];
            const uint32_t rs = d.split[cs] ? ld_relaxed(&d.parent[vtx[j]]) : t.root[cs];
            if (d.newlab[rs] >= 0) keep_a |= 1u << j;
            const uint32_t v = idv[j], c = idc[j], r = idr[j];
            const int32_t nl = d.newlab[r];
            d.lab[v] = nl;
            if (nl >= 0) {
                d.x[v] = __double2float_rn(__dsub_rn((double)d.x[v], d.avg[r]));
                keep_b |= 1u << j;
            } else {
                const bool whole = d.cut_off[c] == kNoCut && d.acc_cnt[r] == t.size[c];
                d.cert[v] = (rounds + 1u) | (whole ? 0u : 0x80000000u);
            }
        }
        const uint64_t kept = ((uint64_t)__popc(keep_b) << 32) | (uint32_t)__popc(keep_a);
        const uint64_t kincl = block_inclusive<PairAdd>(kept, sm.warp_tot, &cta_total);
        if (threadIdx.x == 0) sm.pub[3] = cta_total;
        small_sync();

        // ---- the next lists; slots that now cross clusters; x / degree
        {
            const uint64_t before = small_prefix<PairAdd>(&sm.pub[3], &all);
            uint32_t pa = (uint32_t)before + (uint32_t)kincl - (uint32_t)kept;
            uint32_t pb = (uint32_t)(before >> 32) + (uint32_t)(kincl >> 32) - (uint32_t)(kept >> 32);
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j) {
                if (keep_a & (1u << j)) {
                    act_next[pa] = vtx[j];
                    a.par[a.acur ^ par ^ 1u][pa++] = lab[j];   // the cluster it was swept in: runs of the next list
                }
                if (keep_b & (1u << j)) ids_next[pb++] = idv[j];
            }
            if (gid == 0) {
                ctr->xmax_walk_bits = 0;
                ctr->any_split = 0;
            }
            for (uint32_t q = threadIdx.x; q < kSmallHash; q += kSmallThreads) {
                sm.hash.key[q] = 0xFFFFFFFFu;
                sm.hash.val[q] = 0u;
            }
            __syncthreads();
            uint32_t vmax = 0;
            small_rows(ids, na, W, [&](uint32_t v, bool in, uint32_t gl) {
                const int32_t lv = in ? d.lab[v] : -1;
                const bool kept_v = lv >= 0;
                const bool scan = kept_v && d.nflag[lv] == kRowsScan;
                OffT beg = scan ? d.off[v] : 0;
                const OffT end = scan ? d.off[v + 1] : 0;
                const bool light = scan && (uint64_t)(end - beg) <= d.light_max;
                if (!light) beg = end;
                uint32_t deg = 0;
                for (OffT s = beg + gl; s < end; s += kSlotUnroll * W) {
                    uint32_t nb[kSlotUnroll];
#pragma unroll
                    for (int u = 0; u < kSlotUnroll; ++u) nb[u] = s + u * W < end ? d.cols[s + u * W] : kInvalidEdge;
                    int32_t ln[kSlotUnroll];
#pragma unroll
                    for (int u = 0; u < kSlotUnroll; ++u) ln[u] = slot_valid(nb[u]) ? d.lab[nb[u]] : lv;
#pragma unroll
                    for (int u = 0; u < kSlotUnroll; ++u) {
                        if (!slot_valid(nb[u])) continue;
                        if (ln[u] != lv) d.cols[s + u * W] = nb[u] | kDisabledBit;
                        else ++deg;
                    }
                }
                for (uint32_t o = W >> 1; o > 0; o >>= 1) deg += __shfl_xor_sync(0xFFFFFFFFu, deg, o);
                if (gl != 0 || !kept_v || (scan && !light)) return;   // long rows: disable_long_rows
                if (scan) d.ideg[v] = deg; else deg = d.ideg[v];
                const float xv = d.x[v];
                xt_out[v] = deg ? __double2float_rn(__ddiv_rn((double)xv, (double)deg)) : 0.0f;
                const uint32_t b = __float_as_uint(fabsf(xv));
                vmax = b > vmax ? b : vmax;
                if (!scan) return;
                uint32_t h = ((uint32_t)lv * 2654435761u) & (kSmallHash - 1u);
                for (;;) {   // at most kSmallTile + 1024 labels: never full
                    const uint32_t prev = atomicCAS(&sm.hash.key[h], 0xFFFFFFFFu, (uint32_t)lv);
                    if (prev == 0xFFFFFFFFu || prev == (uint32_t)lv) { atomicAdd(&sm.hash.val[h], deg); break; }
                    h = (h + 1u) & (kSmallHash - 1u);
                }
            });
            vmax = max(vmax, disable_long_rows<OffT, 32>(d, xt_out, nt_tab, blockIdx.x, gridDim.x, sm.row_cnt));
            vmax = max(vmax, disable_long_rows<OffT, kSmallThreads>(d, xt_out, nt_tab, blockIdx.x, gridDim.x, sm.row_cnt));
            vmax = small_block_max(vmax, sm.red);
            if (threadIdx.x == 0 && vmax) atomicMax(&ctr->xmax_bits, vmax);
            for (uint32_t q = threadIdx.x; q < kSmallHash; q += kSmallThreads)
                if (sm.hash.key[q] != 0xFFFFFFFFu && sm.hash.val[q]) atomicAdd(&nt_tab.vol[sm.hash.key[q]], sm.hash.val[q]);
        }
        small_sync();
        st_items += na;
        last_na = na;
        last_k = k;
        na = na_next;
        k = n_keep;
        smallest = (int32_t)ld_relaxed(reinterpret_cast<const uint32_t*>(&ctr->smallest_next));
        err = ld_relaxed(&ctr->err) != 0;
        max_parent = max_csize;
        max_csize = ld_relaxed(&ctr->max_csize_next);
        full = 0;
        ++rounds;
    }

    // ---- leave the state as a round of the general path leaves it
    const uint32_t ran = rounds - first_round;
    const ClusterTables& t = a.tab[a.tcur ^ (ran & 1u)];
    if (ran > 0 && na > 0) {   // stopped early: the start volumes the next sweep reads
        const uint32_t cper = (k + gridDim.x - 1) / gridDim.x, c0 = blockIdx.x * cper;
        const uint32_t cend = min(k, c0 + cper), cfirst = c0 + 2u * threadIdx.x;
        uint32_t cvol[2] = {0, 0};
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j)
            if (cfirst + j < cend) cvol[j] = t.vol[cfirst + j];
        uint64_t cta_total, all;
        const uint64_t cincl = block_inclusive<Add64>((uint64_t)cvol[0] + cvol[1], sm.warp_tot, &cta_total);
        if (threadIdx.x == 0) sm.pub[0] = cta_total;
        small_sync();
        uint32_t p = (uint32_t)(small_prefix<Add64>(&sm.pub[0], &all) + cincl) - cvol[0] - cvol[1];
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j)
            if (cfirst + j < cend) {
                t.vol_start[cfirst + j] = p;
                p += cvol[j];
            }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        st_v += __shfl_xor_sync(0xFFFFFFFFu, st_v, o);
        st_s += __shfl_xor_sync(0xFFFFFFFFu, st_s, o);
        st_g += __shfl_xor_sync(0xFFFFFFFFu, st_g, o);
    }
    if (lane == 0) {
        unsigned long long* slot = d.walk_stats + 3 * ((blockIdx.x * kSmallWarps + warp) % kStatSlots);
        if (st_v) atomicAdd(&slot[0], st_v);
        if (st_s) atomicAdd(&slot[1], st_s);
        if (st_g) atomicAdd(&slot[2], st_g);
    }
    if (gid == 0) {
        ctr->n_active = na;
        ctr->n_clusters = k;
        ctr->rounds = rounds;
        ctr->done = (na == 0 || k == 0) ? 1u : 0u;
        ctr->n_cut = 0;
        if (ran > 0) {
            ctr->smallest = smallest;
            ctr->full_components = 0;
            ctr->max_parent = 0xFFFFFFFFu;   // the next sweep sorts globally
            ctr->max_csize = d.n;
            ctr->main_sel = 0;
            ctr->sweep_n = last_na;
            ctr->sweep_k = last_k;
            ctr->stat_sort_items += st_items;
            ctr->stat_sort_passes += ran;
            ctr->stat_swept_items += st_items;
        }
    }
    small_sync();   // no CTA leaves while another may read its shared memory
}

}  // namespace pxr
