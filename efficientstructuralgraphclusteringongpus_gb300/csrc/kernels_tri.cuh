// Full common-neighbour counts by triangles: every count of the graph at once, each triangle
// found once.
//
// Orient every edge from its lower to its higher endpoint in (degree, id) order and let N+(a)
// be the higher neighbours of a.  A triangle a < b < c in that order is found exactly once, at
// its middle vertex b: c lies in N+(a) and in N+(b).  It adds one to the counts of its three
// edges.  Streaming the lists N+(a) of b's lower neighbours reads sum d+(a)^2 entries in all,
// against the sum of d(a) over the edges for a count per edge (R-MAT s20: 2.5e9 entries against
// 6.9e9, and the longest N+ has 668), so hubs cost no more than others and no list is long.
//
// Counts are kept in the reference's edge order (GPUSCAN++/Graph.cpp:87-111), which is the
// order of the concatenated lists N+: edge (a, c) is at c's place in N+(a).  For pivot b, N+(b)
// is a bucketed table in shared memory with a counter per entry:
//   (b, c)  the counter of c, added to the counts when the pivot's slice is done;
//   (a, c)  one atomic at the streamed entry's own place;
//   (a, b)  the list's total, at b's place in N+(a) (binary search, once per edge).
#pragma once

#include "device_common.cuh"
#include "device_graph.h"
#include "kernels_cn.cuh"

namespace scan {

constexpr uint32_t kTriChunk = 1024;       // entries of N+(b) staged at once by a CTA
constexpr uint32_t kTriSliceEdges = 1024;   // lower neighbours per CTA task
constexpr int kTriWarps = 8, kTriCtas = 7;   // per CTA; CTAs per SM

__device__ __forceinline__ uint32_t hi_begin(const uint32_t* __restrict__ off, const uint32_t* __restrict__ lo_off,
                                             uint32_t v) {
    return off[v] - lo_off[v];             // both are prefix sums: higher neighbours of the vertices before v
}

// hi_adj: the lists N+ in adjacency order.  Entry j is a higher neighbour unless its bit in
// lowbits is set; wpre is the exclusive scan of the words' popcounts.
__global__ void k_fill_higher(uint64_t m, const uint32_t* __restrict__ adj, const uint32_t* __restrict__ lowbits,
                              const uint32_t* __restrict__ wpre, uint32_t* __restrict__ hi_adj) {
    for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < m; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t word = lowbits[j >> 5], bit = (uint32_t)j & 31u;
        if (!((word >> bit) & 1u)) hi_adj[j - (wpre[j >> 5] + __popc(word & ((1u << bit) - 1u)))] = adj[j];
    }
}

// Pivots with both lower and higher neighbours: up to kSmallDeg neighbours to `small` (a warp
// each), the others in slices of kTriSliceEdges lower edges to `big` as (pivot, first edge).
// counts[0], counts[1]: their numbers, zero before.
__global__ void k_tri_plan(uint32_t n, const uint32_t* __restrict__ off, const uint32_t* __restrict__ lo_off,
                           uint32_t* __restrict__ counts, uint32_t* __restrict__ small, uint2* __restrict__ big) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t v0 = blockIdx.x * (uint64_t)blockDim.x; v0 < n; v0 += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = v0 + threadIdx.x;
        uint32_t e0 = 0, lower = 0, d = 0;
        if (v < n) {
            e0 = lo_off[v];
            lower = lo_off[v + 1] - e0;
            d = off[v + 1] - off[v];
        }
        const bool pivot = lower > 0 && d > lower;
        const uint32_t ms = __ballot_sync(0xFFFFFFFFu, pivot && d <= kSmallDeg);
        uint32_t at = 0;
        if (lane == 0 && ms) at = atomicAdd(&counts[0], (uint32_t)__popc(ms));
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
        if (pivot && d <= kSmallDeg) small[at + __popc(ms & ((1u << lane) - 1u))] = (uint32_t)v;
        if (pivot && d > kSmallDeg) {
            const uint32_t slices = (lower + kTriSliceEdges - 1) / kTriSliceEdges;
            const uint32_t first = atomicAdd(&counts[1], slices);
            for (uint32_t s = 0; s < slices; ++s) big[first + s] = make_uint2((uint32_t)v, e0 + s * kTriSliceEdges);
        }
    }
}

// Place of w in a bucketed table of nb buckets, kEmpty when absent.
__device__ __forceinline__ uint32_t bucket_find(const uint32_t* tab, uint32_t nb, uint32_t w) {
    uint32_t b = hash_slot(w, nb);
    for (uint32_t it = 0; it < nb; ++it) {
        const uint4 q = *reinterpret_cast<const uint4*>(tab + 4 * b);
        const uint32_t i = q.x == w ? 0u : q.y == w ? 1u : q.z == w ? 2u : q.w == w ? 3u : 4u;
        if (i < 4) return 4 * b + i;
        if (q.w == kEmpty) return kEmpty;
        b = (b + 1 == nb) ? 0 : b + 1;
    }
    return kEmpty;
}

// The staged N+(b) (or a chunk of it): a bitmap of hashed entries, 16 bits each, in front of
// the table with the counters.  Most streamed entries are not in it: those cost one 4-byte
// probe; the rest queue up per warp and are looked up by full warps.  Looking every entry up in
// place left half the lanes idle (R-MAT of 500K vertices, 6M edges: 1.98 ms for the pivots above
// 128 neighbours, with the queue 1.66, at seven CTAs per SM 1.35).
struct TriStage {
    uint32_t *bits, *tab, *hits;
    uint32_t entries, buckets, log2bits;
};
// Load 1/2: few entries reach the table, and half the size leaves room for seven CTAs on an SM.
__host__ __device__ constexpr uint32_t tri_buckets(uint32_t entries) { return entries / 2 + 1; }
constexpr uint32_t kTriQueue = 31 + 128;       // what is left of a warp's queue plus one round

__host__ __device__ constexpr uint32_t tri_log2bits(uint32_t entries) {
    uint32_t l = 7;
    while ((1u << l) < 16u * entries) ++l;
    return l;
}

// Lower edges [kb, min(kb + 32, e1)) of pivot b, one per lane: their lists N+ as one stream of
// 16-byte words, a word per lane and round.  qw, qp: the warp's queue (entry; owner lane << 27
// and place in the owner's list); tot: 32 words.
__device__ __forceinline__ void tri_batch(uint32_t kb, uint32_t e1, uint32_t b, const uint32_t* __restrict__ off,
                                          const uint32_t* __restrict__ lo_off, const uint32_t* __restrict__ lo_adj,
                                          const uint32_t* __restrict__ hi_adj, const TriStage& st, uint32_t* qw,
                                          uint32_t* qp, uint32_t* tot, uint32_t* __restrict__ cnt, uint32_t lane) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const uint32_t lower = (1u << lane) - 1u;
    uint32_t ub = 0, ue = 0;
    if (kb + lane < e1) {
        const uint32_t a = lo_adj[kb + lane];
        ub = hi_begin(off, lo_off, a);
        ue = hi_begin(off, lo_off, a + 1);
    }
    const uint32_t sw = ue > ub ? (((ue + 3u) & ~3u) - (ub & ~3u)) >> 2 : 0u;
    uint32_t incl = sw;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, s);
        if ((int)lane >= s) incl += y;
    }
    const uint32_t excl = incl - sw, total = __shfl_sync(kFull, incl, 31);
    tot[lane] = 0;
    __syncwarp();
    uint32_t queued = 0;
    auto look_up = [&](uint32_t first, uint32_t n) {          // queue entries [first, first + n), n <= 32
        const uint32_t item = lane < n ? qp[first + lane] : 0u, owner = item >> 27;
        const uint32_t place = __shfl_sync(kFull, ub, owner) + (item & 0x7FFFFFFu);
        if (lane < n) {
            const uint32_t s = bucket_find(st.tab, st.buckets, qw[first + lane]);
            if (s != kEmpty) {
                atomicAdd(&st.hits[s], 1u);
                atomicAdd(&cnt[place], 1u);
                atomicAdd(&tot[owner], 1u);
            }
        }
        __syncwarp();
    };
    for (uint32_t y0 = 0; y0 < total; y0 += 32u) {
        const uint32_t y = y0 + lane;
        uint32_t j = 0;   // owner: first lane whose inclusive prefix exceeds y
#pragma unroll
        for (int st2 = 16; st2 > 0; st2 >>= 1) {
            const uint32_t pj = __shfl_sync(kFull, incl, j + st2 - 1);
            if (pj <= y) j += st2;
        }
        j &= 31u;
        const uint32_t lb = __shfl_sync(kFull, ub, j), le = __shfl_sync(kFull, ue, j);
        const uint32_t p = (lb & ~3u) + 4u * (y - __shfl_sync(kFull, excl, j));
        uint4 x = make_uint4(0, 0, 0, 0);
        uint32_t in = 0;                                       // which of the four belong to the list
        if (y < total) {
            x = __ldg(reinterpret_cast<const uint4*>(hi_adj + p));
            in = (0xFu << (lb > p ? lb - p : 0u)) & (0xFu >> (p + 4u > le ? p + 4u - le : 0u));
        }
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t h = w[i] * 0x9E3779B1u;
            const uint32_t word = st.bits[h >> (37u - st.log2bits)];
            const bool maybe = __funnelshift_r(word, word, h >> (32u - st.log2bits)) & (in >> i) & 1u;
            const uint32_t m = __ballot_sync(kFull, maybe);
            if (maybe) {
                const uint32_t at = queued + __popc(m & lower);
                qw[at] = w[i];
                qp[at] = j << 27 | (p + i - lb);
            }
            queued += __popc(m);
        }
        __syncwarp();
        while (queued >= 32) {
            queued -= 32;
            look_up(queued, 32);
        }
    }
    if (queued) look_up(0, queued);
    const uint32_t t = tot[lane];
    if (t) {
        const uint32_t at = lower_bound_u32(hi_adj, ub, ue, b);
        if (at < ue && hi_adj[at] == b) atomicAdd(&cnt[at], t);   // always, in a symmetric graph
    }
    __syncwarp();
}

// Threads first, first + step, ... of those that share the stage; a barrier among them between
// the two and after.
__device__ __forceinline__ void tri_stage_clear(const TriStage& st, uint32_t first, uint32_t step) {
    for (uint32_t i = first; i < (1u << st.log2bits) / 32; i += step) st.bits[i] = 0;
    for (uint32_t i = first; i < st.buckets; i += step) {
        reinterpret_cast<uint4*>(st.tab)[i] = make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
        reinterpret_cast<uint4*>(st.hits)[i] = make_uint4(0, 0, 0, 0);
    }
}

__device__ __forceinline__ void tri_stage_fill(const TriStage& st, const uint32_t* __restrict__ list, uint32_t first,
                                               uint32_t step) {
    for (uint32_t i = first; i < st.entries; i += step) {
        const uint32_t w = list[i], h = (w * 0x9E3779B1u) >> (32u - st.log2bits);
        atomicOr(&st.bits[h >> 5], 1u << (h & 31u));
        bucket_insert(st.tab, st.buckets, w);
    }
}

__device__ __forceinline__ void tri_stage_flush(const TriStage& st, const uint32_t* __restrict__ list,
                                                uint32_t* __restrict__ cnt, uint32_t first, uint32_t step) {
    for (uint32_t i = first; i < st.entries; i += step) {
        const uint32_t s = bucket_find(st.tab, st.buckets, list[i]);
        const uint32_t h = s != kEmpty ? st.hits[s] : 0u;
        if (h) atomicAdd(&cnt[i], h);
    }
}

__global__ void __launch_bounds__(kTriWarps * 32, kTriCtas)
k_tri_big(const uint2* __restrict__ tasks, const uint32_t* __restrict__ counts, uint32_t* queue,
          const uint32_t* __restrict__ off, const uint32_t* __restrict__ lo_off, const uint32_t* __restrict__ lo_adj,
          const uint32_t* __restrict__ hi_adj, uint32_t* __restrict__ cnt) {
    __shared__ __align__(16) uint32_t tab[4 * tri_buckets(kTriChunk)];
    __shared__ __align__(16) uint32_t hits[4 * tri_buckets(kTriChunk)];
    __shared__ uint32_t bits[(1u << tri_log2bits(kTriChunk)) / 32];
    __shared__ uint32_t qw[kTriWarps][kTriQueue], qp[kTriWarps][kTriQueue], tot[kTriWarps][32];
    __shared__ uint32_t next_batch, task_slot;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t ntasks = counts[1];
    for (uint32_t t = next_task(queue, 0, true, &task_slot); t < ntasks; t = next_task(queue, t, false, &task_slot)) {
        const uint2 tk = tasks[t];
        const uint32_t b = tk.x, e1 = min(tk.y + kTriSliceEdges, lo_off[b + 1]);
        const uint32_t hb = hi_begin(off, lo_off, b), he = hi_begin(off, lo_off, b + 1);
        for (uint32_t c0 = hb; c0 < he; c0 += kTriChunk) {        // nearly always one
            const uint32_t nb = min(kTriChunk, he - c0);
            const TriStage st{bits, tab, hits, nb, tri_buckets(nb), tri_log2bits(nb)};
            tri_stage_clear(st, threadIdx.x, blockDim.x);
            if (threadIdx.x == 0) next_batch = 0;
            __syncthreads();
            tri_stage_fill(st, hi_adj + c0, threadIdx.x, blockDim.x);
            __syncthreads();
            for (;;) {
                uint32_t j = 0;
                if (lane == 0) j = atomicAdd(&next_batch, 1u);
                const uint32_t kb = tk.y + 32u * __shfl_sync(0xFFFFFFFFu, j, 0);
                if (kb >= e1) break;
                tri_batch(kb, e1, b, off, lo_off, lo_adj, hi_adj, st, qw[wib], qp[wib], tot[wib], cnt, lane);
            }
            __syncthreads();
            tri_stage_flush(st, hi_adj + c0, cnt + c0, threadIdx.x, blockDim.x);
            __syncthreads();
        }
    }
}

__global__ void __launch_bounds__(kTriWarps * 32)
k_tri_small(const uint32_t* __restrict__ pivots, const uint32_t* __restrict__ counts, uint32_t* queue,
            const uint32_t* __restrict__ off, const uint32_t* __restrict__ lo_off, const uint32_t* __restrict__ lo_adj,
            const uint32_t* __restrict__ hi_adj, uint32_t* __restrict__ cnt) {
    __shared__ __align__(16) uint32_t tab[kTriWarps][4 * tri_buckets(kSmallDeg)];
    __shared__ __align__(16) uint32_t hits[kTriWarps][4 * tri_buckets(kSmallDeg)];
    __shared__ uint32_t bits[kTriWarps][(1u << tri_log2bits(kSmallDeg)) / 32];
    __shared__ uint32_t qw[kTriWarps][kTriQueue], qp[kTriWarps][kTriQueue], tot[kTriWarps][32];
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint32_t npiv = counts[0];
    for (;;) {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(queue, 4u);                  // four at a time: half a microsecond each
        t = __shfl_sync(0xFFFFFFFFu, t, 0);
        if (t >= npiv) break;
        for (uint32_t q = t; q < min(t + 4, npiv); ++q) {
            const uint32_t b = pivots[q];
            const uint32_t hb = hi_begin(off, lo_off, b), nb = hi_begin(off, lo_off, b + 1) - hb;   // <= kSmallDeg
            const uint32_t e0 = lo_off[b], e1 = lo_off[b + 1];
            const TriStage st{bits[wib], tab[wib], hits[wib], nb, tri_buckets(nb), tri_log2bits(nb)};
            tri_stage_clear(st, lane, 32);
            __syncwarp();
            tri_stage_fill(st, hi_adj + hb, lane, 32);
            __syncwarp();
            for (uint32_t kb = e0; kb < e1; kb += 32)
                tri_batch(kb, e1, b, off, lo_off, lo_adj, hi_adj, st, qw[wib], qp[wib], tot[wib], cnt, lane);
            __syncwarp();
            tri_stage_flush(st, hi_adj + hb, cnt + hb, lane, 32);
            __syncwarp();
        }
    }
}

// cn[] (edges by higher endpoint) from the counts in the reference's order.
__global__ void k_from_reference_order(uint64_t E, const uint32_t* __restrict__ off,
                                       const uint32_t* __restrict__ lo_off, const uint32_t* __restrict__ lo_adj,
                                       const uint32_t* __restrict__ lo_src, const uint32_t* __restrict__ hi_adj,
                                       const uint32_t* __restrict__ cnt, uint32_t* __restrict__ cn) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t u = lo_adj[e], v = lo_src[e], end = hi_begin(off, lo_off, u + 1);
        const uint32_t at = lower_bound_u32(hi_adj, hi_begin(off, lo_off, u), end, v);
        cn[e] = at < end && hi_adj[at] == v ? cnt[at] : 0u;       // found, in a symmetric graph
    }
}

// Whether the list kernels count faster: graphs of nearly complete neighbourhoods.  A streamed
// entry that is in the table costs two to three times one that is not (the queue, the lookup, three
// atomics), and where degrees are alike the lists are only 1.5 to 2 times the entries the triangles
// stream.  Full counts, ms, by lists / by triangles: complete graphs of 1,500 and 4,000 vertices
// 2.5 / 3.8 and 39 / 72, disjoint ones of 120, 300 and 800 1.70 / 1.98, 3.37 / 3.76 and 7.2 / 9.2,
// ring lattices of degree 200 and 600 1.33 / 1.52 and 2.32 / 2.55; half of the entries of each are
// hits.  With a quarter hits (communities of degree 170) 1.75 / 1.61, a sixth 5.0 / 4.0; and at
// lower degrees launches and latency decide (disjoint ones of 48 0.97 / 0.85, a ring lattice of
// degree 32 1.43 / 0.85).  So graphs of at least kTriDenseDegree neighbours on average are looked
// at: random entries of the lists of random edges (the first few thousand multiples of a prime),
// about 20 us.  sums[0] entries of the lists, [1] of those the triangles stream, [2] samples found.
constexpr uint64_t kTriDenseEdges = 1u << 19;
constexpr uint32_t kTriDenseDegree = 96, kTriSamples = 8192;
__host__ __device__ constexpr bool tri_dense(uint64_t lists, uint64_t streamed, uint64_t hits) {
    return 4 * lists <= 9 * streamed && 5 * hits >= 2 * streamed;
}

__global__ void k_tri_sample(uint64_t E, const uint32_t* __restrict__ off, const uint32_t* __restrict__ lo_off,
                             const uint32_t* __restrict__ lo_adj, const uint32_t* __restrict__ lo_src,
                             const uint32_t* __restrict__ hi_adj, unsigned long long* __restrict__ sums) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t lists = 0, streamed = 0, hits = 0;
    if (i < kTriSamples) {
        const uint64_t e = (i * 2654435761ull) % E;
        const uint32_t a = lo_adj[e], b = lo_src[e];
        const uint32_t ab = hi_begin(off, lo_off, a), ae = hi_begin(off, lo_off, a + 1);
        lists = off[a + 1] - off[a];
        streamed = ae - ab;
        if (streamed) {
            const uint32_t c = hi_adj[ab + __umulhi(i * 0x9E3779B1u, streamed)];
            const uint32_t be = hi_begin(off, lo_off, b + 1);
            const uint32_t at = lower_bound_u32(hi_adj, hi_begin(off, lo_off, b), be, c);
            if (at < be && hi_adj[at] == c) hits = streamed;      // an entry stands for its list
        }
    }
    lists = __reduce_add_sync(0xFFFFFFFFu, lists);
    streamed = __reduce_add_sync(0xFFFFFFFFu, streamed);
    hits = __reduce_add_sync(0xFFFFFFFFu, hits);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sums[0], (unsigned long long)lists);
        atomicAdd(&sums[1], (unsigned long long)streamed);
        atomicAdd(&sums[2], (unsigned long long)hits);
    }
}

}  // namespace scan
