// Neighbourhood sketches: an upper bound on every edge's common-neighbour count from two
// short bitmaps, before any neighbour list is read.
//
// A vertex of degree d >= 2 keeps its neighbours hashed into a bitmap of 2^L bits, L the
// least with 2^L >= 12 d (16 d above 85 neighbours; at least 2^7, at most 2^20), and every
// fold of that bitmap down to 2^7 bits: the fold of 2^l bits is the lower half OR the upper
// half of the one of 2^(l+1), which is the bitmap the same hash gives with l bits.  So two
// vertices can be compared at any size both have.  A bit set for u and clear for v is a
// neighbour of u that v does not have, and distinct bits are distinct neighbours, so
//     |N(u) & N(v)| <= d_u - popcount(bits_u & ~bits_v).
// An edge whose count must reach tlo (count_floor) is decided, not similar, once more than
// d_u - tlo such bits are seen; the rest are left to the list kernels (kernels_cn.cuh).
//
// Layout, in 16-byte units: all bitmaps of 2^l bits are one array, 2^(l-7) units each, in the
// order of the vertices' ranks; ranks descend by L, so the vertices that have a size are the
// first ones.  Every bitmap is aligned to its own size (up to 128 bytes), and what a run reads
// (mostly one or two sizes per vertex) lies together: with each vertex's sizes side by side
// instead, the similarity stage of R-MAT s22 at eps 0.5 took 2.06 ms, so 1.87.  All arrays and
// what goes with them take 0.9 times the adjacency (random graphs, rings) to 1.5 times (R-MAT s22),
// plans with split pivots half the adjacency more.
#pragma once

#include "device_common.cuh"
#include "device_graph.h"
#include "kernels_cn.cuh"
#include "pending_slices.cuh"

namespace scan {

// Bits per neighbour, rounded up to a power of two.  More decide more edges at low eps and are
// read only where fewer cannot; longer lists cost more to count when left open (R-MAT s21 at
// eps 0.2, whole run: 6.0 ms with 12 throughout, 5.0 with 16 above 85 neighbours, 5.95 with 24
// above 682).
constexpr uint32_t kSketchBits = 12, kSketchBitsLarge = 16, kSketchLargeDeg = 85;
constexpr int kSketchMinLog = 7;          // one 16-byte unit
constexpr int kSketchMaxLog = 20;         // 128 KB: larger hubs share bits
static_assert(kSketchClasses == kSketchMaxLog - kSketchMinLog + 1, "bitmap sizes");
constexpr int kSketchMidLog = 17;         // classes up to here are built by small CTAs, larger by whole-SM ones
constexpr int kSketchWarpLog = 13;        // classes up to here are built by one warp

// log2 of the bitmap size of a vertex of degree d >= 1.
__host__ __device__ __forceinline__ int sketch_log(uint32_t d) {
    if (d <= (1u << kSketchMinLog) / kSketchBits) return kSketchMinLog;
    if (d >= (1u << kSketchMaxLog) / kSketchBitsLarge) return kSketchMaxLog;
    const uint32_t x = (d > kSketchLargeDeg ? kSketchBitsLarge : kSketchBits) * d - 1u;   // ceil(log2(x + 1))
#ifdef __CUDA_ARCH__
    return 32 - __clz(x);
#else
    return 32 - __builtin_clz(x);
#endif
}

// Bit of neighbour w in a bitmap of 2^l bits: the low l bits.  The reversal puts the product's
// well-mixed high bits lowest.
__device__ __forceinline__ uint32_t sketch_hash(uint32_t w) { return __brev(w * 0x9E3779B1u); }

// cls[c] = vertices of size class c (degree >= 2).
__global__ void k_sketch_classes(uint32_t n, const uint32_t* __restrict__ off, uint32_t* __restrict__ cls) {
    __shared__ uint32_t h[kSketchClasses];
    if (threadIdx.x < kSketchClasses) h[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t v0 = blockIdx.x * (uint64_t)blockDim.x; v0 < n; v0 += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = v0 + threadIdx.x;
        const uint32_t d = v < n ? off[v + 1] - off[v] : 0u;
        const int c = d >= 2 ? sketch_log(d) - kSketchMinLog : -1;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, c);
        if (c >= 0 && (__ffs(peers) - 1) == (int)(threadIdx.x & 31)) atomicAdd(&h[c], (uint32_t)__popc(peers));
    }
    __syncthreads();
    if (threadIdx.x < kSketchClasses && h[threadIdx.x]) atomicAdd(&cls[threadIdx.x], h[threadIdx.x]);
}

// First rank of each class and the lists of the vertices that CTAs build.
struct SketchPlan {
    uint32_t first[kSketchClasses];
    uint32_t list_mid, list_hub;      // entries of the two lists
};

// The bitmap of 2^l bits of the vertex of a rank: its first unit.
__device__ __forceinline__ uint32_t sketch_unit(const SketchLevels& lv, int l, uint32_t rank) {
    return lv.base[l - kSketchMinLog] + (rank << (l - kSketchMinLog));
}

// info[v] = (rank, degree).  rank: one counter per class, then the mid and
// hub list counters, all zero.  The order within a class is whatever the atomics give; nothing
// depends on it.
__global__ void k_sketch_assign(uint32_t n, const uint32_t* __restrict__ off, SketchPlan plan,
                                uint32_t* __restrict__ rank, uint2* __restrict__ info, uint32_t* __restrict__ mid,
                                uint32_t* __restrict__ hub) {
    __shared__ uint32_t h[kSketchClasses], base[kSketchClasses];
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t v0 = blockIdx.x * (uint64_t)blockDim.x; v0 < n; v0 += (uint64_t)gridDim.x * blockDim.x) {
        if (threadIdx.x < kSketchClasses) h[threadIdx.x] = 0;
        __syncthreads();
        const uint64_t v = v0 + threadIdx.x;
        const uint32_t d = v < n ? off[v + 1] - off[v] : 0u;
        const int c = d >= 2 ? sketch_log(d) - kSketchMinLog : -1;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, c);
        const int lead = __ffs(peers) - 1;
        uint32_t r = 0;
        if (c >= 0 && lead == (int)lane) r = atomicAdd(&h[c], (uint32_t)__popc(peers));
        r = __shfl_sync(0xFFFFFFFFu, r, lead) + __popc(peers & ((1u << lane) - 1u));
        __syncthreads();
        if (threadIdx.x < kSketchClasses)
            base[threadIdx.x] = h[threadIdx.x] ? atomicAdd(&rank[threadIdx.x], h[threadIdx.x]) : 0u;
        __syncthreads();
        if (v < n) {
            uint32_t place = 0;
            if (c >= 0) {
                place = plan.first[c] + base[c] + r;
                const int l = c + kSketchMinLog;
                if (l > kSketchMidLog) {
                    const uint32_t i = atomicAdd(&rank[kSketchClasses + 1], 1u);
                    if (i < plan.list_hub) hub[i] = (uint32_t)v;
                } else if (l > kSketchWarpLog) {
                    const uint32_t i = atomicAdd(&rank[kSketchClasses], 1u);
                    if (i < plan.list_mid) mid[i] = (uint32_t)v;
                }
            }
            info[v] = make_uint2(place, d);
        }
    }
}

// Vertices [v_begin, v_end) of the classes up to kSketchWarpLog, 32 per warp: those of the
// smallest class one per lane (four words in registers), up to kSketchOctetLog four at a time
// by eight lanes each (folds by shuffle), the others one after the other by the whole warp in
// shared memory.  Latency bounds it (a list load, the shared atomics, the folds), so several
// loads are in flight per lane (R-MAT s22: 0.87 ms with a warp per vertex, now 0.66 in eight
// parts, of which all but the last run while the adjacency arrives).
constexpr int kSketchWarps = 8;
constexpr int kSketchOctetLog = 10;    // 8 units, up to 85 neighbours
__global__ void __launch_bounds__(kSketchWarps * 32) k_sketch_build_small(uint32_t v_begin, uint32_t v_end,
                                                                          const uint32_t* __restrict__ off,
                                                                          const uint32_t* __restrict__ adj,
                                                                          const uint2* __restrict__ info,
                                                                          uint4* __restrict__ sk, SketchLevels lv) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    __shared__ __align__(16) uint32_t smem[kSketchWarps][(1u << kSketchWarpLog) / 32];
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5, gl = lane & 7u, gi = lane >> 3;
    uint32_t* bits = smem[wib];
    uint4* bits4 = reinterpret_cast<uint4*>(bits);
    const uint64_t step = (uint64_t)gridDim.x * kSketchWarps * 32;
    for (uint64_t v0 = v_begin + ((uint64_t)blockIdx.x * kSketchWarps + wib) * 32; v0 < v_end; v0 += step) {
        const uint64_t v = v0 + lane;
        const uint2 iv = v < v_end ? info[v] : make_uint2(0, 0);
        const uint32_t b = v < v_end ? off[v] : 0u;
        const int l = iv.y >= 2 ? sketch_log(iv.y) : 0;
        if (l == kSketchMinLog) {
            uint4 q = make_uint4(0, 0, 0, 0);
            for (uint32_t j = 0; j < iv.y; ++j) {
                const uint32_t h = sketch_hash(adj[b + j]) & 127u, bit = 1u << (h & 31u), w = h >> 5;
                if (w == 0) q.x |= bit; else if (w == 1) q.y |= bit; else if (w == 2) q.z |= bit; else q.w |= bit;
            }
            sk[sketch_unit(lv, kSketchMinLog, iv.x)] = q;
        }
        uint32_t octets = __ballot_sync(kFull, l > kSketchMinLog && l <= kSketchOctetLog);
        while (octets) {
            // the gi-th of the lowest four set bits
            uint32_t rest = octets;
            for (uint32_t i = 0; i < gi; ++i) rest &= rest - 1;
            const int j = rest ? __ffs(rest) - 1 : 0;
            for (int i = 0; i < 4; ++i) octets &= octets - 1;
            const uint32_t dj = __shfl_sync(kFull, iv.y, j), a = __shfl_sync(kFull, b, j);
            const uint32_t rank = __shfl_sync(kFull, iv.x, j);
            const int lj = __shfl_sync(kFull, l, j);
            const uint32_t d = rest ? dj : 0u;
            const uint32_t units = rest ? 1u << (lj - kSketchMinLog) : 0u, mask = rest ? (1u << lj) - 1u : 0u;
            uint32_t* mine = bits + 32 * gi;               // 8 units
            reinterpret_cast<uint4*>(mine)[gl] = make_uint4(0, 0, 0, 0);
            __syncwarp();
            for (uint32_t i = gl; i < d; i += 48) {
                uint32_t w[6];
#pragma unroll
                for (int q = 0; q < 6; ++q) w[q] = i + 8 * q < d ? __ldg(adj + a + i + 8 * q) : 0u;
#pragma unroll
                for (int q = 0; q < 6; ++q)
                    if (i + 8 * q < d) {
                        const uint32_t h = sketch_hash(w[q]) & mask;
                        atomicOr(&mine[h >> 5], 1u << (h & 31u));
                    }
            }
            __syncwarp();
            uint4 x = reinterpret_cast<uint4*>(mine)[gl];
            if (gl < units) sk[sketch_unit(lv, lj, rank) + gl] = x;
#pragma unroll
            for (int f = 2; f >= 0; --f) {                 // the fold of 2^f units
                const uint32_t half = 1u << f;
                uint4 y;
                y.x = __shfl_down_sync(kFull, x.x, half, 8);
                y.y = __shfl_down_sync(kFull, x.y, half, 8);
                y.z = __shfl_down_sync(kFull, x.z, half, 8);
                y.w = __shfl_down_sync(kFull, x.w, half, 8);
                if (half < units) {
                    x.x |= y.x; x.y |= y.y; x.z |= y.z; x.w |= y.w;
                    if (gl < half) sk[sketch_unit(lv, kSketchMinLog + f, rank) + gl] = x;
                }
            }
            __syncwarp();
        }
        uint32_t todo = __ballot_sync(kFull, l > kSketchOctetLog && l <= kSketchWarpLog);
        while (todo) {
            const int j = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t d = __shfl_sync(kFull, iv.y, j), a = __shfl_sync(kFull, b, j);
            const uint32_t rank = __shfl_sync(kFull, iv.x, j);
            const int lj = __shfl_sync(kFull, l, j);
            const uint32_t units = 1u << (lj - kSketchMinLog), mask = (1u << lj) - 1u;
            for (uint32_t i = lane; i < units; i += 32) bits4[i] = make_uint4(0, 0, 0, 0);
            __syncwarp();
            for (uint32_t i = lane; i < d; i += 256) {
                uint32_t w[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) w[q] = i + 32 * q < d ? __ldg(adj + a + i + 32 * q) : 0u;
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (i + 32 * q < d) {
                        const uint32_t h = sketch_hash(w[q]) & mask;
                        atomicOr(&bits[h >> 5], 1u << (h & 31u));
                    }
            }
            __syncwarp();
            const uint32_t at = sketch_unit(lv, lj, rank);
            for (uint32_t i = lane; i < units; i += 32) sk[at + i] = bits4[i];
            for (int f = lj - 1; f >= kSketchMinLog; --f) {        // folds, in place
                const uint32_t half = 1u << (f - kSketchMinLog), to = sketch_unit(lv, f, rank);
                __syncwarp();
                for (uint32_t i = lane; i < half; i += 32) {
                    uint4 x = bits4[i];
                    const uint4 y = bits4[i + half];
                    x.x |= y.x; x.y |= y.y; x.z |= y.z; x.w |= y.w;
                    bits4[i] = x;
                    sk[to + i] = x;
                }
            }
            __syncwarp();
        }
    }
}

// The larger classes: one CTA per vertex of a list, the bitmap in dynamic shared memory.
__global__ void k_sketch_build_cta(const uint32_t* __restrict__ list, uint32_t count, const uint32_t* __restrict__ off,
                                   const uint32_t* __restrict__ adj, const uint2* __restrict__ info,
                                   uint4* __restrict__ sk, SketchLevels lv) {
    extern __shared__ __align__(16) uint32_t sketch_smem[];
    uint32_t* bits = sketch_smem;
    uint4* bits4 = reinterpret_cast<uint4*>(bits);
    for (uint32_t t = blockIdx.x; t < count; t += gridDim.x) {
        const uint32_t v = list[t];
        const uint2 iv = info[v];
        const uint32_t b = off[v];
        const int l = sketch_log(iv.y);
        const uint32_t units = 1u << (l - kSketchMinLog), mask = (1u << l) - 1u;
        for (uint32_t i = threadIdx.x; i < units; i += blockDim.x) bits4[i] = make_uint4(0, 0, 0, 0);
        __syncthreads();
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < iv.y; i += blockDim.x) {
            const uint32_t h = sketch_hash(__ldg(adj + b + i)) & mask;
            atomicOr(&bits[h >> 5], 1u << (h & 31u));
        }
        __syncthreads();
        const uint32_t at = sketch_unit(lv, l, iv.x);
        for (uint32_t i = threadIdx.x; i < units; i += blockDim.x) sk[at + i] = bits4[i];
        for (int f = l - 1; f >= kSketchMinLog; --f) {
            const uint32_t half = 1u << (f - kSketchMinLog), to = sketch_unit(lv, f, iv.x);
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < half; i += blockDim.x) {
                uint4 x = bits4[i];
                const uint4 y = bits4[i + half];
                x.x |= y.x; x.y |= y.y; x.z |= y.z; x.w |= y.w;
                bits4[i] = x;
                sk[to + i] = x;
            }
        }
        __syncthreads();
    }
}

// ---- the bound ------------------------------------------------------------------------------

// Bitmap size to try first for an edge that needs `need` missing bits: the expected number of
// bits of u that v lacks, were their lists unrelated, is about d_u exp(-(d_u / 2 + d_v) / 2^l)
// (bits shared within u's list, and bits v has by chance); the least l at which that is
// need / kSketchMargin.  0: even u's largest bitmap cannot be expected to decide the edge; tried
// it is up to half the square root of `need` above what is expected, the spread of such a count
// (random graphs, whole runs against trying only what is expected to fall 3% short: 50K vertices of
// degree 200 at eps 0.1 1.78 -> 0.82 ms, 1M of degree 32 at eps 0.15 2.50 -> 2.12 and at 0.2 2.40 ->
// 1.39; a whole square root, or a flat 10%, costs 0.1 ms where none is decided).  Only speed depends
// on this choice.
constexpr float kSketchMargin = 0.9f;      // first try (R-MAT, SBM, power laws: 0.8-0.95 read about the same bytes)
constexpr float kSketchSpread = 0.5f;      // whether to try at all
__device__ __forceinline__ int sketch_level(uint32_t du, uint32_t dv, uint32_t need, int top) {
    const float num = 0.5f * (float)du + (float)dv, inv = (float)du / (float)need;
    const float g = __logf(kSketchMargin * inv);
    const float cap = (float)(1u << top);
    if (g <= 0.f || num > g * cap) return num < __logf((1.f + kSketchSpread * rsqrtf((float)need)) * inv) * cap ? top : 0;
    const uint32_t bits = (uint32_t)__fdividef(num, g);      // < 2^top
    const int l = 32 - __clz(bits | ((1u << kSketchMinLog) - 1u));
    return min(max(l, kSketchMinLog), top);
}

struct SketchSlot {      // one edge of a warp's batch that needs its bitmaps
    uint32_t ru, rv;     // ranks of the endpoints
    uint32_t need;       // missing bits that decide it
    uint32_t code;       // edge within the batch | level << 8 | top level << 16
};
__device__ __forceinline__ uint32_t slot_level(const SketchSlot& s) { return (s.code >> 8) & 0xFFu; }
__device__ __forceinline__ uint32_t slot_top(const SketchSlot& s) { return (s.code >> 16) & 0xFFu; }

__device__ __forceinline__ uint32_t missing_bits(const uint4 x, const uint4 y) {
    return __popc(x.x & ~y.x) + __popc(x.y & ~y.y) + __popc(x.z & ~y.z) + __popc(x.w & ~y.w);
}

// Two units (32 bytes, 32-byte aligned) in one load.  What L1 does for a request follows the
// lines it touches: with 16-byte loads a group's four lanes asked for half a line at a time and
// L1 was 82% busy (similarity stage, R-MAT s22 at eps
// 0.2: 19.4 -> 17.9 ms; power law of 57M edges 1.65 -> 1.54).
struct UnitPair {
    uint4 lo, hi;
};

__device__ __forceinline__ UnitPair load_pair(const uint4* p) {
    UnitPair r;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r.lo.x), "=r"(r.lo.y), "=r"(r.lo.z), "=r"(r.lo.w), "=r"(r.hi.x), "=r"(r.hi.y), "=r"(r.hi.z), "=r"(r.hi.w)
        : "l"(p));
    return r;
}

__device__ __forceinline__ uint32_t missing_bits(const UnitPair& x, const UnitPair& y) {
    return missing_bits(x.lo, y.lo) + missing_bits(x.hi, y.hi);
}

// Warps take `chunk` consecutive edges at a time (*queue counts those beyond the first) and
// work through them in batches of kSketchBatch.  Lane i reads edge i's endpoints and their (base, degree) pairs, prunes it
// by the degrees and picks a bitmap size for what is left.  By that size:
//   * up to kSketchLaneLog: one edge per lane, its few units read by that lane;
//   * up to kSketchGroupLog: groups of G lanes take one edge each, compare 2 G U units at a
//     time until it is decided, and move on to the next;
//   * larger: the list of k_sketch_long, a warp per edge.  A hub's edges of this kind sit
//     together in its list (low ids in power-law graphs), and the few warps that drew them
//     would work on long after the others are done (power law, 57M edges: 4.35 -> 1.35 ms).
// An edge that its size leaves undecided is tried again at four times that, up to the lower
// endpoint's largest.
// A pivot's bitmaps are shared by its consecutive edges and stay in L1.
// sim[k] = kEdgePending for an edge the list kernels must count, 0 otherwise (decided: both
// predicates reject it).  The pending work of pivots above small_deg goes to pivot[v] and, in
// all, *total (see pending_work).
// ctr[0] += units read of the lower endpoints' bitmaps, ctr[1] += edges not pruned.
constexpr int kSketchBatch = 128;
// R-MAT s20 / s22, similarity stage: 4 lanes x 2 loads 0.48 / 1.83 ms, 4 x 1 0.51 / 1.96, 8 x 1
// 0.52 / 1.99, 2 x 4 0.50 / 1.95.
constexpr int kSketchGroup = 4, kSketchUnroll = 2;   // lanes; 32-byte loads of each bitmap in flight per lane
constexpr uint32_t kSketchLaneLog = 10;    // 8 units
constexpr uint32_t kSketchGroupLog = 15;   // 256 units

// List work of a pending edge: 1 + d_u / 64, so that a pivot's sum (at most its degree plus a
// 64th of the adjacency) stays below 2^32.
__device__ __forceinline__ uint32_t pending_work(uint32_t du) { return 1u + (du >> 6); }

struct PendingWork {
    uint32_t* pivot;                // n, zeroed: pending work per pivot above small_deg
    unsigned long long* total;
    uint32_t small_deg;
};

// Edge k found undecided after its bitmaps were read.
__device__ __forceinline__ uint32_t edge_pending(uint8_t* sim, const PendingWork& pw,
                                                 const uint32_t* __restrict__ lo_adj,
                                                 const uint32_t* __restrict__ lo_src, const uint2* __restrict__ info,
                                                 uint64_t k) {
    sim[k] = kEdgePending;
    const uint32_t v = lo_src[k];
    if (info[v].y <= pw.small_deg) return 0;
    const uint32_t w = pending_work(info[lo_adj[k]].y);
    atomicAdd(&pw.pivot[v], w);
    return w;
}

template <bool kPerGraph>
__global__ void __launch_bounds__(256, 4) k_sketch_filter(uint64_t E, const uint32_t* __restrict__ lo_adj,
                                                       const uint32_t* __restrict__ lo_src,
                                                       const uint2* __restrict__ info, const uint4* __restrict__ sk,
                                                       SketchLevels levels, CnPrune pr, uint32_t chunk, uint32_t* queue,
                                                       uint8_t* __restrict__ sim, PendingWork pw, LongEdges ll,
                                                       unsigned long long* __restrict__ ctr) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    constexpr int G = kSketchGroup, U = kSketchUnroll;
    constexpr uint32_t kGroups = 32 / G, kStep = 2 * G * U;
    static_assert(kStep <= (2u << (kSketchLaneLog - kSketchMinLog)), "a group step must not exceed its smallest bitmap");
    __shared__ SketchSlot slots[8][kSketchBatch];
    __shared__ SketchLevels lv;               // indexed by lane: shared memory, not a parameter
    if (threadIdx.x < kSketchClasses) lv.base[threadIdx.x] = levels.base[threadIdx.x];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, gl = lane % G, gi = lane / G;
    const uint32_t lower = (1u << lane) - 1u;
    SketchSlot* slot = slots[threadIdx.x >> 5];
    const uint64_t nchunks = (E + chunk - 1) / chunk;
    uint32_t words = 0, counted = 0, pending = 0;
    // A long edge for k_sketch_long; false when the list is full.
    auto defer = [&](const SketchSlot& s, uint64_t k, uint32_t at) {
        if (at >= ll.cap) return false;
        ll.slot[at] = make_uint4(s.ru, s.rv, s.need, s.code);
        ll.edge[at] = (uint32_t)k;
        return true;
    };
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);   // the first chunk is the warp's own
    while (c < nchunks) {
        const uint64_t kend = min((uint64_t)E, (uint64_t)(c + 1ull) * chunk);
        for (uint64_t kb = (uint64_t)c * chunk; kb < kend; kb += kSketchBatch) {
            uint32_t groups = 0, lanes = 0;   // slots for the groups from the front, for the lanes from the back
            // all loads of the batch first: two round trips for its 128 edges
            constexpr int kParts = kSketchBatch / 32;
            uint32_t us[kParts], vs[kParts];
            uint2 ius[kParts], ivs[kParts];
#pragma unroll
            for (int q = 0; q < kParts; ++q) {
                const uint64_t k = min(kb + 32 * q + lane, kend - 1);
                us[q] = __ldcs(lo_adj + k);
                vs[q] = __ldcs(lo_src + k);
            }
#pragma unroll
            for (int q = 0; q < kParts; ++q) {
                ius[q] = __ldg(info + us[q]);
                ivs[q] = __ldg(info + vs[q]);
            }
#pragma unroll
            for (int q = 0; q < kParts; ++q) {
                const uint64_t k = kb + 32 * q + lane;
                uint32_t l = 0;               // bitmap size, 0: none needed
                SketchSlot s{0, 0, 0, 0};
                if (k < kend) {
                    const uint32_t v = vs[q];
                    const uint2 iu = ius[q], iv = ivs[q];
                    float floor2 = pr.eps2_floor;
                    double eps = pr.eps;
                    if constexpr (kPerGraph) {
                        const PredParams* g = pr.gpp + pr.vgid[v];
                        floor2 = g->eps2_floor;
                        eps = g->eps;
                    }
                    PivotTests pt;
                    pt.np = 0;
                    pt.tscale = floor2 * (float)(iv.y + 1u);
                    uint8_t state = 0;
                    // A margin above the float roundings: at or below it both predicates' degree
                    // prune holds in exact arithmetic; an edge it misses only reads its bitmaps.
                    if ((float)(iu.y + 1u) >= pt.tscale * 0.999999f) {
                        ++counted;
                        const uint32_t tlo = count_floor(iu.y, iv.y, pt, eps);
                        if (tlo == 0) {
                            state = kEdgePending;              // any count may be similar
                        } else if (tlo <= iu.y) {
                            const int top = sketch_log(iu.y);
                            s.need = iu.y - tlo + 1;
                            if (iu.y >= 2) l = sketch_level(iu.y, iv.y, s.need, top);
                            if (l == 0) state = kEdgePending;
                            s.ru = iu.x;
                            s.rv = iv.x;
                            s.code = (32 * q + lane) | l << 8 | (uint32_t)top << 16;
                        }
                    }
                    sim[k] = state;
                    if (state && iv.y > pw.small_deg) {
                        const uint32_t w = pending_work(iu.y);
                        atomicAdd(&pw.pivot[v], w);
                        pending += w;
                    }
                }
                const uint32_t large = __ballot_sync(kFull, l > kSketchGroupLog);
                bool deferred = false;
                if (large) {
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(ll.count, __popc(large));
                    at = __shfl_sync(kFull, at, 0);
                    if (l > kSketchGroupLog) deferred = defer(s, k, at + __popc(large & lower));
                }
                const bool by_lane = l > 0 && l <= kSketchLaneLog, by_group = l > kSketchLaneLog && !deferred;
                const uint32_t ml = __ballot_sync(kFull, by_lane), mg = __ballot_sync(kFull, by_group);
                if (by_lane) slot[kSketchBatch - 1 - lanes - __popc(ml & lower)] = s;
                if (by_group) slot[groups + __popc(mg & lower)] = s;
                lanes += __popc(ml);
                groups += __popc(mg);
            }
            __syncwarp();
            for (uint32_t i = lane; i < lanes; i += 32) {
                const SketchSlot s = slot[kSketchBatch - 1 - i];
                uint32_t l = slot_level(s);
                const uint32_t top = slot_top(s);
                for (;;) {
                    const uint32_t units = 1u << (l - kSketchMinLog);
                    const uint4* pu = sk + sketch_unit(lv, l, s.ru);
                    const uint4* pv = sk + sketch_unit(lv, l, s.rv);
                    uint32_t miss = 0, pos = 0;
                    if (units == 1) {
                        miss = missing_bits(__ldg(pu), __ldg(pv));
                        pos = 1;
                    }
                    for (; pos < units && miss < s.need; pos += 2)
                        miss += missing_bits(load_pair(pu + pos), load_pair(pv + pos));
                    words += pos;
                    if (miss >= s.need) break;
                    if (l == top) {
                        pending += edge_pending(sim, pw, lo_adj, lo_src, info, kb + (s.code & 0xFFu));
                        break;
                    }
                    l = min(l + 2, top);
                }
            }
            if (groups) {
                uint32_t mine = gi, next = kGroups;        // slot of this group, first slot not taken
                bool on = mine < groups;
                SketchSlot s{0, 0, 0, 0};
                const uint4 *pu = sk, *pv = sk;
                uint32_t left = 0, miss = 0;               // units left at this size
                auto open = [&]() {
                    left = 1u << (slot_level(s) - kSketchMinLog);
                    pu = sk + sketch_unit(lv, slot_level(s), s.ru) + 2 * gl;
                    pv = sk + sketch_unit(lv, slot_level(s), s.rv) + 2 * gl;
                    miss = 0;
                };
                if (on) {
                    s = slot[mine];
                    open();
                }
                for (;;) {
                    uint32_t m = 0;
                    if (on) {
                        UnitPair x[U], y[U];
#pragma unroll
                        for (int q = 0; q < U; ++q) {
                            x[q] = load_pair(pu + 2 * q * G);
                            y[q] = load_pair(pv + 2 * q * G);
                        }
#pragma unroll
                        for (int q = 0; q < U; ++q) m += missing_bits(x[q], y[q]);
                    }
#pragma unroll
                    for (int o = G / 2; o > 0; o >>= 1) m += __shfl_xor_sync(kFull, m, o);
                    pu += kStep;
                    pv += kStep;
                    left -= kStep;
                    miss += m;
                    bool done = on && (miss >= s.need || left == 0);
                    if (!__any_sync(kFull, done)) continue;
                    if (done) {
                        if (gl == 0) words += (1u << (slot_level(s) - kSketchMinLog)) - left;
                        if (miss < s.need) {
                            const uint64_t k = kb + (s.code & 0xFFu);
                            if (slot_level(s) < slot_top(s)) {     // the size chosen was too coarse
                                s.code = (s.code & ~0xFF00u) | min(slot_level(s) + 2, slot_top(s)) << 8;
                                bool deferred = false;
                                if (slot_level(s) > kSketchGroupLog) {
                                    if (gl == 0) deferred = defer(s, k, atomicAdd(ll.count, 1u));
                                    deferred = __shfl_sync(((1u << G) - 1u) << (gi * G), deferred, gi * G);
                                }
                                if (!deferred) {
                                    open();
                                    done = false;
                                }
                            } else if (gl == 0) {
                                pending += edge_pending(sim, pw, lo_adj, lo_src, info, k);
                            }
                        }
                    }
                    // groups that finished take the next slots in group order
                    const uint32_t freed = __ballot_sync(kFull, done && gl == 0);
                    if (done) {
                        mine = next + __popc(freed & ((1u << (gi * G)) - 1u));
                        on = mine < groups;
                        if (on) {
                            s = slot[mine];
                            open();
                        }
                    }
                    next += __popc(freed);
                    if (!__any_sync(kFull, on)) break;
                }
            }
            __syncwarp();                                  // slots are rewritten by the next batch
        }
        if (lane == 0) c = nwarps + atomicAdd(queue, 1u);
        c = __shfl_sync(kFull, c, 0);
    }
    words = __reduce_add_sync(kFull, words);
    counted = __reduce_add_sync(kFull, counted);
    // 64 bits: a total short of the pivots' sums would be cut into more slices than fit
    const uint32_t pend_lo = __reduce_add_sync(kFull, pending & 0xFFFFu);
    const uint32_t pend_hi = __reduce_add_sync(kFull, pending >> 16);
    if (lane == 0 && (words | counted)) {
        atomicAdd(&ctr[0], (unsigned long long)words);
        atomicAdd(&ctr[1], (unsigned long long)counted);
        if (pend_lo | pend_hi) atomicAdd(pw.total, pend_lo + ((unsigned long long)pend_hi << 16));
    }
}

// The long edges, one per warp, 128 units at a time; a CTA's warps take consecutive ones,
// which mostly share their pivot and so its bitmaps in L1.
__global__ void __launch_bounds__(256) k_sketch_long(LongEdges ll, const uint32_t* __restrict__ lo_adj,
                                                     const uint32_t* __restrict__ lo_src,
                                                     const uint2* __restrict__ info, const uint4* __restrict__ sk,
                                                     SketchLevels lv, uint8_t* __restrict__ sim, PendingWork pw,
                                                     unsigned long long* __restrict__ ctr) {
    static_assert(kSketchGroupLog + 1 - kSketchMinLog >= 7, "a long edge has whole steps of 128 units");
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t count = min(*ll.count, ll.cap);
    uint32_t words = 0, pending = 0;
    const uint32_t step = gridDim.x * (blockDim.x >> 5);
    for (uint64_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < count; i += step) {
        const uint4 e = ll.slot[i];
        const SketchSlot s{e.x, e.y, e.z, e.w};
        for (uint32_t level = slot_level(s);; level = min(level + 2, slot_top(s))) {
            const uint32_t units = 1u << (level - kSketchMinLog);
            const uint4* pu = sk + sketch_unit(lv, level, s.ru) + 2 * lane;
            const uint4* pv = sk + sketch_unit(lv, level, s.rv) + 2 * lane;
            uint32_t miss = 0, left = units;
            do {
                UnitPair x[2], y[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    x[q] = load_pair(pu + 64 * q);
                    y[q] = load_pair(pv + 64 * q);
                }
                const uint32_t m = missing_bits(x[0], y[0]) + missing_bits(x[1], y[1]);
                miss += __reduce_add_sync(0xFFFFFFFFu, m);
                pu += 128;
                pv += 128;
                left -= 128;
            } while (left && miss < s.need);
            if (lane == 0) words += units - left;
            if (miss >= s.need) break;
            if (level == slot_top(s)) {
                if (lane == 0) pending += edge_pending(sim, pw, lo_adj, lo_src, info, ll.edge[i]);
                break;
            }
        }
    }
    if (lane == 0 && words) {
        atomicAdd(&ctr[0], (unsigned long long)words);
        if (pending) atomicAdd(pw.total, (unsigned long long)pending);
    }
}

// ---- pending edges of small pivots ------------------------------------------------------------

// What the sketches left open, from the edge states: four edges per lane, pending ones as bits.
__device__ __forceinline__ uint32_t pending_bits(const uint8_t* sim, uint64_t k, uint64_t E) {
    if (k >= E) return 0;
    // the scratch pads sim to 256 bytes; states: 0, 1, kEdgePending = 2
    const uint32_t p = (*reinterpret_cast<const uint32_t*>(sim + k) >> 1) & 0x01010101u;
    const uint32_t bits = (p | p >> 7 | p >> 14 | p >> 21) & 0xFu;
    return k + 4 > E ? bits & ((1u << (uint32_t)(E - k)) - 1u) : bits;
}

// The predicate of one pending edge with count t; lanes of a warp take different edges.
// Writes the edge's final state; the similar-degree counts are added by the caller's warp.
__device__ __forceinline__ bool settle_edge(const CnPrune& P, uint32_t t, uint32_t du, uint32_t dv,
                                            unsigned long long& nsim, unsigned long long& ndis) {
    const PivotTests pt{0, P.eps2_floor * (float)(dv + 1ull)};
    if (t < count_floor(du, dv, pt, P.eps)) return false;      // both predicates reject it
    const bool r = ref_f64_similar(t, du, dv, P.eps), x = exact_similar(t, du, dv, P.p, P.q);
    const bool s = P.mode ? r : x;
    ndis += r != x;
    nsim += s;
    return s;
}

__device__ __forceinline__ void add_similar(int32_t* sd, bool s, uint32_t u, uint32_t v, uint32_t lane) {
    if (s) atomicAdd(&sd[u], 1);
    const uint32_t peers = __match_any_sync(0xFFFFFFFFu, s ? v : kEmpty);
    if (s && (__ffs(peers) - 1) == (int)lane) atomicAdd(&sd[v], __popc(peers));
}

// Pending edges whose pivot has at most small_deg neighbours, in tiles of consecutive edges, so
// that those of one pivot come in runs.  A run of kTableRun edges and more is counted against
// a bucketed table of the pivot's list, a shorter one by binary search in the list itself
// (which stays in L1): either way groups of eight lanes take an edge each and read 32 entries
// of its lower list per round.  The predicate runs afterwards with an edge per lane, so its
// double arithmetic is not paid at an eighth of the width.
constexpr uint32_t kTableRun = 4;
constexpr int kSmallTile = 128;    // edges a warp takes at a time

template <bool kPerGraph>
__global__ void __launch_bounds__(256) k_cn_pending_small(uint64_t E, uint32_t small_deg,
                                                          const uint32_t* __restrict__ lo_adj,
                                                          const uint32_t* __restrict__ lo_src,
                                                          const uint32_t* __restrict__ off,
                                                          const uint32_t* __restrict__ adj, CnPrune pr,
                                                          uint8_t* sim, int32_t* sd, RunCounters* rc,
                                                          unsigned long long* ctr) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    __shared__ uint32_t slots[8][kSmallTile];      // edge within the tile | count << 16
    const uint32_t lane = threadIdx.x & 31, gl = lane & 7u, gi = lane >> 3, lower = (1u << lane) - 1u;
    __shared__ __align__(16) uint32_t tabs[8][4 * kSmallDeg];
    uint32_t* slot = slots[threadIdx.x >> 5];
    __shared__ uint8_t lones[8][kSmallTile];       // slots of the edges counted by search
    uint8_t* lone = lones[threadIdx.x >> 5];
    uint32_t* tab = tabs[threadIdx.x >> 5];
    uint4* tab4 = reinterpret_cast<uint4*>(tab);
    const uint64_t ntiles = (E + kSmallTile - 1) / kSmallTile;
    const uint64_t warp0 = blockIdx.x * (uint64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint64_t nwarps = gridDim.x * (uint64_t)(blockDim.x >> 5);
    unsigned long long nsim = 0, ndis = 0;
    uint32_t words = 0;
    for (uint64_t tile = warp0; tile < ntiles; tile += nwarps) {
        const uint64_t kb = tile * kSmallTile;
        uint32_t bits = pending_bits(sim, kb + 4 * lane, E);
        if (!__any_sync(kFull, bits)) continue;
        uint32_t incl = __popc(bits);
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, incl, s);
            if ((int)lane >= s) incl += y;
        }
        const uint32_t total = __shfl_sync(kFull, incl, 31);
        for (uint32_t at = incl - __popc(bits); bits; bits &= bits - 1, ++at) slot[at] = 4 * lane + __ffs(bits) - 1;
        __syncwarp();
        uint32_t nlone = 0;
        for (uint32_t at = 0; at < total; at += 32) {          // 32 slots; runs of one pivot within them
            const bool in = at + lane < total;
            const uint64_t k = kb + (in ? slot[at + lane] : 0u);
            const uint32_t v = in ? lo_src[k] : kEmpty;
            uint32_t vb = 0, dv = 0, ub = 0, ue = 0;
            if (in) {
                const uint32_t u = lo_adj[k];
                vb = off[v];
                dv = off[v + 1] - vb;
                ub = off[u];
                ue = off[u + 1];
            }
            const bool here = in && dv <= small_deg;
            const uint32_t before = __shfl_up_sync(kFull, v, 1);
            const uint32_t heads = __ballot_sync(kFull, lane == 0 || v != before);
            const uint32_t head = 31 - __clz(heads & (lower << 1 | 1u));
            const uint32_t rest = lane == 31 ? 0u : heads >> (lane + 1);
            const uint32_t end = rest ? lane + __ffs(rest) : 32u;
            const bool single = here && end - head < kTableRun;
            const uint32_t ms = __ballot_sync(kFull, single);
            if (single) lone[nlone + __popc(ms & lower)] = (uint8_t)(at + lane);
            nlone += __popc(ms);
            uint32_t mc = here ? 0u : 0xFFFFu;                 // 0xFFFF: not counted here
            uint32_t runs = __ballot_sync(kFull, here && !single && head == lane);
            while (runs) {
                const uint32_t h = __ffs(runs) - 1;
                runs &= runs - 1;
                const uint32_t stop = __shfl_sync(kFull, end, h), b0 = __shfl_sync(kFull, vb, h);
                const uint32_t d0 = __shfl_sync(kFull, dv, h);
                for (uint32_t i = lane; i < d0; i += 32) tab4[i] = make_uint4(kEmpty, kEmpty, kEmpty, kEmpty);
                __syncwarp();
                for (uint32_t i = lane; i < d0; i += 32) bucket_insert(tab, d0, __ldg(adj + b0 + i));
                __syncwarp();
                for (uint32_t j0 = h; j0 < stop; j0 += 4) {
                    const uint32_t j = min(j0 + gi, 31u);
                    const uint32_t b = __shfl_sync(kFull, ub, j), e = __shfl_sync(kFull, ue, j);
                    uint32_t c = 0;
                    if (j0 + gi < stop)
                        for (uint32_t p = (b & ~3u) + 4 * gl; p < e; p += 32) {
                            c += probe_word(__ldg(reinterpret_cast<const uint4*>(adj + p)), p, b, e, tab, d0);
                            ++words;
                        }
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
                    const uint32_t mine = __shfl_sync(kFull, c, 8 * ((lane - j0) & 3u));
                    if (lane - j0 < 4u && lane < stop) mc = mine;
                }
                __syncwarp();                                  // the table is rebuilt for the next run
            }
            if (in) slot[at + lane] |= mc << 16;
        }
        __syncwarp();
        for (uint32_t i0 = 0; i0 < nlone; i0 += 4) {
            const uint32_t i = i0 + gi;
            uint32_t c = 0;
            if (i < nlone) {
                const uint64_t k = kb + slot[lone[i]];
                const uint32_t u = lo_adj[k], v = lo_src[k];
                const uint32_t ub = off[u], ue = off[u + 1], vb = off[v], dv = off[v + 1] - vb;
                const uint32_t* list = adj + vb;
                const uint32_t half = 1u << (31 - __clz(dv));
                for (uint32_t p = (ub & ~3u) + 4 * gl; p < ue; p += 32) {
                    const uint4 x = __ldg(reinterpret_cast<const uint4*>(adj + p));
                    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
                    uint32_t n[4] = {0, 0, 0, 0};              // entries of the pivot known to be <= w
                    for (uint32_t s = half; s; s >>= 1) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (n[q] + s <= dv && __ldg(list + n[q] + s - 1) <= w[q]) n[q] += s;
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) c += p + q >= ub && p + q < ue && n[q] && __ldg(list + n[q] - 1) == w[q];
                    ++words;
                }
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
            if (i < nlone && gl == 0) slot[lone[i]] |= c << 16;
        }
        __syncwarp();
        for (uint32_t i0 = 0; i0 < total; i0 += 32) {
            const uint32_t i = i0 + lane;
            bool s = false;
            uint32_t u = 0, v = 0;
            if (i < total) {
                const uint32_t t = slot[i] >> 16;
                if (t != 0xFFFFu) {
                    const uint64_t k = kb + (slot[i] & 0xFFFFu);
                    u = lo_adj[k];
                    v = lo_src[k];
                    CnPrune Pg;
                    if constexpr (kPerGraph) Pg = prune_of_graph(pr, v);
                    const CnPrune& P = kPerGraph ? Pg : pr;
                    s = settle_edge(P, t, off[u + 1] - off[u], off[v + 1] - off[v], nsim, ndis);
                    sim[k] = s;
                }
            }
            add_similar(sd, s, u, v, lane);
        }
        __syncwarp();                                          // slots are rewritten by the next tile
    }
    fused_totals(FusedPred{sim, sd, rc, nullptr}, lane, nsim, ndis);
    words = __reduce_add_sync(kFull, words);
    if (lane == 0 && words) atomicAdd(&ctr[0], (unsigned long long)words);
}

// Plans with split pivots: the list kernels leave cn[] of the pending edges, whose predicate
// runs here (one byte per edge is read; k_predicate would read every edge, its count and both
// degrees: 1.03 ms on a power law of 57M edges).
__global__ void __launch_bounds__(256) k_predicate_pending(uint64_t E, const uint32_t* __restrict__ lo_adj,
                                                           const uint32_t* __restrict__ lo_src,
                                                           const uint32_t* __restrict__ off,
                                                           const uint32_t* __restrict__ cn, CnPrune pr, uint8_t* sim,
                                                           int32_t* sd, RunCounters* rc) {
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long nsim = 0, ndis = 0;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x * 4;
    for (uint64_t k0 = ((uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) * 4; k0 < E; k0 += step) {
        const uint64_t kb = k0 + 4 * lane;
        uint32_t bits = pending_bits(sim, kb, E);
        while (__any_sync(0xFFFFFFFFu, bits)) {
            bool s = false;
            uint32_t u = 0, v = 0;
            if (bits) {
                const uint64_t k = kb + __ffs(bits) - 1;
                bits &= bits - 1;
                u = lo_adj[k];
                v = lo_src[k];
                s = settle_edge(pr, cn[k], off[u + 1] - off[u], off[v + 1] - off[v], nsim, ndis);
                sim[k] = s;
            }
            add_similar(sd, s, u, v, lane);
        }
    }
    fused_totals(FusedPred{sim, sd, rc, nullptr}, lane, nsim, ndis);
}

// ---- pending edges of larger pivots -----------------------------------------------------------

// The pending edges of every task of the plan, gathered at the task's place in edges[] (of E
// entries), and the task cut into slices of about equal pending work: the plan's tasks are
// sized for counting every edge, so a hub's few pending edges would be sought among all of
// its edges and keep one CTA busy after the others are done.  Per task list, entries of
// TaskPick::order; counts[c] hash class c, counts[kNumBigClasses] the hubs.
constexpr int kPendingLists = kNumBigClasses + 1;
struct PendingLists {
    const CnTask* tasks[kPendingLists];
    uint32_t count[kPendingLists];
    TaskSlice* out[kPendingLists];            // count + kPendingSlices per SM entries
};

// Sum of the lanes before this one, and of all.
__device__ __forceinline__ uint32_t warp_exclusive(uint32_t n, uint32_t lane, uint32_t* total) {
    uint32_t incl = n;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, s);
        if (lane >= (uint32_t)s) incl += y;
    }
    *total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    return incl - n;
}

// The pending edges of [e0, e1) in order to edges[e0...]; returns their number.  In order: the
// chunk tasks of a split pivot gather the same edges at the same place, perhaps at the same
// time.
__device__ __forceinline__ uint32_t gather_pending_warp(const uint8_t* sim, uint32_t e0, uint32_t e1,
                                                        uint32_t* __restrict__ edges, uint32_t lane) {
    uint32_t found = 0;
    for (uint64_t s0 = e0 & ~3ull; s0 < e1; s0 += 128) {
        const uint64_t k = s0 + 4 * lane;
        uint32_t bits = pending_bits(sim, k, e1);
        if (k < e0) bits &= 0xFu << (e0 - (uint32_t)k);    // the first word may start before the task
        uint32_t total;
        uint32_t at = e0 + found + warp_exclusive(__popc(bits), lane, &total);
        for (; bits; bits &= bits - 1) edges[at++] = (uint32_t)k + __ffs(bits) - 1;
        found += total;
    }
    return found;
}

__device__ __forceinline__ uint32_t gather_pending_cta(const uint8_t* sim, uint32_t e0, uint32_t e1,
                                                       uint32_t* __restrict__ edges, uint32_t lane,
                                                       uint32_t* warp_sums) {
    uint32_t found = 0;
    const uint32_t wib = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (uint64_t s0 = e0 & ~15ull; s0 < e1; s0 += 16ull * blockDim.x) {
        const uint64_t k = s0 + 16ull * threadIdx.x;
        uint32_t bits = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) bits |= pending_bits(sim, k + 4 * q, e1) << (4 * q);
        if (k < e0) bits &= 0xFFFFu << (e0 - (uint32_t)k);
        uint32_t total;
        const uint32_t before = warp_exclusive(__popc(bits), lane, &total);
        if (lane == 0) warp_sums[wib] = total;
        __syncthreads();
        uint32_t at = e0 + found + before;
        for (uint32_t w = 0; w < warps; ++w) {
            if (w < wib) at += warp_sums[w];
            found += warp_sums[w];
        }
        for (; bits; bits &= bits - 1) edges[at++] = (uint32_t)k + __ffs(bits) - 1;
        __syncthreads();
    }
    return found;
}

// Lists of hubs and of the largest class: a CTA per task; the others: a warp per task.
__global__ void __launch_bounds__(256) k_pending_tasks(PendingLists pl, PendingWork pw,
                                                       const uint32_t* __restrict__ off,
                                                       const uint32_t* __restrict__ lo_off, const uint8_t* sim,
                                                       uint32_t slices, uint32_t* __restrict__ edges,
                                                       uint32_t* __restrict__ counts) {
    __shared__ uint32_t warp_sums[8], place;
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint64_t even = pending_even(*pw.total, slices);
    auto cut = [&](const CnTask& t, uint32_t work, uint32_t found) {
        const uint32_t dv = off[t.v + 1] - off[t.v], all = lo_off[t.v + 1] - lo_off[t.v];
        return pending_slices(even, work, t.e1 - t.e0, all, t.chunked ? t.ce - t.cb : dv, dv, found);
    };
    for (int a = 2; a < kPendingLists; ++a)
        for (uint32_t i = blockIdx.x; i < pl.count[a]; i += gridDim.x) {
            const CnTask t = pl.tasks[a][i];
            const uint32_t work = pw.pivot[t.v];
            if (!work) continue;                                             // the same in every thread
            const uint32_t found = gather_pending_cta(sim, t.e0, t.e1, edges, lane, warp_sums);
            const uint32_t n = cut(t, work, found);
            if (threadIdx.x == 0 && n) place = atomicAdd(&counts[a], n);
            __syncthreads();
            for (uint32_t q = threadIdx.x; q < n; q += blockDim.x) pl.out[a][place + q] = TaskSlice{i, q, n, found};
            __syncthreads();
        }
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + wib, warps = gridDim.x * (blockDim.x >> 5);
    for (int a = 0; a < 2; ++a)
        for (uint32_t i = warp; i < pl.count[a]; i += warps) {
            const CnTask t = pl.tasks[a][i];
            const uint32_t work = pw.pivot[t.v];
            if (!work) continue;
            const uint32_t found = gather_pending_warp(sim, t.e0, t.e1, edges, lane);
            const uint32_t n = cut(t, work, found);
            uint32_t at = 0;
            if (lane == 0 && n) at = atomicAdd(&counts[a], n);
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            for (uint32_t q = lane; q < n; q += 32) pl.out[a][at + q] = TaskSlice{i, q, n, found};
        }
}

}  // namespace scan
