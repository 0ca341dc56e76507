// From common-neighbour counts to clusters: predicate, cores, union-find, attachment,
// hub/outlier classification.  All passes are edge-parallel over the E undirected edges
// (lo_adj/lo_src) or vertex-parallel; per-vertex arrays (n x 4 B) stay L2-resident.
#pragma once

#include "device_common.cuh"
#include "predicate.cuh"

namespace scan {

// sim[e] and the similar-degree count sd[] of both endpoints (core rule: a vertex is a
// core when at least mu of its neighbours are similar, GPUSCAN++/GPUScan.cu:147-165).
// Edges of one pivot are contiguous, so the pivot side is summed per warp segment.
// Batched runs (many graphs as one disjoint union) pass vgid[] (graph of each vertex) and
// per-graph parameters gpp[]; single runs pass null and use pp.
__global__ void k_predicate(uint64_t E, const uint32_t* __restrict__ lo_adj, const uint32_t* __restrict__ lo_src,
                            const uint32_t* __restrict__ off, const uint32_t* __restrict__ cn, PredParams pp,
                            const uint32_t* __restrict__ vgid, const PredParams* __restrict__ gpp,
                            uint8_t* __restrict__ sim, int32_t* __restrict__ sd, RunCounters* __restrict__ ctr) {
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long nsim = 0, ndis = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t e0 = (uint64_t)blockIdx.x * blockDim.x; e0 < E; e0 += stride) {
        const uint64_t e = e0 + threadIdx.x;
        bool s = false;
        uint32_t v = kEmpty;
        if (e < E) {
            const uint32_t u = lo_adj[e];
            v = lo_src[e];
            const uint32_t du = off[u + 1] - off[u], dv = off[v + 1] - off[v];
            const uint32_t t = cn[e];
            const PredParams P = vgid ? gpp[vgid[u]] : pp;
            const bool r = ref_f64_similar(t, du, dv, P.eps);
            const bool x = exact_similar(t, du, dv, P.p, P.q);
            s = P.mode ? r : x;
            ndis += (r != x);
            nsim += s;
            sim[e] = s;
            if (s) atomicAdd(&sd[u], 1);
        }
        // pivot side: one atomic per run of equal pivots within the warp
        const uint32_t key = s ? v : kEmpty;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
        if (s && (__ffs(peers) - 1) == (int)lane) atomicAdd(&sd[v], __popc(peers));
    }
    for (int o = 16; o > 0; o >>= 1) {
        nsim += __shfl_xor_sync(0xFFFFFFFFu, nsim, o);
        ndis += __shfl_xor_sync(0xFFFFFFFFu, ndis, o);
    }
    if (lane == 0) {
        if (nsim) atomicAdd(&ctr->similar_edges, nsim);
        if (ndis) atomicAdd(&ctr->disagreements, ndis);
    }
}

// Served queries on cached counts: each edge's similarity threshold, precomputed once per
// graph, so the predicate is one compare per edge.  Edge e is similar at eps exactly when
// eps^2 <= tau(e): tau_x = (t+2)^2 / ((du+1)(dv+1)) for the exact test, tau_r =
// min((du+1)/(dv+1), max(4, t2)/((du+1)(dv+1))) for the reference's doubles: its 'N' prune,
// then its 'Y' prune or its intersect test (t2 the int square, which can wrap negative; the
// 'Y' threshold 4/((du+1)(dv+1)) still holds then).  Both are monotone in eps because IEEE
// products are.  Stored as floats; an edge whose tau lies within a relative kTauBand of
// eps^2 (float rounding is 6e-8) is decided by the predicate itself.
constexpr double kTauBand = 1e-6;

__global__ void k_tau(uint64_t E, const uint32_t* __restrict__ lo_adj, const uint32_t* __restrict__ lo_src,
                      const uint32_t* __restrict__ off, const uint32_t* __restrict__ cn, float* __restrict__ tau) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t u = lo_adj[e], v = lo_src[e];
        const uint32_t du = off[u + 1] - off[u], dv = off[v + 1] - off[v], t = cn[e];
        const double du1 = (double)(du + 1u), dv1 = (double)(dv + 1u);
        const double a = (double)(t + 2u);
        tau[e] = (float)(a * a / (du1 * dv1));
        const int32_t t2 = (int32_t)((t + 2u) * (t + 2u));
        tau[E + e] = (float)fmin(du1 / dv1, fmax(4.0, (double)t2) / (du1 * dv1));
    }
}

// The threads that share a pass: this one's index among them (a multiple of 32 for lane 0) and
// their number.  Each pass is a function of these, so that the kernels below run it over a grid
// and k_cluster_small over one thread-block cluster.  Arrays that another pass writes carry no
// __restrict__: in the fused kernel a non-coherent load could miss the write.
struct Team {
    uint64_t index, size;
};
__device__ __forceinline__ Team grid_team() {
    return Team{blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, (uint64_t)gridDim.x * blockDim.x};
}

// k_predicate for a served graph: the cached thresholds decide every edge outside the
// band; the disagreement counter is not kept (the server does not report it).
__device__ __forceinline__ void predicate_tau_pass(Team team, uint64_t E, const uint32_t* __restrict__ lo_adj,
                                                   const uint32_t* __restrict__ lo_src,
                                                   const uint32_t* __restrict__ off, const uint32_t* __restrict__ cn,
                                                   const float* __restrict__ tau, const PredParams& pp, uint8_t* sim,
                                                   int32_t* sd, RunCounters* ctr) {
    const uint32_t lane = threadIdx.x & 31;
    const float* tm = tau + (pp.mode ? E : 0);
    double theta;
    if (pp.mode) theta = pp.eps * pp.eps;
    else theta = pp.q == 0 ? 2.0 : ((double)pp.p / (double)pp.q) * ((double)pp.p / (double)pp.q);
    const double hi = theta * (1.0 + kTauBand), lo = theta * (1.0 - kTauBand);
    unsigned long long nsim = 0;
    for (uint64_t e0 = team.index - lane; e0 < E; e0 += team.size) {
        const uint64_t e = e0 + lane;
        bool s = false;
        uint32_t v = kEmpty;
        if (e < E) {
            const double tv = (double)tm[e];
            if (tv >= hi) {
                s = true;
            } else if (tv > lo || (theta == 0.0 && tv == 0.0)) {
                const uint32_t u = lo_adj[e], w = lo_src[e];
                const uint32_t du = off[u + 1] - off[u], dw = off[w + 1] - off[w];
                s = pp.mode ? ref_f64_similar(cn[e], du, dw, pp.eps) : exact_similar(cn[e], du, dw, pp.p, pp.q);
            }
            sim[e] = s;
            if (s) {
                v = lo_src[e];
                atomicAdd(&sd[lo_adj[e]], 1);
                ++nsim;
            }
        }
        const uint32_t key = s ? v : kEmpty;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, key);
        if (s && (__ffs(peers) - 1) == (int)lane) atomicAdd(&sd[v], __popc(peers));
    }
    for (int o = 16; o > 0; o >>= 1) nsim += __shfl_xor_sync(0xFFFFFFFFu, nsim, o);
    if (lane == 0 && nsim) atomicAdd(&ctr->similar_edges, nsim);
}

__global__ void k_predicate_tau(uint64_t E, const uint32_t* __restrict__ lo_adj, const uint32_t* __restrict__ lo_src,
                                const uint32_t* __restrict__ off, const uint32_t* __restrict__ cn,
                                const float* __restrict__ tau, PredParams pp, uint8_t* __restrict__ sim,
                                int32_t* __restrict__ sd, RunCounters* __restrict__ ctr) {
    predicate_tau_pass(grid_team(), E, lo_adj, lo_src, off, cn, tau, pp, sim, sd, ctr);
}

// parent[v] = v for cores, -1 otherwise; border/neighbour label ranges reset.  Batched
// runs pass vgid[] and per-graph gmu[].
__device__ __forceinline__ void core_init_pass(Team team, uint32_t n, const int32_t* sd, int mu, const uint32_t* __restrict__ vgid,
                                               const int32_t* __restrict__ gmu, int32_t* parent, int32_t* bmin,
                                               int32_t* bmax, int32_t* nmin, int32_t* nmax, RunCounters* ctr) {
    bool core = false;
    for (uint64_t v = team.index; v < n; v += team.size) {
        const int m = vgid ? gmu[vgid[v]] : mu;
        const bool c = sd[v] >= m;
        core |= c;
        parent[v] = c ? (int32_t)v : -1;
        bmin[v] = 0x7FFFFFFF;
        bmax[v] = -1;
        nmin[v] = 0x7FFFFFFF;
        nmax[v] = -1;
    }
    if (__any_sync(0xFFFFFFFFu, core) && (threadIdx.x & 31) == 0) atomicOr(&ctr->any_core, 1u);
}
__global__ void k_core_init(uint32_t n, const int32_t* __restrict__ sd, int mu, const uint32_t* __restrict__ vgid,
                            const int32_t* __restrict__ gmu, int32_t* __restrict__ parent, int32_t* __restrict__ bmin,
                            int32_t* __restrict__ bmax, int32_t* __restrict__ nmin, int32_t* __restrict__ nmax,
                            RunCounters* __restrict__ ctr) {
    core_init_pass(grid_team(), n, sd, mu, vgid, gmu, parent, bmin, bmax, nmin, nmax, ctr);
}

// Root of x with path halving.  parent[y] < y for every non-root y, so every write keeps
// the forest acyclic and the walk terminates.
__device__ __forceinline__ int32_t uf_find(volatile int32_t* parent, int32_t x) {
    int32_t p = parent[x];
    while (p != x) {
        const int32_t g = parent[p];
        if (g != p) parent[x] = g;
        x = p;
        p = g;
    }
    return x;
}

// Lock-free union by smaller root id: the root of a component is its smallest core id,
// which is the reference's cluster id (GPUSCAN++/GPUScan.cu:500-523 hooks the larger
// root under the smaller one).  At most `limit` CAS attempts; false if they all lost.
__device__ __forceinline__ bool uf_union(int32_t* parent, int32_t a, int32_t b, uint32_t limit) {
    volatile int32_t* vp = parent;
    for (uint32_t it = 0; it < limit; ++it) {
        a = uf_find(vp, a);
        b = uf_find(vp, b);
        if (a == b) return true;
        if (a < b) { const int32_t t = a; a = b; b = t; }   // a > b: hang a under b
        if (atomicCAS(&parent[a], a, b) == a) return true;
    }
    return false;
}

// The similar ones of the W edges from k on as bits.  W = 4 (k a multiple of 4; the scratch pads
// sim to 256 bytes): most edges of a sparse result are not similar, four per load and test (R-MAT
// s22, mu 2: unions 107 -> 38 us, borders 104 -> 38).  W = 1 in the fused kernel, whose threads
// would work through their four edges one after the other.
template <int W>
__device__ __forceinline__ uint32_t similar_bits(const uint8_t* sim, uint64_t k, uint64_t E) {
    if (k >= E) return 0;
    if constexpr (W == 1) return sim[k];
    const uint32_t p = *reinterpret_cast<const uint32_t*>(sim + k) & 0x01010101u;   // 0 or 1 each by now
    const uint32_t bits = (p | p >> 7 | p >> 14 | p >> 21) & 0xFu;
    return k + 4 > E ? bits & ((1u << (uint32_t)(E - k)) - 1u) : bits;
}

// Edges of one pivot v are consecutive, so a warp holds runs of them.  Hanging v's root under
// each lower neighbour's in turn would let one CAS per round succeed; instead the lanes of a
// run agree on the smallest of their roots and hang their own root under that (all different
// words), the first lane v's root as well.  Edges whose endpoints already point to one vertex
// end after two loads, and since L1 may keep a pointer from before the unions, after two from
// L2.  Cluster stage of communities of 6M edges 0.50 -> 0.30 ms.
//
// A warp takes 32 W edges: where many of them are similar in turns of 32 consecutive ones, else
// in turns of each lane's next.  (Each lane's next throughout: grid of 2000 x 2000 at eps 0.2
// 1.4-1.7 ms, now 0.8.)
//
// Of the tiles of 32 W edges, every `every`-th is visited.
template <int W>
__device__ __forceinline__ void union_pass(Team team, uint64_t E, const uint32_t* __restrict__ lo_adj,
                                           const uint32_t* __restrict__ lo_src, const uint8_t* sim, int32_t* parent,
                                           RunCounters* ctr, uint32_t limit, uint32_t every) {
    if (!*(volatile uint32_t*)&ctr->any_core) return;   // no core: nothing to join
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t e0 = W * (team.index - lane) * every; e0 < E; e0 += W * team.size * every) {
        uint32_t bits = similar_bits<W>(sim, e0 + W * lane, E);
        const uint32_t most = __reduce_max_sync(kFull, (uint32_t)__popc(bits));
        const bool dense = most > 2;
        for (uint32_t q = 0; q < (dense ? (uint32_t)W : most); ++q) {
            uint32_t i = W * lane + __ffs(bits) - 1;     // this lane's edge of the turn
            bool mine = bits != 0;
            if (dense) {
                i = 32 * q + lane;
                mine = __shfl_sync(kFull, bits, i / W) >> (i % W) & 1u;
            } else {
                bits &= bits - 1;
            }
            int32_t u = 0, v = 0;
            bool join = false;
            if (mine) {
                const uint64_t e = e0 + i;
                u = (int32_t)lo_adj[e];
                v = (int32_t)lo_src[e];
                const int32_t pu = parent[u], pv = parent[v];
                join = pu >= 0 && pv >= 0 && pu != pv;      // core-core only (cores never change)
                if (join) {
                    const volatile int32_t* vp = parent;
                    join = vp[u] != vp[v];
                }
            }
            if (!__any_sync(kFull, join)) continue;
            if (join) {
                u = uf_find(parent, u);
                const int32_t rv = uf_find(parent, v);
                join = u != rv;
            }
            const uint32_t run = __match_any_sync(kFull, join ? (uint32_t)v : kEmpty);
            if (join) {
                const bool first = (__ffs(run) - 1) == (int)lane;
                const int32_t rv = uf_find(parent, v);
                const int32_t m = (int32_t)__reduce_min_sync(run, (uint32_t)min(u, rv));
                bool ok = u == m || uf_union(parent, u, m, limit);
                if (first && rv != m) ok &= uf_union(parent, rv, m, limit);
                if (!ok) atomicOr(&ctr->error_flags, kErrUnionFindLimit);
            }
        }
    }
}
__global__ void k_union(uint64_t E, const uint32_t* __restrict__ lo_adj, const uint32_t* __restrict__ lo_src,
                        const uint8_t* __restrict__ sim, int32_t* parent, RunCounters* ctr, uint32_t limit) {
    union_pass<4>(grid_team(), E, lo_adj, lo_src, sim, parent, ctr, limit, 1);
}

// A sample of the edges, before the others.  When a run starts every core is its own root, and
// where most cores belong to one cluster all resident warps then swing the same few pointers:
// the fewer the edges, the more of them do so at once (served query at eps 0.2 on R-MAT of 213K
// edges 70-330 us of unions, of 15.7M 40-180; complete graph of 1,500 vertices 140-370).  A
// sample of few warps joins most of such a cluster, and the others find it joined (31, 41-60
// and 50-75 us, both launches).  Where there is no such cluster it costs its launch, about 3 us,
// and where the cores form small clusters up to 10 (run on communities of 6M edges 843 -> 858
// us): served queries, whose unions are most of their time, take it, runs do not.
constexpr uint64_t kUnionSample = 1u << 15;      // edges; 2^17 is no faster and costs up to 25 us where nothing contends
constexpr uint32_t kUnionSampleLeast = 16;       // at most every 16th tile
__global__ void k_union_sample(uint64_t E, const uint32_t* __restrict__ lo_adj, const uint32_t* __restrict__ lo_src,
                               const uint8_t* __restrict__ sim, int32_t* parent, RunCounters* ctr, uint32_t limit,
                               uint32_t every) {
    union_pass<1>(grid_team(), E, lo_adj, lo_src, sim, parent, ctr, limit, every);
}

// Flatten by pointer jumping: a round moves parent[v] of every core up to kJumpSteps ancestors on
// and raises flags[r] if any pointer moved, so the distance a pointer spans grows by that
// factor per round.  The host queues enough rounds for any depth (ceil(log16 n) + 2: eight for
// 4M vertices, where steps of one took 24 launches); a round whose predecessor moved nothing
// returns at once, so the pass needs no host synchronisation.  Every value stored is an ancestor of v in the final
// forest and only v's own thread writes parent[v], so concurrent jumps never undo one
// another.  (A find with path halving would not be safe here: its halving store can
// overwrite a vertex whose root another thread has just written with an intermediate
// ancestor.)
constexpr int kJumpSteps = 16;

// The ancestor of v up to kJumpSteps beyond p = parent[v], or its root.
__device__ __forceinline__ int32_t jump_target(const volatile int32_t* parent, int32_t p) {
    for (int i = 0; i < kJumpSteps; ++i) {
        const int32_t g = parent[p];
        if (g == p) break;
        p = g;
    }
    return p;
}


__device__ __forceinline__ uint32_t jump_pass(Team team, uint32_t n, int32_t* parent) {
    volatile int32_t* vp = parent;
    uint32_t ch = 0;
    for (uint64_t v = team.index; v < n; v += team.size) {
        const int32_t p = vp[v];
        if (p < 0) continue;
        const int32_t g = jump_target(vp, p);
        if (g != p) {
            vp[v] = g;
            ch = 1;
        }
    }
    return ch;
}

__global__ void k_jump_round(uint32_t n, int32_t* parent, uint32_t* flags, uint32_t round) {
    if (round > 0 && *(volatile uint32_t*)&flags[round - 1] == 0) return;
    const uint32_t ch = jump_pass(grid_team(), n, parent);
    if (__any_sync(0xFFFFFFFFu, ch) && (threadIdx.x & 31) == 0) atomicOr(&flags[round], 1u);
}

// The same rounds in one CTA, for graphs of up to kJumpBlockMax vertices: a block barrier
// separates the rounds, so one launch replaces the chain of k_jump_round launches (the
// launch count matters for the many small queries of the serving loop).  flags follow the
// chain's convention: flags[i] != 0 when round i moved a pointer, so flags[rounds - 1] == 0
// means converged.
constexpr uint32_t kJumpBlockMax = 1u << 16;

__global__ void __launch_bounds__(1024) k_jump_block(uint32_t n, int32_t* parent, uint32_t* flags, uint32_t rounds) {
    constexpr int kPer = 8;
    volatile int32_t* vp = parent;
    for (uint32_t round = 0; round < rounds; ++round) {
        int ch = 0;
        for (uint32_t v0 = threadIdx.x; v0 < n; v0 += kPer * blockDim.x) {   // loads of kPer vertices in flight
            int32_t p[kPer], g[kPer];
#pragma unroll
            for (int q = 0; q < kPer; ++q) p[q] = v0 + q * blockDim.x < n ? vp[v0 + q * blockDim.x] : -1;
#pragma unroll
            for (int q = 0; q < kPer; ++q) g[q] = p[q] < 0 ? p[q] : vp[p[q]];
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if (g[q] != p[q]) {
                    vp[v0 + q * blockDim.x] = jump_target(vp, g[q]);
                    ch = 1;
                }
        }
        ch = __syncthreads_or(ch);
        if (threadIdx.x == 0) flags[round] = ch ? 1u : 0u;
        if (!ch) break;
    }
}

// Border attachment: a non-core similar to a core joins that core's cluster.  The
// reference keeps the last write among several clusters (GPUSCAN++/GPUScan.cu:716,722);
// here the smallest cluster id wins, and bmin != bmax marks a multi-cluster border.
template <int W>
__device__ __forceinline__ void attach_pass(Team team, uint64_t E, const uint32_t* __restrict__ lo_adj,
                                            const uint32_t* __restrict__ lo_src, const uint8_t* sim,
                                            const int32_t* parent, int32_t* bmin, int32_t* bmax,
                                            const RunCounters* ctr) {
    if (!*(const volatile uint32_t*)&ctr->any_core) return;   // no core: no border
    for (uint64_t e0 = W * team.index; e0 < E; e0 += W * team.size)
        for (uint32_t bits = similar_bits<W>(sim, e0, E); bits; bits &= bits - 1) {
            const uint64_t e = e0 + __ffs(bits) - 1;
            const uint32_t u = lo_adj[e], v = lo_src[e];
            const int32_t pu = parent[u], pv = parent[v];
            if (pu >= 0 && pv < 0) { atomicMin(&bmin[v], pu); atomicMax(&bmax[v], pu); }
            else if (pv >= 0 && pu < 0) { atomicMin(&bmin[u], pv); atomicMax(&bmax[u], pv); }
        }
}
__global__ void k_attach(uint64_t E, const uint32_t* __restrict__ lo_adj, const uint32_t* __restrict__ lo_src,
                         const uint8_t* __restrict__ sim, const int32_t* __restrict__ parent,
                         int32_t* __restrict__ bmin, int32_t* __restrict__ bmax, const RunCounters* ctr) {
    attach_pass<4>(grid_team(), E, lo_adj, lo_src, sim, parent, bmin, bmax, ctr);
}

// Label after attachment: cluster id for cores and borders, -2 for the rest.
__device__ __forceinline__ void label_pass(Team team, uint32_t n, const int32_t* parent, const int32_t* bmin, int32_t* lab,
                                           RunCounters* ctr) {
    bool member = false;
    for (uint64_t v = team.index; v < n; v += team.size) {
        const int32_t p = parent[v];
        const int32_t l = p >= 0 ? p : (bmin[v] != 0x7FFFFFFF ? bmin[v] : -2);
        lab[v] = l;
        member |= l >= 0;
    }
    if (__any_sync(0xFFFFFFFFu, member) && (threadIdx.x & 31) == 0) atomicOr(&ctr->any_member, 1u);
}
__global__ void k_label(uint32_t n, const int32_t* __restrict__ parent, const int32_t* __restrict__ bmin,
                        int32_t* __restrict__ lab, RunCounters* __restrict__ ctr) {
    label_pass(grid_team(), n, parent, bmin, lab, ctr);
}

// Hub test inputs: for each unlabelled vertex, the smallest and largest label among its
// neighbours.  Two distinct labels make it a hub (GPUSCAN++/GPUScan.cu:757-780 looks for a
// second neighbour label different from the first).
__device__ __forceinline__ void neighbour_labels_pass(Team team, uint64_t E, const uint32_t* __restrict__ lo_adj,
                                                      const uint32_t* __restrict__ lo_src, const int32_t* lab,
                                                      int32_t* nmin, int32_t* nmax, const RunCounters* ctr) {
    if (!*(const volatile uint32_t*)&ctr->any_member) return;   // no cluster: every other vertex is an outlier
    for (uint64_t e = team.index; e < E; e += team.size) {
        const uint32_t u = lo_adj[e], v = lo_src[e];
        const int32_t lu = lab[u], lv = lab[v];
        if (lu < 0 && lv >= 0) { atomicMin(&nmin[u], lv); atomicMax(&nmax[u], lv); }
        else if (lv < 0 && lu >= 0) { atomicMin(&nmin[v], lu); atomicMax(&nmax[v], lu); }
    }
}
__global__ void k_neighbour_labels(uint64_t E, const uint32_t* __restrict__ lo_adj,
                                   const uint32_t* __restrict__ lo_src, const int32_t* __restrict__ lab,
                                   int32_t* __restrict__ nmin, int32_t* __restrict__ nmax, const RunCounters* ctr) {
    neighbour_labels_pass(grid_team(), E, lo_adj, lo_src, lab, nmin, nmax, ctr);
}

// Final labels, roles and counters.
__device__ __forceinline__ void finalize_pass(Team team, uint32_t n, const int32_t* parent, const int32_t* bmin,
                                              const int32_t* bmax, const int32_t* nmin, const int32_t* nmax,
                                              int32_t* label, uint8_t* role,
                                              const unsigned long long* __restrict__ stage, RunCounters* ctr) {
    if (team.index == 0) {   // so that one copy brings every counter back
        ctr->list_words = stage[0];
        ctr->edges_counted = stage[1];
    }
    unsigned long long c_core = 0, c_clu = 0, c_hub = 0, c_out = 0, c_bor = 0, c_multi = 0;
    for (uint64_t v = team.index; v < n; v += team.size) {
        const int32_t p = parent[v];
        int32_t l;
        uint8_t r;
        if (p >= 0) {
            l = p; r = kRoleCore; ++c_core; c_clu += (p == (int32_t)v);
        } else if (bmin[v] != 0x7FFFFFFF) {
            l = bmin[v]; r = kRoleBorder; ++c_bor; c_multi += (bmin[v] != bmax[v]);
        } else if (nmin[v] < nmax[v]) {
            l = -1; r = kRoleHub; ++c_hub;
        } else {
            l = -2; r = kRoleOutlier; ++c_out;
        }
        label[v] = l;
        if (role) role[v] = r;
    }
    for (int o = 16; o > 0; o >>= 1) {
        c_core += __shfl_xor_sync(0xFFFFFFFFu, c_core, o);
        c_clu += __shfl_xor_sync(0xFFFFFFFFu, c_clu, o);
        c_hub += __shfl_xor_sync(0xFFFFFFFFu, c_hub, o);
        c_out += __shfl_xor_sync(0xFFFFFFFFu, c_out, o);
        c_bor += __shfl_xor_sync(0xFFFFFFFFu, c_bor, o);
        c_multi += __shfl_xor_sync(0xFFFFFFFFu, c_multi, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (c_core) atomicAdd(&ctr->cores, c_core);
        if (c_clu) atomicAdd(&ctr->clusters, c_clu);
        if (c_hub) atomicAdd(&ctr->hubs, c_hub);
        if (c_out) atomicAdd(&ctr->outliers, c_out);
        if (c_bor) atomicAdd(&ctr->borders, c_bor);
        if (c_multi) atomicAdd(&ctr->multi_borders, c_multi);
    }
}
__global__ void k_finalize(uint32_t n, const int32_t* __restrict__ parent, const int32_t* __restrict__ bmin,
                           const int32_t* __restrict__ bmax, const int32_t* __restrict__ nmin,
                           const int32_t* __restrict__ nmax, int32_t* __restrict__ label,
                           uint8_t* __restrict__ role, const unsigned long long* __restrict__ stage,
                           RunCounters* __restrict__ ctr) {
    finalize_pass(grid_team(), n, parent, bmin, bmax, nmin, nmax, label, role, stage, ctr);
}

// The whole cluster stage of a small graph as one launch over one cluster of eight CTAs: what
// bounds it there is the chain of eight to sixteen dependent launches, and the hardware's
// cluster barrier between the passes costs about a microsecond.  A run of 10K edges spends 22 us
// here instead of 35; from about 80K edges eight SMs take longer over the edges than the launches
// do (communities: 148 us a run by launches, 171 fused).  A served query also has the predicate
// over every edge in it, so its line lies lower (a query alone / sixteen at once, us, fused and by
// launches: R-MAT of 10K edges 155 / 550 and 170 / 540, complete graph of 20K 160 / 800 and 165 /
// 530, R-MAT of 213K at eps 0.5 195 / 580 and 169 / 550, communities of 750K 860 / 3150 and 235 /
// 810).  predicate: 0 done by the similarity stage, 1 cached thresholds (tau); with 1 it also
// clears what the passes start from.
constexpr uint64_t kFusedEdgesRun = 1u << 16, kFusedEdgesServed = 1u << 14;
constexpr uint32_t kFusedVertices = 1u << 17;
constexpr int kFusedCtas = 8, kFusedThreads = 1024;

struct FusedCluster {
    uint64_t E;
    uint32_t n;
    const uint32_t *lo_adj, *lo_src, *off, *cn;
    const float* tau;
    uint8_t* sim;
    int32_t *sd, *parent, *bmin, *bmax, *nmin, *nmax, *lab, *label;
    uint8_t* role;
    RunCounters* ctr;
    uint32_t* flags;
    const unsigned long long* stage;
    uint32_t rounds, limit;
    int mu, predicate;
};

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

__global__ void __cluster_dims__(kFusedCtas, 1, 1) __launch_bounds__(kFusedThreads)
k_cluster_small(FusedCluster f, PredParams pp) {
    const Team team = grid_team();
    if (f.predicate == 1) {
        for (uint64_t i = team.index; i < f.n; i += team.size) f.sd[i] = 0;
        if (team.index == 0) *f.ctr = RunCounters{};
        if (team.index < kMaxJumpRounds) f.flags[team.index] = 0;
        cluster_barrier();
        predicate_tau_pass(team, f.E, f.lo_adj, f.lo_src, f.off, f.cn, f.tau, pp, f.sim, f.sd, f.ctr);
        cluster_barrier();
    }
    core_init_pass(team, f.n, f.sd, f.mu, nullptr, nullptr, f.parent, f.bmin, f.bmax, f.nmin, f.nmax, f.ctr);
    cluster_barrier();
    if (*(volatile uint32_t*)&f.ctr->any_core) {          // the same in every thread, as below
        union_pass<1>(team, f.E, f.lo_adj, f.lo_src, f.sim, f.parent, f.ctr, f.limit, 1);
        cluster_barrier();
        for (uint32_t r = 0; r < f.rounds; ++r) {
            const uint32_t ch = jump_pass(team, f.n, f.parent);
            if (__any_sync(0xFFFFFFFFu, ch) && (threadIdx.x & 31) == 0) atomicOr(&f.flags[r], 1u);
            cluster_barrier();
            if (*(volatile uint32_t*)&f.flags[r] == 0) break;
        }
        attach_pass<1>(team, f.E, f.lo_adj, f.lo_src, f.sim, f.parent, f.bmin, f.bmax, f.ctr);
        cluster_barrier();
        label_pass(team, f.n, f.parent, f.bmin, f.lab, f.ctr);
        cluster_barrier();
        neighbour_labels_pass(team, f.E, f.lo_adj, f.lo_src, f.lab, f.nmin, f.nmax, f.ctr);
        cluster_barrier();
    }
    finalize_pass(team, f.n, f.parent, f.bmin, f.bmax, f.nmin, f.nmax, f.label, f.role, f.stage, f.ctr);
}

// Memberships: every (cluster, border) pair from similar core-border edges.
__global__ void k_border_pairs(uint64_t E, const uint32_t* __restrict__ lo_adj, const uint32_t* __restrict__ lo_src,
                               const uint8_t* __restrict__ sim, const int32_t* __restrict__ parent,
                               unsigned long long* __restrict__ count, unsigned long long* __restrict__ out,
                               unsigned long long cap) {
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < E; e += (uint64_t)gridDim.x * blockDim.x) {
        if (!sim[e]) continue;
        const uint32_t u = lo_adj[e], v = lo_src[e];
        const int32_t pu = parent[u], pv = parent[v];
        unsigned long long key;
        if (pu >= 0 && pv < 0) key = ((unsigned long long)(uint32_t)pu << 32) | v;
        else if (pv >= 0 && pu < 0) key = ((unsigned long long)(uint32_t)pv << 32) | u;
        else continue;
        const unsigned long long i = atomicAdd(count, 1ull);
        if (i < cap) out[i] = key;
    }
}

}  // namespace scan
