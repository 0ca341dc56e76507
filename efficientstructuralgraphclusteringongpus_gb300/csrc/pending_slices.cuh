// Into how many slices a task's pending edges are cut (k_pending_tasks).
#pragma once

#include <cstdint>

namespace scan {

constexpr uint32_t kPendingSlices = 8;        // slices aimed at per SM, over all lists
constexpr uint32_t kPendingMinWork = 512;     // 32K list entries: a slice stages its pivot again

// A slice's share of the whole pending work, `slices` of which make it up.
__host__ __device__ __forceinline__ uint64_t pending_even(uint64_t total, uint32_t slices) { return total / slices + 1; }

// Slices of a task that has `found` pending edges.  pivot_work: pending work of its pivot, of
// degree dv; the task holds `edges` of the pivot's `pivot_edges` edges and, where the pivot's
// list is split, `chunk` of its dv entries (else chunk = dv).  Every chunk gathers the same
// edges but reads its part of their lists only, so it is charged that part: the tasks of a
// pivot then share its work at most once, and all tasks together get at most one slice each
// and `slices` more, which is what the lists hold.
__host__ __device__ __forceinline__ uint32_t pending_slices(uint64_t even, uint32_t pivot_work, uint32_t edges,
                                                            uint32_t pivot_edges, uint32_t chunk, uint32_t dv,
                                                            uint32_t found) {
    const uint64_t mine = (uint64_t)pivot_work * edges / pivot_edges * chunk / dv;
    uint64_t aim = even > kPendingMinWork ? even : kPendingMinWork;
    if (aim < dv / 16) aim = dv / 16;                       // 4 dv entries at least
    const uint64_t n = mine / aim + 1, most = ((uint64_t)found + 7) / 8;
    return (uint32_t)(n < most ? n : most);
}

}  // namespace scan
