// Host check of the slice rule of pending_slices.cuh: whatever the pivots, their pending work and
// the way their edges and lists are split into tasks, all tasks together get at most one slice
// each and `slices` more, which is the room their lists have.
//
// Test infrastructure: tests/test_pending_slices.py compiles and runs it on the CPU.
//   pending_slices_check       prints "ok <plans> <plans that use more than half of the room>"
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#define __host__
#define __device__
#define __forceinline__ inline
#include "pending_slices.cuh"

using namespace scan;

struct Pivot {
    uint32_t dv, edges, work, chunks, parts;   // list chunks x edge parts tasks, as the planner cuts them
};

static uint64_t all_slices(const std::vector<Pivot>& plan, uint32_t slices, uint64_t* tasks) {
    uint64_t total = 0, used = 0;
    *tasks = 0;
    for (const Pivot& p : plan) total += p.work;
    const uint64_t even = pending_even(total, slices);
    for (const Pivot& p : plan)
        for (uint32_t c = 0; c < p.chunks; ++c)
            for (uint32_t s = 0; s < p.parts; ++s) {
                const uint32_t chunk = (uint32_t)((uint64_t)p.dv * (c + 1) / p.chunks - (uint64_t)p.dv * c / p.chunks);
                const uint32_t e = (uint32_t)((uint64_t)p.edges * (s + 1) / p.parts - (uint64_t)p.edges * s / p.parts);
                used += pending_slices(even, p.work, e, p.edges, p.chunks > 1 ? chunk : p.dv, p.dv, e);
                ++*tasks;
            }
    return used;
}

int main() {
    std::mt19937_64 r(1);
    auto in = [&](uint64_t lo, uint64_t hi) { return lo + r() % (hi - lo + 1); };
    uint64_t plans = 0, full = 0;
    for (int round = 0; round < 4000; ++round) {
        const uint32_t slices = (uint32_t)(kPendingSlices * (round % 3 == 0 ? 1 : in(1, 152)));
        std::vector<Pivot> plan;
        const uint64_t pivots = in(1, 60);
        for (uint64_t i = 0; i < pivots; ++i) {
            Pivot p;
            p.dv = (uint32_t)in(129, round % 2 ? 1000 : round % 5 ? 100000 : 4000000);
            p.edges = (uint32_t)in(1, p.dv);
            // most of a pivot's edges may be pending, with lists up to its own length each
            p.work = (uint32_t)std::min<uint64_t>(in(1, uint64_t(p.edges) * (1 + p.dv / 64)), 0xFFFFFFFFu);
            p.chunks = p.dv > 6144 && in(0, 3) ? (p.dv + 6143) / 6144 : 1;
            p.parts = (uint32_t)in(1, std::min<uint64_t>((p.edges + 63) / 64, 20));
            plan.push_back(p);
        }
        uint64_t tasks = 0;
        const uint64_t used = all_slices(plan, slices, &tasks);
        if (used > tasks + slices) {
            std::printf("plan %d: %llu slices for %llu tasks + %u\n", round, (unsigned long long)used,
                        (unsigned long long)tasks, slices);
            return 1;
        }
        full += used > tasks + slices / 2;
        ++plans;
    }
    std::printf("ok %llu %llu\n", (unsigned long long)plans, (unsigned long long)full);
    return 0;
}
