// How a generation step that runs as one kernel is split over clusters of CTAs (generate_step.cuh); host code.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace ullis {
namespace gen {

struct StepPlan {
    uint32_t cluster = 0, group = 1, stages = 0;   // CTAs of a cluster, its sequences, pieces of the value weights in flight
    bool staged = false;                           // packed weights through shared memory
    size_t smem = 0;
    int clusters = 0;                              // the device holds at once
    unsigned grid = 0;                             // 0: the step does not run as one kernel
};

// One round of clusters if there is a way, with as many CTAs per cluster as the channels allow (a CTA's share of the sums is shortest
// then) and as few sequences per cluster as the clusters that the device holds at once allow.
//   divides(cluster): whether channels and hidden units come out even
//   fit(plan): sets stages, staged and smem for its cluster and group; false: no room
//   room(plan): clusters the device holds at once, by any form of the kernel that is at hand
//   room_of(plan): the same by the form that the plan takes, whose `clusters` are those of `room`; asked once, since a form that is asked for
//     is loaded
template <typename Divides, typename Fit, typename Room, typename RoomOf>
StepPlan plan_step(size_t batch, uint32_t max_cluster, uint32_t max_group, Divides divides, Fit fit, Room room, RoomOf room_of) {
    StepPlan best;
    size_t best_rounds = SIZE_MAX;
    for (uint32_t c = max_cluster; c >= 1 && best_rounds > 1; c /= 2) {
        if (!divides(c)) continue;
        for (uint32_t g = 1; g <= max_group && best_rounds > 1; g *= 2) {
            StepPlan p;
            p.cluster = c;
            p.group = g;
            if (!fit(p)) break;
            p.clusters = room(p);
            if (p.clusters < 1) break;
            const size_t rounds = ((batch + g - 1) / g + p.clusters - 1) / p.clusters;
            if (rounds >= best_rounds) continue;
            best_rounds = rounds;
            best = p;
        }
    }
    if (!best.cluster) return best;
    // The forms differ in registers: a grid of more clusters than this one has room for would run its last ones alone.
    best.clusters = room_of(best);
    if (best.clusters >= 1) best.grid = (unsigned)(std::min<size_t>((batch + best.group - 1) / best.group, (size_t)best.clusters) * best.cluster);
    return best;
}

}  // namespace gen
}  // namespace ullis
