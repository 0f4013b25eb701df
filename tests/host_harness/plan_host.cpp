// Host-compiled harness around the split of a generation step over clusters (generate_plan.hpp), used only by the CPU tests.
#include "../../ullis_b200/csrc/generate_plan.hpp"

using namespace ullis::gen;

// A device with room for any_room / cluster clusters of the form that is asked first and for own_room / cluster of the one taken; groups of
// up to fit_group sequences fit.  out: cluster, group, grid, how often the form taken was asked.
extern "C" void plan_host(uint64_t batch, uint32_t max_cluster, uint32_t max_group, uint32_t divides, uint32_t fit_group, int any_room, int own_room,
                          uint32_t* out) {
    uint32_t asked = 0;
    const StepPlan p = plan_step(
        batch, max_cluster, max_group, [&](uint32_t c) { return divides % c == 0; },
        [&](StepPlan& plan) {
            plan.stages = 2;
            plan.smem = 1024 * plan.group;
            return plan.group <= fit_group;
        },
        [&](const StepPlan& plan) { return any_room / (int)plan.cluster; },
        [&](const StepPlan& plan) {
            ++asked;
            return own_room / (int)plan.cluster;
        });
    out[0] = p.cluster; out[1] = p.group; out[2] = p.grid; out[3] = asked;
}
