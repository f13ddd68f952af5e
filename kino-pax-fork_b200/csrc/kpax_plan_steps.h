// kpax_plan_steps.h — the planner's kernels that integrate segments, chosen by model (KPAX_MODEL_*), block
// size (validated by kpax_config_validate) and steps per collision query: K = kGroup or 1 (run_steps).  They
// are most of the library's device code, so each K is compiled in a unit of its own.
#pragma once
#include <stddef.h>

#include "kpax_plan_kernels.cuh"

namespace kpax {
namespace plan {

using ExpandFn = void (*)(const QueryDev*, const uint32_t*, uint32_t*);                           // k_expand
using ExpandAllFn = void (*)(const QueryDev*, const Ctl*, const uint32_t*, uint32_t, uint32_t*);  // k_expand_all, _mixed
using IterateFn = void (*)(const QueryDev*, const Ctl*, uint32_t*, uint32_t);                     // k_iterate

template <int K>
struct StepKernels {
    static ExpandFn expand(int model, int bs);
    static ExpandAllFn expand_all(int model, int bs);
    static IterateFn iterate(int model, int bs);
    static IterateFn iterate_back(int bs);  // the quadrotor's part behind the proposal pass
};

// The part before the proposal pass (it integrates no steps).
IterateFn iterate_front_kernel(int bs);
// One launch for every model's queries, in groups of kGroup steps.
ExpandAllFn expand_mixed_kernel(int bs);

// Shared memory of the kept states of a block of bs children (run_steps).
inline size_t save_bytes(int model, int group, int bs)
{
    return group > 1 ? sizeof(float) * group * (model == KPAX_MODEL_QUADROTOR ? 12 : 6) * (size_t)bs : 0;
}

}  // namespace plan
}  // namespace kpax
