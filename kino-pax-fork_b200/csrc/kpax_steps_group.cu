// kpax_steps_group.cu — the planner's kernels with a collision query per group of steps.
#include "kpax_plan_steps.cuh"

namespace kpax {
namespace plan {

template struct StepKernels<kGroup>;

IterateFn iterate_front_kernel(int bs)
{
    return by_block(bs, [](auto b) -> IterateFn { return k_iterate<KPAX_MODEL_QUADROTOR, decltype(b)::value, kIterFront, kGroup>; });
}

ExpandAllFn expand_mixed_kernel(int bs)
{
    return by_block(bs, [](auto b) -> ExpandAllFn { return k_expand_mixed<decltype(b)::value>; });
}

}  // namespace plan
}  // namespace kpax
