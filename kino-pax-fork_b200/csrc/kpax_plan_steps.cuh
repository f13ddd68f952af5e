// kpax_plan_steps.cuh — definitions behind kpax_plan_steps.h, for the units that instantiate them.
#pragma once
#include <type_traits>

#include "kpax_batch_kernels.cuh"
#include "kpax_plan_steps.h"

namespace kpax {
namespace plan {

// f(block size) with the block size as a constant.
template <class F>
auto by_block(int bs, F&& f)
{
    using std::integral_constant;
    switch(bs) {
        case 128: return f(integral_constant<int, 128>{});
        case 256: return f(integral_constant<int, 256>{});
        case 512: return f(integral_constant<int, 512>{});
        default: return f(integral_constant<int, kExpandBS>{});
    }
}

// f(model, block size) with both as constants.
template <class F>
auto by_model_block(int model, int bs, F&& f)
{
    using std::integral_constant;
    return by_block(bs, [&](auto b) {
        return model == KPAX_MODEL_DOUBLE_INTEGRATOR ? f(integral_constant<int, KPAX_MODEL_DOUBLE_INTEGRATOR>{}, b)
               : model == KPAX_MODEL_DUBINS_AIRPLANE ? f(integral_constant<int, KPAX_MODEL_DUBINS_AIRPLANE>{}, b)
                                                     : f(integral_constant<int, KPAX_MODEL_QUADROTOR>{}, b);
    });
}

template <int K>
ExpandFn StepKernels<K>::expand(int model, int bs)
{
    return by_model_block(model, bs, [](auto m, auto b) -> ExpandFn { return k_expand<decltype(m)::value, decltype(b)::value, K>; });
}

template <int K>
ExpandAllFn StepKernels<K>::expand_all(int model, int bs)
{
    return by_model_block(model, bs, [](auto m, auto b) -> ExpandAllFn { return k_expand_all<decltype(m)::value, decltype(b)::value, K>; });
}

template <int K>
IterateFn StepKernels<K>::iterate(int model, int bs)
{
    return by_model_block(model, bs,
                          [](auto m, auto b) -> IterateFn { return k_iterate<decltype(m)::value, decltype(b)::value, kIterWhole, K>; });
}

template <int K>
IterateFn StepKernels<K>::iterate_back(int bs)
{
    return by_block(bs, [](auto b) -> IterateFn { return k_iterate<KPAX_MODEL_QUADROTOR, decltype(b)::value, kIterBack, K>; });
}

}  // namespace plan
}  // namespace kpax
