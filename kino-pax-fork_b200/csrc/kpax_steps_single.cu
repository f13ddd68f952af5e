// kpax_steps_single.cu — the planner's kernels with a collision query per step.
#include "kpax_plan_steps.cuh"

template struct kpax::plan::StepKernels<1>;
