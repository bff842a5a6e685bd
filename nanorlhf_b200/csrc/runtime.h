// Host-side sampler runtime (C++): paged-KV block manager + continuous-batching scheduler.
// Replaces the scheduler / block-manager half of the vLLM engine the reference boots per rollout
// (GRPO/grpo_trainer.py:141-142).
#pragma once
#include <pybind11/pybind11.h>

namespace nrl {
void bind_runtime(pybind11::module_& m);
}
