// FP64 instantiation of the staged MPDATA step (compiled without FMA contraction).
#include "stages_impl.cuh"

namespace mpdx {
template struct stage_engine<double>;
}  // namespace mpdx
