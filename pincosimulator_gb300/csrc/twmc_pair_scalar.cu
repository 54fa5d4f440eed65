// twmc_pair_scalar.cu -- the packed real-space kernel, no per-site parameters.
#include "twmc_pair_launch.cuh"

namespace twmc {
bool pair_launch_scalar(const StepArgs& a, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err) {
  return pair_launch_par<PAIR_SCALAR>(a, p, s, info, err);
}
}  // namespace twmc
