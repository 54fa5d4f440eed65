// twmc_pair_rsl.cu -- the packed real-space kernel, per-site rsl with one real part.
#include "twmc_pair_launch.cuh"

namespace twmc {
bool pair_launch_rsl(const StepArgs& a, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err) {
  return pair_launch_par<PAIR_RSL_IM>(a, p, s, info, err);
}
}  // namespace twmc
