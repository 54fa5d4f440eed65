// twmc_pair_site.cu -- the packed real-space kernel, any per-site parameters.
#include "twmc_pair_launch.cuh"

namespace twmc {
bool pair_launch_site(const StepArgs& a, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err) {
  return pair_launch_par<PAIR_SITE>(a, p, s, info, err);
}
}  // namespace twmc
