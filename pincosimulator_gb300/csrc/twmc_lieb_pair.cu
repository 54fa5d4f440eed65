// twmc_lieb_pair.cu -- launcher of the packed Lieb kernel.
#include <algorithm>

#include "twmc_lieb_pair.cuh"
#include "twmc_pair_launch.cuh"

namespace twmc {

namespace {
constexpr int kLiebMost = 512;  // threads: 128 registers each hold six sites, their U and two values of F

template <int PAR, bool TIMEDEP>
__global__ void __launch_bounds__(kLiebMost, 1) lieb_pair_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  lieb_pair_body<PAR, TIMEDEP>(a, smem_raw, blockIdx.x);
}
}  // namespace

bool lieb_pair_ok(const StepArgs& a) {
  return a.hop_kind == 0 && a.nsites >= 6 && a.nsites % 6 == 0 && a.nsites / 6 <= kLiebMost;
}

bool lieb_pair_launch(const StepArgs& a, cudaStream_t s, LaunchInfo* info, std::string* err) {
  const bool td = a.ft_vals != nullptr;
  const bool im = (!a.rsl || a.rsl_re_uniform) && (!a.iU || a.iU_re_uniform) && !a.iF;
  const int par = !a.rsl && !a.iU && !a.iF ? LIEB_SCALAR : im ? LIEB_IM : LIEB_SITE;
  void (*fn)(const StepArgs) = par == LIEB_SCALAR ? (td ? lieb_pair_kernel<LIEB_SCALAR, true> : lieb_pair_kernel<LIEB_SCALAR, false>)
                               : par == LIEB_IM   ? (td ? lieb_pair_kernel<LIEB_IM, true> : lieb_pair_kernel<LIEB_IM, false>)
                                                  : (td ? lieb_pair_kernel<LIEB_SITE, true> : lieb_pair_kernel<LIEB_SITE, false>);
  // one trajectory per CTA, or short ones together up to about 128 threads
  // while that leaves every SM two CTAs
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tpt = int(a.nsites / 6);
  const int64_t batch = std::max(a.ntraj, a.batch_traj);
  const int want = int(std::max<int64_t>(1, std::min<int64_t>(128 / tpt, batch / (2 * sms))));
  const int threads = (tpt * want + 31) / 32 * 32, tpc = threads / tpt;
  const size_t smem = 2 * lieb_buffer_bytes(a.nsites / 3) * size_t(tpc);
  cudaError_t e = allow_smem(fn);
  if (e != cudaSuccess) { cudaGetLastError(); if (err) *err = std::string("packed Lieb smem: ") + cudaGetErrorString(e); return false; }
  const int64_t groups = (a.ntraj + tpc - 1) / tpc;
  if (info) { info->name = "lieb_cell_kernel"; info->kernel = "lieb_pair_kernel"; info->cta = threads; info->grid = int(groups); info->smem = smem; info->blocks_per_sm = 1; }
  if (groups <= 0) return true;
  if (groups > int64_t(0x7fffffff)) { if (err) *err = "packed Lieb kernel: too many trajectories"; return false; }
  fn<<<unsigned(groups), unsigned(threads), smem, s>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess) { if (err) *err = std::string("packed Lieb launch: ") + cudaGetErrorString(e); return false; }
  return true;
}

}  // namespace twmc
