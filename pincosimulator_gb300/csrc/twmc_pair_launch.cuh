// twmc_pair_launch.cuh -- the packed real-space kernel's instantiations for
// one kind of per-site parameters (one translation unit each, built in
// parallel); which of them a run takes is chosen in twmc_pair.cu.
#pragma once

#include <string>

#include "twmc_launch.h"
#include "twmc_pair.cuh"

namespace twmc {

// A choice of the run-splitting parameters of pair_body (twmc_pair.cuh) and
// the launch geometry that goes with it.
struct PairPlan {
  int v = 0, nb = 0, cl = 1;
  bool chain = false;
  bool wide = false;  // up to 1024 threads at 64 registers instead of 512 at 128
  int tpt = 0, tpc = 1, threads = 0;
  size_t smem = 0;
};

// Which 128-register splits keep the step-independent Philox rounds in registers
// of their own (WienerSite) instead of as the compiler hoists them. It pays where
// the compiler's own hoisting reaches the cap and keeping does not (registers,
// bytes of spills without / with; GB300, 1e11 site-updates/s without / with):
//   runs of five rows, per-site omega   128, 4 / 128, 0    3.93 / 4.36 (50x50)
//                      scalars          128, 12 / 126, 0   4.00 / 4.30
//   2 x 2 slots, per-site omega         128, 0 / 122, 0    5.03 / 5.17 (64x64)
//                scalars                124, 0 / 120, 0    5.32 / 5.23
//   clusters of four, scalars           128, 132 / 128, 60 4.15 / 4.25 (128x128)
//                     per-site omega    128, 192 / 128, 120 4.24 / 4.16
//   one slot, chain                     52, 0 / 48, 0      2.58 / 2.42 (1x64)
// (clusters spill either way, and only measuring told). Not timed by themselves: the
// other splits of four and more slots, which follow their neighbours here.
// For a new split: compile both with -Xptxas -v, keep if only that leaves the
// cap, and time it.
constexpr bool pair_keep(int v, int nb, bool ch, int par, int cl) {
  if (cl > 1) return par == PAIR_SCALAR;
  return !ch && ((par == PAIR_RSL_IM && v * nb >= 4) || (par == PAIR_SCALAR && v >= 4));
}

// Register caps. 128 registers hold four slots of state (32), what is kept of
// the Philox rounds and the loads in flight without spilling; measured on GB300 at
// 32x32 with 128-thread CTAs, four per SM: 5.55e11 site-updates/s at 128
// registers, 5.3e11 at 80, 5.1e11 at 64 (144 bytes of spills).
template <int V, int NB, bool CH, int PAR>
__global__ void __launch_bounds__(512, 1) pair_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pair_body<V, NB, CH, PAR, 1, pair_keep(V, NB, CH, PAR, 1)>(a, smem_raw, blockIdx.x);
}
template <int V, int NB, bool CH, int PAR>
__global__ void __launch_bounds__(1024, 1) pair_kernel_wide(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pair_body<V, NB, CH, PAR>(a, smem_raw, blockIdx.x);
}
template <int V, int CL, int PAR>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(256, 2) pair_cluster_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pair_body<V, 1, false, PAR, CL, pair_keep(V, 1, false, PAR, CL)>(a, smem_raw, blockIdx.x / CL);
}
template <int V, int CL, int PAR>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(1024, 1) pair_cluster_kernel_wide(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pair_body<V, 1, false, PAR, CL>(a, smem_raw, blockIdx.x / CL);
}

// The instantiations: X(V, NB, chain, wide) and Y(V, clusters, wide).
#define TWMC_PAIR_VARIANTS(X)                                                                                  \
  X(1, 1, false, false) X(2, 1, false, false) X(3, 1, false, false) X(4, 1, false, false) X(5, 1, false, false) \
  X(2, 2, false, false) X(4, 2, false, false) X(1, 2, false, false) X(1, 4, false, false) X(4, 1, false, true)  \
  X(1, 4, false, true) X(1, 8, false, true)                                                                    \
  X(1, 1, true, false) X(2, 1, true, false) X(3, 1, true, false) X(4, 1, true, false) X(5, 1, true, false)     \
  X(1, 2, true, false) X(1, 4, true, false) X(1, 4, true, true) X(4, 1, true, true) X(8, 1, true, true)
#define TWMC_PAIR_CLUSTERS(Y) Y(8, 4, false) Y(4, 4, true) Y(2, 4, true) Y(5, 2, true) Y(4, 2, true) Y(3, 2, true) Y(1, 2, true)

template <int PAR>
bool pair_launch_par(const StepArgs& a, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err) {
  void (*fn)(const StepArgs) = nullptr;
#define TWMC_X(V, NB, CH, WIDE)                                                             \
  if (p.cl == 1 && p.v == V && p.nb == NB && p.chain == CH && p.wide == WIDE) {             \
    if constexpr (WIDE) fn = pair_kernel_wide<V, NB, CH, PAR>; else fn = pair_kernel<V, NB, CH, PAR>; \
  }
#define TWMC_Y(V, CL, WIDE)                                                                 \
  if (p.cl == CL && p.v == V && p.nb == 1 && !p.chain && p.wide == WIDE) {                  \
    if constexpr (WIDE) fn = pair_cluster_kernel_wide<V, CL, PAR>; else fn = pair_cluster_kernel<V, CL, PAR>; \
  }
  TWMC_PAIR_VARIANTS(TWMC_X)
  TWMC_PAIR_CLUSTERS(TWMC_Y)
#undef TWMC_X
#undef TWMC_Y
  if (!fn) { if (err) *err = "packed real-space kernel: variant not compiled"; return false; }
  cudaError_t e = allow_smem(fn);
  if (e != cudaSuccess) { cudaGetLastError(); if (err) *err = std::string("packed real-space smem: ") + cudaGetErrorString(e); return false; }
  const int64_t groups = p.cl > 1 ? a.ntraj : (a.ntraj + p.tpc - 1) / p.tpc;
  if (info) {
    info->kernel = std::string(p.cl > 1 ? "pair_cluster_kernel" : "pair_kernel") + (p.wide ? "_wide<" : "<") +
                   std::to_string(p.v) + "," + std::to_string(p.cl > 1 ? p.cl : p.nb) + (p.chain ? ",chain>" : ">");
    info->cta = p.threads; info->grid = int(groups * p.cl); info->smem = p.smem; info->blocks_per_sm = 1;
  }
  if (groups <= 0) return true;
  if (groups * p.cl > int64_t(0x7fffffff)) { if (err) *err = "packed real-space kernel: too many trajectories"; return false; }
  fn<<<unsigned(groups * p.cl), unsigned(p.threads), p.smem, s>>>(a);
  e = cudaGetLastError();
  if (e != cudaSuccess) { if (err) *err = std::string("packed real-space launch: ") + cudaGetErrorString(e); return false; }
  return true;
}

bool pair_launch_scalar(const StepArgs& a, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err);
bool pair_launch_rsl(const StepArgs& a, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err);
bool pair_launch_site(const StepArgs& a, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err);

// Whether a run (FP32, Philox noise, no F(t), no work / area: the caller's
// check) has the packed form's geometry, and the plan for it.
bool pair_plan(const StepArgs& a, PairPlan* p);
// Launches it (plan from pair_plan; a.tpt is taken from the plan).
bool pair_launch(const StepArgs& a, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err);

// The packed Lieb kernel (twmc_lieb_pair.cu) for the same kind of run, F(t)
// allowed: an even number of cells, at most 1024.
bool lieb_pair_ok(const StepArgs& a);
bool lieb_pair_launch(const StepArgs& a, cudaStream_t s, LaunchInfo* info, std::string* err);

}  // namespace twmc
