// twmc_pair.cu -- which split of the packed real-space kernel
// (twmc_pair.cuh) a run takes.
#include <algorithm>

#include "twmc_pair_launch.cuh"

namespace twmc {

namespace {

constexpr int64_t kSmemPerSm = 227 * 1024;

// Cycles per warp and slot of a split on a full SM, measured on GB300 with
// per-site omega (32x32, 64x64, 50x50, 80x80, 1x4096, 128x128 and others): a
// pair's instructions, the loads that a shorter run needs beside them, and
// the spills of a tighter register cap.
double slot_cycles(const PairPlan& p) {
  const int s = p.v * p.nb;
  if (p.chain) return s >= 8 ? 125.0 : p.nb > 1 ? 116.0 : 104.0;
  if (p.cl > 1) return !p.wide ? 165.0 : p.v >= 4 ? 185.0 : 165.0;
  if (p.wide) return s >= 8 ? 275.0 : 174.0;
  return s >= 8 ? 159.0 : s == 5 ? 148.0 : s == 4 ? (p.v == 1 ? 140.0 : p.v == 2 ? 131.0 : 132.0) : s == 3 ? 120.0 : s == 2 ? 114.0 : 122.0;
}

// Estimated cycles of one step of the whole batch: the slots' work on the
// fullest scheduler of an SM on top of a latency (exchange, barrier, Philox
// and the update's chain) that only the SM's other CTAs hide; a cluster
// barrier adds to it. Over 28 shapes and batch sizes the split it picked was
// within 5 % of the fastest for 22, within 15 % for all. All splits give the same bits, so only time
// depends on it.
double step_cycles(const PairPlan& p, int64_t ntraj, int sms) {
  const int64_t regs = p.wide ? 64 : 128;
  int64_t per_sm = std::min<int64_t>(65536 / (regs * p.threads), kSmemPerSm / (int64_t(p.smem) + 1024));
  per_sm = std::min<int64_t>(std::max<int64_t>(per_sm, 1), 32);
  const int64_t ctas = p.cl > 1 ? ntraj * p.cl : (ntraj + p.tpc - 1) / p.tpc;
  per_sm = std::min(per_sm, (ctas + sms - 1) / sms);
  const double waves = double(ctas) / double(per_sm * sms);
  const int64_t warps = per_sm * (p.threads / 32);
  const double slots = double(p.v * p.nb);
  const double latency = 420.0 + 40.0 * slots + (p.cl > 1 ? 700.0 : 0.0);
  const double work = double((warps + 3) / 4) * slots * slot_cycles(p);
  const double hidden = latency / double(per_sm);
  return (waves <= 6.0 ? double(int64_t(waves + 0.999999)) : waves + 0.5) * (work + hidden);
}

}  // namespace

bool pair_plan(const StepArgs& a, PairPlan* best) {
  const int64_t n = a.nsites;
  if (a.hop_kind != 1 || n < 2 || n % 2 || a.nx * a.ny != n) return false;
  const bool chain = a.nx == 1 || a.ny == 1;
  if (!chain && a.nx % 2) return false;  // a row's partner row must be a whole row
  const int64_t ny = chain ? 1 : a.ny, rows = n / 2 / ny;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  double best_t = -1.0;
  auto consider = [&](int v, int nb, bool ch, bool wide, int cl, int most) {
    if (ch != chain || rows % (int64_t(v) * cl)) return;
    const int64_t rl = rows / cl, tpt = (rl / v * ny + nb - 1) / nb;
    if (tpt > most) return;
    PairPlan p;
    p.v = v; p.nb = nb; p.cl = cl; p.chain = ch; p.wide = wide;
    p.tpt = int(tpt);
    const size_t buf = 2 * pair_buffer_bytes(ch, v, rl, ny);
    // short trajectories: one per CTA, or as many as make up about 128 threads
    for (int64_t want : {int64_t(1), (96 + tpt - 1) / tpt}) {
      if (cl > 1 && want > 1) continue;
      p.threads = int((tpt * want + 31) / 32 * 32);
      p.tpc = cl > 1 ? 1 : int(p.threads / tpt);  // as the kernel counts them
      p.smem = buf * size_t(p.tpc);
      if (p.threads > most || int64_t(p.smem) > kSmemPerSm) continue;
      const double t = step_cycles(p, std::max(a.ntraj, a.batch_traj), sms);
      if (best_t < 0 || t < best_t) { best_t = t; *best = p; }
    }
  };
#define TWMC_X(V, NB, CH, WIDE) consider(V, NB, CH, WIDE, 1, WIDE ? 1024 : 512);
#define TWMC_Y(V, CL, WIDE) consider(V, 1, false, WIDE, CL, WIDE ? 1024 : 256);
  TWMC_PAIR_VARIANTS(TWMC_X)
  if (n > 4096) { TWMC_PAIR_CLUSTERS(TWMC_Y) }
#undef TWMC_X
#undef TWMC_Y
  return best_t >= 0;
}

bool pair_launch(const StepArgs& a0, const PairPlan& p, cudaStream_t s, LaunchInfo* info, std::string* err) {
  StepArgs a = a0;
  a.tpt = p.tpt;
  if (a.nx == 1 || a.ny == 1) { a.nx = 1; a.ny = a.nsites; }
  if (!a.rsl && !a.iU && !a.iF) return pair_launch_scalar(a, p, s, info, err);
  if (!a.iU && !a.iF && a.rsl_re_uniform) return pair_launch_rsl(a, p, s, info, err);
  return pair_launch_site(a, p, s, info, err);
}

}  // namespace twmc
