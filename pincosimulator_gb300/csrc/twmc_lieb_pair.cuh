// twmc_lieb_pair.cuh -- 1-D Lieb lattice step with cells c and c + Nc/2 as
// the two lanes of packed FP32 instructions: the FP32 run with Philox noise
// and an even number of cells (scheme, rounding and helpers: twmc_pair.cuh).
//
// Thread t of a trajectory holds the sites A, B, C of cells t and t + Nc/2, so
// every Philox pair (p, p + N/2) and the couplings inside a cell are its own;
// of the neighbouring cells it needs C of the previous one and B of the
// next, one 16-byte shared load each (lanes of both cells). Beyond the last
// slot the chain continues at slot 0 with the lanes exchanged (cell Nc/2 - 1's
// next is cell Nc/2); on an open chain the lane beyond the end is zero.
// Couplings: TWMCLiebSolver::Setup (TWMCLiebSolver.cpp:52-85). F(t) is held
// as dt times the value and slope of its current table segment, reloaded when
// the segment changes (every five steps of the 0.01 records at dt = 0.002)
// instead of read every step.
#pragma once

#include "twmc_pair.cuh"

namespace twmc {

// LIEB_IM: any of rsl and iU per site with one real part each, their imaginary parts
// held in registers for the launch; LIEB_SITE: any of rsl, iU, iF per site,
// read every step.
enum { LIEB_SCALAR = 0, LIEB_IM = 1, LIEB_SITE = 2 };

__host__ __device__ __forceinline__ size_t lieb_buffer_bytes(int64_t cells) { return 2 * size_t(cells / 2 + 2) * 16; }

template <int PAR, bool TIMEDEP>
__device__ __forceinline__ void lieb_pair_body(const StepArgs& a, unsigned char* smem_raw, int64_t group) {
  const int N = int(a.nsites), half = N >> 1, H = N / 6;
  const int tpt = H, tpc = int(blockDim.x) / tpt;
  const int slot0 = int(threadIdx.x) / tpt;
  const bool in_slot = slot0 < tpc;
  const int slot = in_slot ? slot0 : 0;
  const int t = in_slot ? int(threadIdx.x) - slot * tpt : 0;
  const uint32_t bufsz = uint32_t(lieb_buffer_bytes(N / 3)), coff = uint32_t(H + 2) * 16u;
  // B of slot i at base + (i + 1) 16, C behind all B
  const uint32_t base0 = smem_addr(smem_raw) + uint32_t(slot) * 2u * bufsz;
  const bool pbc = a.lieb_pbc != 0;
  const PairConst& k = a.pk;
  const float2 dt = make_float2(a.f_dt, a.f_dt);

  const int64_t traj = group * tpc + slot;
  const bool active = in_slot && traj < a.ntraj;
  const int64_t tr = active ? traj : 0;
  float2* st = reinterpret_cast<float2*>(a.state) + tr * N;
  const float2* __restrict__ g_rsl = PAR != LIEB_SCALAR && a.rsl ? reinterpret_cast<const float2*>(a.rsl) + tr * a.par_stride : nullptr;
  const float2* __restrict__ g_iU = PAR != LIEB_SCALAR && a.iU ? reinterpret_cast<const float2*>(a.iU) + tr * a.par_stride : nullptr;
  const float2* __restrict__ g_iF = PAR == LIEB_SITE && a.iF ? reinterpret_cast<const float2*>(a.iF) + tr * a.par_stride : nullptr;
  auto both = [&](const float2* __restrict__ g, int q, float2 sc, float2* x, float2* y) {
    const float2 l = g ? __ldg(g + q) : sc, h = g ? __ldg(g + q + half) : sc;
    *x = make_float2(l.x, h.x);
    *y = make_float2(l.y, h.y);
  };
  const float2 rsl_s = make_float2(a.f_par[0], a.f_par[1]), iU_s = make_float2(a.f_par[2], a.f_par[3]),
               iF_s = make_float2(a.f_par[4], a.f_par[5]);

  Pair v[3];
  float2 ay[PAR == LIEB_IM ? 3 : 1], by[PAR == LIEB_IM ? 3 : 1];
  Pair f0[TIMEDEP ? 3 : 1], f1[TIMEDEP ? 3 : 1];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int q = 3 * t + j;
    const float2 lo = active ? st[q] : make_float2(0.f, 0.f), hi = active ? st[q + half] : make_float2(0.f, 0.f);
    v[j] = Pair{make_float2(lo.x, hi.x), make_float2(lo.y, hi.y)};
    if constexpr (PAR == LIEB_IM) {
      float2 rx, ry, ux, uy;
      both(g_rsl, q, rsl_s, &rx, &ry);
      both(g_iU, q, iU_s, &ux, &uy);
      ay[j] = __fmul2_rn(dt, __fadd2_rn(ry, neg2(uy)));
      by[j] = __fmul2_rn(dt, uy);
    }
  }
  const uint32_t seed = a.seeds[tr], id = a.ids[tr];
  uint32_t buf = 0;
  int seg = -1;
  for (int64_t step = 0; step < a.nsteps; ++step) {
    const uint32_t gstep = a.step0 + uint32_t(step);
    const uint32_t cur = base0 + buf, at = cur + uint32_t(t + 1) * 16u;
    buf ^= bufsz;
    if (in_slot) {
      sts_pair(at, v[1]);
      sts_pair(at + coff, v[2]);
      if (t == 0) {  // the next cells of the last slot: cell Nc/2, and cell 0 on a ring
        Pair g = swapped(v[1]);
        if (!pbc) g.x.y = g.y.y = 0.f;
        sts_pair(cur + uint32_t(H + 1) * 16u, g);
      }
      if (t == H - 1) {  // the previous cells of slot 0: the last cell on a ring, and cell Nc/2 - 1
        Pair g = swapped(v[2]);
        if (!pbc) g.x.x = g.y.x = 0.f;
        sts_pair(cur + coff, g);
      }
    }
    float2 dtt = make_float2(0.f, 0.f);
    if constexpr (TIMEDEP) {
      const int s = a.ft_id[gstep];
      const float d = a.ft_dt_f[gstep];
      dtt = make_float2(d, d);
      if (s != seg) {
        seg = s;
        const float2* __restrict__ gv = reinterpret_cast<const float2*>(a.ft_vals) + int64_t(s) * N;
        const float2* __restrict__ gs = reinterpret_cast<const float2*>(a.ft_slopes) + int64_t(s) * N;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          both(gv, 3 * t + j, iF_s, &f0[j].x, &f0[j].y);
          both(gs, 3 * t + j, iF_s, &f1[j].x, &f1[j].y);
          f0[j] = Pair{__fmul2_rn(dt, f0[j].x), __fmul2_rn(dt, f0[j].y)};
          f1[j] = Pair{__fmul2_rn(dt, f1[j].x), __fmul2_rn(dt, f1[j].y)};
        }
      }
    }
    __syncthreads();
    const Pair cp = lds_pair(at + coff - 16u), bn = lds_pair(at + 16u);
    const Pair A = v[0], B = v[1], C = v[2];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int q = 3 * t + j;
      float2 ax = k.ax, ayj = k.ay, bx = k.bx, byj = k.by, fx = k.fx, fy = k.fy;
      if constexpr (PAR == LIEB_IM) {
        ayj = ay[j];
        byj = by[j];
      } else if constexpr (PAR == LIEB_SITE) {
        float2 rx, ry, ux, uy;
        both(g_rsl, q, rsl_s, &rx, &ry);
        both(g_iU, q, iU_s, &ux, &uy);
        ax = __fmul2_rn(dt, __fadd2_rn(rx, neg2(ux)));
        ayj = __fmul2_rn(dt, __fadd2_rn(ry, neg2(uy)));
        bx = __fmul2_rn(dt, ux);
        byj = __fmul2_rn(dt, uy);
        if constexpr (!TIMEDEP) {
          both(g_iF, q, iF_s, &fx, &fy);
          fx = __fmul2_rn(dt, fx);
          fy = __fmul2_rn(dt, fy);
        }
      }
      if constexpr (TIMEDEP) {
        fx = __ffma2_rn(dtt, f1[j].x, f0[j].x);
        fy = __ffma2_rn(dtt, f1[j].y, f0[j].y);
      }
      // the hopping's dt (-i J) b enters as one more term beside F'
      if (j == 0) {         // A: its B
        fx = __ffma2_rn(k.jab, B.y, fx);
        fy = __ffma2_rn(neg2(k.jab), B.x, fy);
        v[0] = pair_update<false>(A, fx, fy, ax, ayj, bx, byj, fx, fy, k.jt,
                                  pair_noise(wiener_words(uint32_t(q), gstep, seed, id), k.kn));
      } else if (j == 1) {  // B: its A, its C and the previous cell's C
        fx = __ffma2_rn(k.jab, A.y, fx);
        fy = __ffma2_rn(neg2(k.jab), A.x, fy);
        v[1] = pair_update(B, __fadd2_rn(cp.x, C.x), __fadd2_rn(cp.y, C.y), ax, ayj, bx, byj, fx, fy, k.jt,
                           pair_noise(wiener_words(uint32_t(q), gstep, seed, id), k.kn));
      } else {              // C: its B and the next cell's B
        v[2] = pair_update(C, __fadd2_rn(bn.x, B.x), __fadd2_rn(bn.y, B.y), ax, ayj, bx, byj, fx, fy, k.jt,
                           pair_noise(wiener_words(uint32_t(q), gstep, seed, id), k.kn));
      }
    }
  }
  if (active) {
    bool bad = false;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int q = 3 * t + j;
      const float2 lo = make_float2(v[j].x.x, v[j].y.x), hi = make_float2(v[j].x.y, v[j].y.y);
      st[q] = lo;
      st[q + half] = hi;
      bad |= !finite_c(lo) || !finite_c(hi);
    }
    set_status(a.status, traj, bad);
  }
}

}  // namespace twmc
