// twmc_pair.cuh -- real-space step with site p and its Philox partner
// p + N/2 as the two lanes of packed FP32 instructions (fma / add / mul
// .f32x2): the FP32 run with Philox noise and no F(t), work or area.
//
// Why packed: the unpacked stencil kernels issued 70 to 112 instructions per
// site-update with the FMA pipe under 40 % busy, so the issue slots bound
// them. Both sites of a pair share one Philox call and do the same
// arithmetic on different values, so every FP32 operation of the step is one
// instruction for the two, operands included: the field is held and
// exchanged as (x_p, x_p', y_p, y_p'), never repacked.
//
// Layout: slot q < N/2 holds sites q and q + N/2. With an even number of
// rows the slots are a lattice of nx / 2 rows whose vertical wrap exchanges
// the lanes (the row below the last one is row 0 with its lanes swapped); a
// chain of N sites is a column of N/2 slots with the same twist. A thread
// holds V consecutive rows of one column (times NB blocks of rows): vertical
// neighbours inside the run are its own registers, and a slot's left / right
// neighbours are one 16-byte shared load each, consecutive threads on
// consecutive columns. The two rows beyond the wrap are kept as ghost rows,
// stored with swapped lanes by the threads that own the originals.
//
// Rounding: every operation is an explicit round-to-nearest intrinsic in one
// order, so a trajectory's bits depend neither on V, NB, the CTA geometry nor
// the launch (single system or batch) it runs in.
#pragma once

#include "twmc_kernels.cuh"

namespace twmc {

struct Pair {
  float2 x, y;  // (site p, site p + N/2)
};

__device__ __forceinline__ float2 neg2(float2 v) { return make_float2(-v.x, -v.y); }
__device__ __forceinline__ float2 swap2(float2 v) { return make_float2(v.y, v.x); }

__device__ __forceinline__ Pair lds_pair(uint32_t a) {
  Pair v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x.x), "=f"(v.x.y), "=f"(v.y.x), "=f"(v.y.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_pair(uint32_t a, Pair v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x.x), "f"(v.x.y), "f"(v.y.x), "f"(v.y.y)
               : "memory");
}
__device__ __forceinline__ void stc_pair(uint32_t a, Pair v) {  // into another CTA of the cluster
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x.x), "f"(v.x.y), "f"(v.y.x),
               "f"(v.y.y) : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ Pair swapped(Pair v) { return Pair{swap2(v.x), swap2(v.y)}; }

// The two Wiener terms of one Philox call, sqrt(gamma dt / 4) xi = r (c, s)
// per lane: scaled_normal_pair with the products left to the update's
// multiply-adds. |kn log2 u| is kn log2 u wherever the logarithm is not above
// 0 (u <= 1), so the absolute value, an operand modifier, stands for the clamp.
struct PairNoise {
  float2 r, c, s;
};
__device__ __forceinline__ PairNoise pair_noise(u32x4 w, float2 kn) {
  PairNoise n;
  const float2 u = __ffma2_rn(make_float2(__uint2float_rn(w.x), __uint2float_rn(w.z)),
                              make_float2(0x1p-32f, 0x1p-32f), make_float2(0x1p-33f, 0x1p-33f));
  const float2 th = __ffma2_rn(make_float2(__uint2float_rn(w.y), __uint2float_rn(w.w)),
                               make_float2(1.46291807926715968e-9f, 1.46291807926715968e-9f),
                               make_float2(-3.14159265285833420f, -3.14159265285833420f));
  const float2 t = __fmul2_rn(kn, make_float2(lg2_approx(u.x), lg2_approx(u.y)));
  n.r = make_float2(sqrt_approx(fabsf(t.x)), sqrt_approx(fabsf(t.y)));
  __sincosf(th.x, &n.s.x, &n.c.x);
  __sincosf(th.y, &n.s.y, &n.c.y);
  return n;
}

// b' = b + ((A + B |b|^2) b + F' - i dt J s + sqrt(gamma dt / 4) xi) with
// A = dt (rsl - iU), B = dt iU, F' = dt iF and s the neighbours' sum: the
// reference's step (TWMCBaseSolver.cpp:245-253) with dt folded into the
// coefficients of the increment, whose terms are accumulated by multiply-adds
// and added to b once. HOP false: no such neighbours (s is not read).
template <bool HOP = true>
__device__ __forceinline__ Pair pair_update(Pair v, float2 sx, float2 sy, float2 ax, float2 ay, float2 bx, float2 by,
                                            float2 fx, float2 fy, float2 jt, const PairNoise& n) {
  const float2 ab2 = __ffma2_rn(v.y, v.y, __fmul2_rn(v.x, v.x));
  const float2 cx = __ffma2_rn(bx, ab2, ax), cy = __ffma2_rn(by, ab2, ay);
  float2 ix = __ffma2_rn(n.r, n.c, fx), iy = __ffma2_rn(n.r, n.s, fy);
  if constexpr (HOP) {
    ix = __ffma2_rn(jt, sy, ix);
    iy = __ffma2_rn(neg2(jt), sx, iy);
  }
  ix = __ffma2_rn(cx, v.x, ix);
  iy = __ffma2_rn(cx, v.y, iy);
  ix = __ffma2_rn(neg2(cy), v.y, ix);
  iy = __ffma2_rn(cy, v.x, iy);
  return Pair{__fadd2_rn(v.x, ix), __fadd2_rn(v.y, iy)};
}

// Per-site parameters: none (PAIR_SCALAR), rsl with one real part (its
// imaginary part held in registers for the launch, PAIR_RSL_IM), or any of
// rsl, iU, iF per site, read from global memory every step (PAIR_SITE).
enum { PAIR_SCALAR = 0, PAIR_RSL_IM = 1, PAIR_SITE = 2 };

// Bytes of one exchange buffer of a trajectory: the slots with two ghost rows,
// or, for a chain, the first and last slot of every run with two ghosts each.
__host__ __device__ __forceinline__ size_t pair_buffer_bytes(bool chain, int v, int64_t rows, int64_t ny) {
  if (chain) return (v == 1 ? 1 : 2) * size_t(rows / v + 2) * 16;
  return size_t(rows + 2) * size_t(ny) * 16;
}

// One group of trajectories (blockDim.x / tpt of them) for a.nsteps steps.
// CH: chain (rows = N/2, one column). CL > 1: one trajectory on a cluster of
// CL CTAs, CTA r holding rows [r rows / CL, (r + 1) rows / CL); every step each
// CTA writes its first and last row into its neighbours' ghost rows (the
// lattice's own two ghost rows among them) through distributed shared
// memory, so that all loads are local and one cluster barrier separates the
// writes from the reads.
// KEEP: the step-independent part of every pair's Philox rounds stays in registers
// (WienerSite, four per pair).
template <int V, int NB, bool CH, int PAR, int CL = 1, bool KEEP = false>
__device__ __forceinline__ void pair_body(const StepArgs& a, unsigned char* smem_raw, int64_t group) {
  static_assert(CL == 1 || !CH, "chains run on one CTA");
  const int N = int(a.nsites), half = N >> 1;
  const int ny = CH ? 1 : int(a.ny), rows = (CH ? half : half / ny) / CL, nblk = rows / V;
  const int tpt = a.tpt, tpc = CL > 1 ? 1 : int(blockDim.x) / tpt;
  const int slot0 = int(threadIdx.x) / tpt;
  const bool in_slot = slot0 < tpc;
  const int slot = in_slot ? slot0 : 0;
  const int t = in_slot ? int(threadIdx.x) - slot * tpt : 0;
  const uint32_t bufsz = uint32_t(pair_buffer_bytes(CH, V, rows, ny));
  const uint32_t base0 = smem_addr(smem_raw) + uint32_t(slot) * 2u * bufsz;
  const uint32_t pitch = uint32_t(ny) * 16u;
  const uint32_t last_off = V == 1 ? 0u : uint32_t(nblk + 2) * 16u;  // chain: the array of last slots
  // where the first row goes (the ghost row below the CTA above) and where
  // the last one goes (the ghost row above the CTA below), column 0, buffer 0
  const int rank = CL > 1 ? int(cluster_rank()) : 0;
  uint32_t g_first = base0 + uint32_t(rows + 1) * pitch, g_last = base0;
  if constexpr (CL > 1) {
    g_first = cluster_addr(g_first, uint32_t(rank == 0 ? CL - 1 : rank - 1));
    g_last = cluster_addr(g_last, uint32_t(rank == CL - 1 ? 0 : rank + 1));
  }

  const int64_t traj = group * tpc + slot;
  const bool active = in_slot && traj < a.ntraj;
  const int64_t tr = active ? traj : 0;
  float2* st = reinterpret_cast<float2*>(a.state) + tr * N;
  const float2* __restrict__ g_rsl = PAR != PAIR_SCALAR && a.rsl ? reinterpret_cast<const float2*>(a.rsl) + tr * a.par_stride : nullptr;
  const float2* __restrict__ g_iU = PAR == PAIR_SITE && a.iU ? reinterpret_cast<const float2*>(a.iU) + tr * a.par_stride : nullptr;
  const float2* __restrict__ g_iF = PAR == PAIR_SITE && a.iF ? reinterpret_cast<const float2*>(a.iF) + tr * a.par_stride : nullptr;
  const PairConst& k = a.pk;

  // block i of the thread: V rows of column c from row blk V on; consecutive
  // threads hold consecutive columns, then the next block of rows
  bool ok[NB];
  int blk[NB], c[NB], q0[NB];  // q0: its first slot, of the CTA's slots
  int dl[CH ? 1 : NB], dr[CH ? 1 : NB];  // offsets of the left and right neighbour columns (periodic)
  const int qr = rank * rows * ny;  // first slot of the CTA
  Pair v[NB][V];
  float2 ay[PAR == PAIR_RSL_IM ? NB : 1][PAR == PAIR_RSL_IM ? V : 1];
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    const int u = t + i * tpt;
    ok[i] = in_slot && (NB == 1 || u < nblk * ny);
    blk[i] = ok[i] ? u / ny : 0;
    c[i] = CH || !ok[i] ? 0 : u - blk[i] * ny;
    q0[i] = blk[i] * V * ny + c[i];
    if constexpr (!CH) {
      dl[i] = c[i] > 0 ? -16 : (ny - 1) * 16;
      dr[i] = c[i] + 1 < ny ? 16 : -(ny - 1) * 16;
    }
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const int q = qr + q0[i] + j * ny;
      const float2 lo = active ? st[q] : make_float2(0.f, 0.f), hi = active ? st[q + half] : make_float2(0.f, 0.f);
      v[i][j] = Pair{make_float2(lo.x, hi.x), make_float2(lo.y, hi.y)};
      if constexpr (PAR == PAIR_RSL_IM)
        ay[i][j] = __fmul2_rn(make_float2(a.f_dt, a.f_dt),
                              __fadd2_rn(make_float2(g_rsl[q].y, g_rsl[q + half].y), neg2(k.uy)));
    }
  }
  const uint32_t seed = a.seeds[tr], id = a.ids[tr];
  WienerSite ws[KEEP ? NB : 1][KEEP ? V : 1];
#pragma unroll
  for (int i = 0; i < (KEEP ? NB : 0); ++i)
#pragma unroll
    for (int j = 0; j < V; ++j) ws[i][j] = wiener_site(uint32_t(qr + q0[i] + j * ny), seed, id);
  uint32_t buf = 0;
  if constexpr (CL > 1) {  // every CTA of the cluster is there, and done with what ran before
    cluster_arrive();
    cluster_wait();
  }
  for (int64_t step = 0; step < a.nsteps; ++step) {
    const uint32_t gstep = a.step0 + uint32_t(step);
    const WienerStep wt = wiener_step(gstep, id);
    const uint32_t cur = base0 + buf;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      if (!ok[i]) continue;
      if constexpr (CH) {
        const uint32_t at = cur + uint32_t(blk[i] + 1) * 16u;
        sts_pair(at, v[i][0]);
        if constexpr (V > 1) sts_pair(at + last_off, v[i][V - 1]);
        if (blk[i] == 0) sts_pair(cur + uint32_t(nblk + 1) * 16u, swapped(v[i][0]));
        if (blk[i] == nblk - 1) sts_pair(cur + last_off, swapped(v[i][V - 1]));
      } else {
        const uint32_t at = cur + pitch + uint32_t(q0[i]) * 16u;
#pragma unroll
        for (int j = 0; j < V; ++j) sts_pair(at + uint32_t(j) * pitch, v[i][j]);
        if constexpr (CL == 1) {
          if (blk[i] == 0) sts_pair(g_first + buf + uint32_t(c[i]) * 16u, swapped(v[i][0]));
          if (blk[i] == nblk - 1) sts_pair(g_last + buf + uint32_t(c[i]) * 16u, swapped(v[i][V - 1]));
        } else {
          if (blk[i] == 0) stc_pair(g_first + buf + uint32_t(c[i]) * 16u, rank == 0 ? swapped(v[i][0]) : v[i][0]);
          if (blk[i] == nblk - 1) stc_pair(g_last + buf + uint32_t(c[i]) * 16u, rank == CL - 1 ? swapped(v[i][V - 1]) : v[i][V - 1]);
        }
      }
    }
    if constexpr (CL == 1) {
      __syncthreads();
    } else {
      cluster_arrive();
      cluster_wait();
    }
    buf ^= bufsz;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const uint32_t at = CH ? cur + uint32_t(blk[i] + 1) * 16u : cur + pitch + uint32_t(q0[i]) * 16u;
      Pair up = lds_pair(CH ? at + last_off - 16u : at - pitch);
      const Pair dn = lds_pair(CH ? at + 16u : at + uint32_t(V) * pitch);
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const int q = qr + q0[i] + j * ny;
        const Pair below = j + 1 < V ? v[i][j + 1] : dn;
        float2 sx = __fadd2_rn(below.x, up.x), sy = __fadd2_rn(below.y, up.y);
        if constexpr (!CH) {
          const uint32_t own = at + uint32_t(j) * pitch;
          const Pair rt = lds_pair(own + uint32_t(dr[i])), lf = lds_pair(own + uint32_t(dl[i]));
          sx = __fadd2_rn(__fadd2_rn(rt.x, lf.x), sx);
          sy = __fadd2_rn(__fadd2_rn(rt.y, lf.y), sy);
        }
        u32x4 w;
        if constexpr (KEEP) w = wiener_words(ws[i][j], wt);
        else w = wiener_words(uint32_t(q), gstep, seed, id);
        const PairNoise nz = pair_noise(w, k.kn);
        up = v[i][j];
        if constexpr (PAR == PAIR_SCALAR) {
          v[i][j] = pair_update(v[i][j], sx, sy, k.ax, k.ay, k.bx, k.by, k.fx, k.fy, k.jt, nz);
        } else if constexpr (PAR == PAIR_RSL_IM) {
          v[i][j] = pair_update(v[i][j], sx, sy, k.ax, ay[i][j], k.bx, k.by, k.fx, k.fy, k.jt, nz);
        } else {
          const float2 dt = make_float2(a.f_dt, a.f_dt);
          auto site = [&](const float2* __restrict__ g, float2 sc, float2* x, float2* y) {
            const float2 l = g ? __ldg(g + q) : sc, h = g ? __ldg(g + q + half) : sc;
            *x = make_float2(l.x, h.x);
            *y = make_float2(l.y, h.y);
          };
          float2 rx, ry, ux, uy, fx, fy;
          site(g_rsl, make_float2(a.f_par[0], a.f_par[1]), &rx, &ry);
          site(g_iU, make_float2(a.f_par[2], a.f_par[3]), &ux, &uy);
          site(g_iF, make_float2(a.f_par[4], a.f_par[5]), &fx, &fy);
          v[i][j] = pair_update(v[i][j], sx, sy, __fmul2_rn(dt, __fadd2_rn(rx, neg2(ux))),
                                __fmul2_rn(dt, __fadd2_rn(ry, neg2(uy))), __fmul2_rn(dt, ux), __fmul2_rn(dt, uy),
                                __fmul2_rn(dt, fx), __fmul2_rn(dt, fy), k.jt, nz);
        }
      }
    }
  }
  if (active) {
    bool bad = false;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      if (!ok[i]) continue;
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const int q = qr + q0[i] + j * ny;
        const float2 lo = make_float2(v[i][j].x.x, v[i][j].y.x), hi = make_float2(v[i][j].x.y, v[i][j].y.y);
        st[q] = lo;
        st[q + half] = hi;
        bad |= !finite_c(lo) || !finite_c(hi);
      }
    }
    set_status(a.status, traj, bad);
  }
}

}  // namespace twmc
