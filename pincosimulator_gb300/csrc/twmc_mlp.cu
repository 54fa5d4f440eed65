// twmc_mlp.cu -- the learned warm start: a small MLP with BF16 weights and
// FP32 accumulation on the tensor cores (forward, backward, Adam), mapping a
// parameter point (F, detuning, U, J, gamma) to its steady-state k-mode mean
// field and density, plus the transforms between engine fields and MLP rows.
//
// No counterpart in the reference (it has no learned component). Layout:
//   parameters, one contiguous FP32 master array: for each layer l,
//     W_l [width[l+1]][width[l]] row-major, then b_l [width[l+1]];
//   a BF16 copy of the same array feeds the GEMMs; gradients, Adam moments
//   use the same offsets.
//   Activations are BF16 (the GEMM operands), pre-activations FP32.
// Operands live in buffers of the network's own, rows padded to 16 bytes, so
// that every tile load is a run of 16-byte asynchronous copies whatever the
// widths. One kernel does every product (mma.sync m16n8k16 BF16 x BF16 ->
// FP32): tiles of 64 x 64, or 32 x 32 where those would be too few for the
// SMs, four stages of operands in flight, either operand row-major along K or
// along its rows (ldmatrix transposes), and the epilogue fused: bias + GELU
// (hidden forward, keeping the FP32 pre-activation), bias (output layer), bias
// + MSE gradient and loss (output layer of a backward call), GELU' (backward),
// weight gradients with the bias gradients' column sums. A backward layer's
// two products are one launch.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "twmc.h"
#include "twmc_mlp_map.h"

namespace {

using twmc::LayerMap;
using twmc::weight_slot;

using bf16 = __nv_bfloat16;

constexpr int kStages = 4;

enum Epi { EPI_BIAS_GELU = 0, EPI_BIAS = 1, EPI_GELU_BWD = 2, EPI_DW = 3, EPI_MSE = 4 };

// C[m][n] = sum_k A(m, k) B(n, k). An operand is stored [row][k] (kmajor) or
// [k][row], ld elements apart (a multiple of 8, base 16-byte aligned).
struct GemmArgs {
  const bf16* A;
  int64_t lda;
  int a_kmajor;
  const bf16* B;
  int64_t ldb;
  int b_kmajor;
  int M, N, K;
  int epi;
  const float* bias;    // [N]            (EPI_BIAS_GELU, EPI_BIAS, EPI_MSE)
  const float* z;       // [M][ldf] FP32  (EPI_GELU_BWD)
  float* outf;          // [M][ldf] FP32  (EPI_BIAS_GELU: z, EPI_BIAS, EPI_DW)
  int64_t ldf;
  bf16* outh;           // [M][ldh] BF16  (EPI_BIAS_GELU: gelu(z), EPI_GELU_BWD, EPI_MSE: the loss gradient)
  int64_t ldh;
  float* colsum;        // [M] sums of A over k (EPI_DW: the bias gradients)
  const float* target;  // [M][N]         (EPI_MSE)
  const float* weight;  // [N] or NULL    (EPI_MSE)
  float* loss;          // (EPI_MSE)
  int tiles_n, tiles;
};
// Up to two products in one launch: CTAs [0, first.tiles) do the first.
struct GemmPair {
  GemmArgs g[2];
};

__device__ __forceinline__ float gelu_f(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
  return cdf + z * pdf;
}

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t sm_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
// 16 bytes from global to shared memory, `valid` of them read and the rest zero.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

// Bytes between consecutive lines of a tile: [R][BK] (kmajor) or [BK][R], 16
// bytes of padding so that the eight lines of an ldmatrix hit all banks.
template <int R, int BK> __device__ __forceinline__ constexpr int tile_pitch(bool kmajor) { return (kmajor ? BK : R) * 2 + 16; }
template <int R, int BK> constexpr int tile_bytes() {
  constexpr int a = R * (BK * 2 + 16), b = BK * (R * 2 + 16);
  return a > b ? a : b;
}

// One thread's share of an operand's R x BK tiles: kChunks pieces of 16 bytes,
// whose sources advance by one tile of k per call. Out of range is zero.
template <int R, int BK> struct TileLoader {
  static constexpr int kChunks = R * BK / 8 / 128;
  static_assert(R * BK % (8 * 128) == 0, "whole chunks per thread");
  const bf16* base;
  const bf16* src[kChunks];
  int dst[kChunks];
  int a[kChunks], b[kChunks];  // kmajor: elements left in the line (0: no such line); else lines left, elements in the line
  int64_t advance;
  bool kmajor;
  __device__ __forceinline__ TileLoader(const bf16* p, int64_t ld, bool km, int rows, int K, int r0) : base(p), kmajor(km) {
    advance = km ? BK : BK * ld;
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      const int id = threadIdx.x + i * 128;
      const int line = km ? id / (BK / 8) : id / (R / 8), c = (km ? id % (BK / 8) : id % (R / 8)) * 8;
      dst[i] = line * tile_pitch<R, BK>(km) + c * 2;
      if (km) {
        src[i] = p + int64_t(r0 + line) * ld + c;
        a[i] = r0 + line < rows ? K - c : 0;
        b[i] = 0;
      } else {
        src[i] = p + int64_t(line) * ld + r0 + c;
        a[i] = K - line;
        b[i] = min(max(rows - (r0 + c), 0), 8);
      }
    }
  }
  __device__ __forceinline__ void load(uint32_t tile) {
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      const int valid = kmajor ? min(max(a[i], 0), 8) : a[i] > 0 ? b[i] : 0;
      cp_async16(tile + uint32_t(dst[i]), valid ? src[i] : base, valid * 2);
      src[i] += advance;
      a[i] -= BK;
    }
  }
};

// What bounds a training step is latency: its products are 0.03 to 0.3 GFLOP, one
// after the other. Hence small tiles on many SMs, four stages of copies ahead
// of the tensor cores, and few launches. Measured on GB300 (5-256-256-256-2049,
// 128 rows): 660 us per step with two-byte loads, no copies ahead and 17
// launches, 72 us in this form with 10.
// The k16 products of an output are accumulated in ascending order, so
// the results do not depend on the tile.
template <int BM, int BN, int BK>
__global__ void __launch_bounds__(128) mlp_gemm_kernel(const __grid_constant__ GemmPair pair) {
  __shared__ __align__(16) unsigned char sA[kStages][tile_bytes<BM, BK>()];
  __shared__ __align__(16) unsigned char sB[kStages][tile_bytes<BN, BK>()];
  const bool second = int(blockIdx.x) >= pair.g[0].tiles;
  const GemmArgs& g = pair.g[second ? 1 : 0];
  const int tile = int(blockIdx.x) - (second ? pair.g[0].tiles : 0);
  const int m0 = (tile / g.tiles_n) * BM, n0 = (tile % g.tiles_n) * BN;
  const bool ak = g.a_kmajor != 0, bk = g.b_kmajor != 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;
  constexpr int MI = BM / 32, NI = BN / 16;  // 16-row and 8-column blocks of a warp (2 x 2 warps)
  const int wm = (warp >> 1) * (BM / 2), wn = (warp & 1) * (BN / 2);
  const int pa = tile_pitch<BM, BK>(ak), pb = tile_pitch<BN, BK>(bk);
  // ldmatrix source of this lane in an operand block (see the two layouts)
  const int mi = lane >> 3, r8 = lane & 7;
  const int a_off = ak ? (wm + (mi & 1) * 8 + r8) * pa + (mi >> 1) * 16 : ((mi >> 1) * 8 + r8) * pa + (wm + (mi & 1) * 8) * 2;
  const int b_off = bk ? (wn + (mi >> 1) * 8 + r8) * pb + (mi & 1) * 16 : ((mi & 1) * 8 + r8) * pb + (wn + (mi >> 1) * 8) * 2;
  float acc[MI][NI][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.0f;
  const int steps = (g.K + BK - 1) / BK;
  TileLoader<BM, BK> la(g.A, g.lda, ak, g.M, g.K, m0);
  TileLoader<BN, BK> lb(g.B, g.ldb, bk, g.N, g.K, n0);
  auto fetch = [&](int s) {
    if (s < steps) {
      la.load(sm_addr(sA[s % kStages]));
      lb.load(sm_addr(sB[s % kStages]));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) fetch(s);
  // column sums of A over k, ascending (the bias gradients), by the CTAs of the first column of tiles
  const bool sums = g.epi == EPI_DW && n0 == 0 && int(threadIdx.x) < BM;
  float csum = 0.0f;
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    fetch(s + kStages - 1);  // into the stage that the barrier has freed
    const uint32_t ta = sm_addr(sA[s % kStages]), tb = sm_addr(sB[s % kStages]);
#pragma unroll
    for (int kk = 0; kk < BK; kk += 16) {
      uint32_t af[MI][4], bfr[NI / 2][4];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        if (ak) ldmatrix4(af[i], ta + uint32_t(a_off + i * 16 * pa + kk * 2));
        else ldmatrix4_trans(af[i], ta + uint32_t(a_off + i * 32 + kk * pa));
      }
#pragma unroll
      for (int j = 0; j < NI / 2; ++j) {
        if (bk) ldmatrix4(bfr[j], tb + uint32_t(b_off + j * 16 * pb + kk * 2));
        else ldmatrix4_trans(bfr[j], tb + uint32_t(b_off + j * 32 + kk * pb));
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j) {
          const uint32_t b2[2] = {bfr[j / 2][(j & 1) * 2], bfr[j / 2][(j & 1) * 2 + 1]};
          mma_bf16_16816(acc[i][j], af[i], b2);
        }
    }
    if (sums) {
#pragma unroll 8
      for (int k = 0; k < BK; ++k)
        csum += __bfloat162float(*reinterpret_cast<const bf16*>(
            sA[s % kStages] + (ak ? threadIdx.x * pa + k * 2 : k * pa + threadIdx.x * 2)));
    }
  }
  if (sums && m0 + int(threadIdx.x) < g.M) g.colsum[m0 + threadIdx.x] = csum;
  float part = 0.0f;
  const float inv = 1.0f / float(int64_t(g.M) * g.N);
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NI; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int row = m0 + wm + i * 16 + gq + 8 * h;
          const int col = n0 + wn + j * 8 + 2 * tq + c;
          if (row >= g.M || col >= g.N) continue;
          const float v = acc[i][j][2 * h + c];
          const int64_t fi = int64_t(row) * g.ldf + col, hi = int64_t(row) * g.ldh + col;
          if (g.epi == EPI_BIAS_GELU) {
            const float z = v + g.bias[col];
            g.outf[fi] = z;
            g.outh[hi] = __float2bfloat16(gelu_f(z));
          } else if (g.epi == EPI_BIAS) {
            g.outf[fi] = v + g.bias[col];
          } else if (g.epi == EPI_GELU_BWD) {
            g.outh[hi] = __float2bfloat16(v * gelu_grad(g.z[fi]));
          } else if (g.epi == EPI_DW) {
            g.outf[fi] = v;
          } else {  // dy = bf16(2 w_o (y - t) / (M O)); loss += sum w_o (y - t)^2 / (M O)
            const float wo = g.weight ? g.weight[col] : 1.0f;
            const float e = (v + g.bias[col]) - g.target[int64_t(row) * g.N + col];
            part += wo * e * e;
            g.outh[hi] = __float2bfloat16(2.0f * wo * e * inv);
          }
        }
  if (g.epi == EPI_MSE) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    __shared__ float red[4];
    if (lane == 0) red[warp] = part;
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(g.loss, ((red[0] + red[1]) + (red[2] + red[3])) * inv);
  }
}

// BF16 copy of x [rows][cols] into y, ld apart; zeroes *loss (NULL: none).
__global__ void cast_input_kernel(const float* __restrict__ x, int64_t rows, int cols, bf16* __restrict__ y, int64_t ld,
                                  float* __restrict__ loss) {
  if (loss && blockIdx.x == 0 && threadIdx.x == 0) *loss = 0.0f;
  const int64_t n = rows * cols;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    y[(i / cols) * ld + i % cols] = __float2bfloat16(x[i]);
}

// The BF16 copy of every layer's weights: grid (rows, layer).
__global__ void cast_params_kernel(const float* __restrict__ w, bf16* __restrict__ w16, const __grid_constant__ LayerMap m) {
  const int l = blockIdx.y, K = m.k[l];
  for (int r = blockIdx.x; r < m.n[l]; r += gridDim.x)
    for (int c = threadIdx.x; c < K; c += blockDim.x)
      w16[m.h[l] + int64_t(r) * m.ld[l] + c] = __float2bfloat16(w[m.off[l] + int64_t(r) * K + c]);
}

// Adam (Kingma & Ba 2015) on the FP32 master copy, P parameters per thread (1 or
// 4); refreshes the BF16 copy. c1 = 1 / (1 - beta1^t), c2 = 1 / (1 - beta2^t).
__device__ __forceinline__ float adam_one(float w, float g, float& m, float& v, float lr, float b1, float b2, float eps,
                                          float c1, float c2) {
  // (one rounding for each form of the kernel: left to the compiler, the two
  // contracted these sums differently)
  m = __fmaf_rn(1.0f - b1, g, __fmul_rn(b1, m));
  v = __fmaf_rn(__fmul_rn(1.0f - b2, g), g, __fmul_rn(b2, v));
  return w - lr * (m * c1) / (sqrtf(v * c2) + eps);
}
// Parameters from which P is 4. GB300, us per step with 1 and 4 per thread:
// 5 thousand 4.1 / 6.2, 265 thousand 5.3 / 6.3, 660 thousand 8.4 / 7.4, 2.1 million
// 14.6 / 12.5, 33.6 million 209 / 158.
constexpr int64_t kAdamWide = 1 << 19;
template <int P>
__global__ void adam_kernel(float* __restrict__ w, bf16* __restrict__ w16, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, int64_t n, const __grid_constant__ LayerMap lm,
                            int nl, float lr, float b1, float b2, float eps, float c1, float c2) {
  if constexpr (P == 1) {
    int l = 0;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
      float mi = m[i], vi = v[i];
      const float wi = adam_one(w[i], g[i], mi, vi, lr, b1, b2, eps, c1, c2);
      w[i] = wi; m[i] = mi; v[i] = vi;
      while (l + 1 < nl && i >= lm.off[l + 1]) ++l;
      const int64_t slot = weight_slot(lm, l, i);
      if (slot >= 0) w16[slot] = __float2bfloat16(wi);
    }
    return;
  }
  for (int64_t i = 4 * (blockIdx.x * int64_t(blockDim.x) + threadIdx.x); i < n; i += 4 * int64_t(gridDim.x) * blockDim.x) {
    float wv[4], gv[4], mv[4], vv[4];
    const int cnt = int(min(int64_t(4), n - i));
    if (cnt == 4) {
      *reinterpret_cast<float4*>(wv) = *reinterpret_cast<const float4*>(w + i);
      *reinterpret_cast<float4*>(gv) = *reinterpret_cast<const float4*>(g + i);
      *reinterpret_cast<float4*>(mv) = *reinterpret_cast<const float4*>(m + i);
      *reinterpret_cast<float4*>(vv) = *reinterpret_cast<const float4*>(v + i);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (c < cnt) { wv[c] = w[i + c]; gv[c] = g[i + c]; mv[c] = m[i + c]; vv[c] = v[i + c]; }
        else wv[c] = gv[c] = mv[c] = vv[c] = 0.0f;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) wv[c] = adam_one(wv[c], gv[c], mv[c], vv[c], lr, b1, b2, eps, c1, c2);
    if (cnt == 4) {
      *reinterpret_cast<float4*>(w + i) = *reinterpret_cast<const float4*>(wv);
      *reinterpret_cast<float4*>(m + i) = *reinterpret_cast<const float4*>(mv);
      *reinterpret_cast<float4*>(v + i) = *reinterpret_cast<const float4*>(vv);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (c < cnt) { w[i + c] = wv[c]; m[i + c] = mv[c]; v[i + c] = vv[c]; }
    }
    int l = 0;
    while (l + 1 < nl && i >= lm.off[l + 1]) ++l;
    const int64_t first = weight_slot(lm, l, i);
    if (first >= 0 && i + 3 < (l + 1 < nl ? lm.off[l + 1] : n) && weight_slot(lm, l, i + 3) == first + 3) {  // side by side
#pragma unroll
      for (int c = 0; c < 4; ++c) w16[first + c] = __float2bfloat16(wv[c]);
      continue;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c >= cnt) break;
      if (l + 1 < nl && i + c >= lm.off[l + 1]) ++l;
      const int64_t slot = weight_slot(lm, l, i + c);
      if (slot >= 0) w16[slot] = __float2bfloat16(wv[c]);
    }
  }
}

// Optional squash v -> asinh(v / s) (s > 0): log-like beyond |v| ~ s, so a
// column spanning decades is fitted to relative accuracy.
__device__ __forceinline__ double squash_f(double v, double s) { return s > 0.0 ? asinh(v / s) : v; }
__device__ __forceinline__ double unsquash_f(double v, double s) { return s > 0.0 ? s * sinh(v) : v; }

__global__ void squash_kernel(float* __restrict__ t, int64_t n, double s) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    t[i] = float(squash_f(double(t[i]), s));
}

// Column statistics of t [rows][cols] in FP64: mean and standard deviation.
__global__ void colstats_kernel(const float* __restrict__ t, int64_t rows, int cols, float* __restrict__ mean,
                                float* __restrict__ stdv) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  double s = 0.0, s2 = 0.0;
  for (int64_t r = 0; r < rows; ++r) s += double(t[r * cols + c]);
  const double mu = s / double(rows);
  for (int64_t r = 0; r < rows; ++r) {
    const double e = double(t[r * cols + c]) - mu;
    s2 += e * e;
  }
  mean[c] = float(mu);
  stdv[c] = float(sqrt(s2 / double(rows > 1 ? rows - 1 : 1)));
}

// With m = max_c std_c: w_c = clamp((std_c / m)^2, 1e-4, 1) (optional), then
// std_c = max(std_c, floor_frac m); one CTA.
__global__ void stdfloor_kernel(float* __restrict__ stdv, int cols, float floor_frac, float* __restrict__ w) {
  __shared__ float red[32];
  float mx = 0.0f;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) mx = fmaxf(mx, stdv[c]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  const float m = fmaxf(red[0], 1e-30f);
  const float fl = fmaxf(floor_frac * m, 1e-30f);
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    const float r = stdv[c] / m;
    if (w) w[c] = fminf(fmaxf(r * r, 1e-4f), 1.0f);
    stdv[c] = fmaxf(stdv[c], fl);
  }
}

__global__ void normalize_kernel(float* __restrict__ t, int64_t rows, int cols, const float* __restrict__ mean,
                                 const float* __restrict__ stdv) {
  const int64_t n = rows * cols;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int c = int(i % cols);
    t[i] = (t[i] - mean[c]) / stdv[c];
  }
}

// Separable unitary 2-D DFT of one nx x ny field held in shared memory
// (site p = x ny + y, natural k order k = kx ny + ky):
//   out_k = N^{-1/2} sum_p in_p exp(sign 2 pi i (kx x / nx + ky y / ny)).
// FP64 with exact twiddle phases (the integer product is reduced mod n).
__device__ void dft2_shared(const double2* in, double2* tmp, double2* out, int nx, int ny, double sign) {
  const int n = nx * ny;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {  // along y
    const int x = i / ny, ky = i % ny;
    double sr = 0.0, si = 0.0;
    for (int y = 0; y < ny; ++y) {
      double s, c;
      sincospi(sign * 2.0 * double((int64_t(ky) * y) % ny) / double(ny), &s, &c);
      const double2 v = in[x * ny + y];
      sr += v.x * c - v.y * s;
      si += v.x * s + v.y * c;
    }
    tmp[i] = make_double2(sr, si);
  }
  __syncthreads();
  const double norm = rsqrt(double(n));
  for (int i = threadIdx.x; i < n; i += blockDim.x) {  // along x
    const int kx = i / ny, ky = i % ny;
    double sr = 0.0, si = 0.0;
    for (int x = 0; x < nx; ++x) {
      double s, c;
      sincospi(sign * 2.0 * double((int64_t(kx) * x) % nx) / double(nx), &s, &c);
      const double2 v = tmp[x * ny + ky];
      sr += v.x * c - v.y * s;
      si += v.x * s + v.y * c;
    }
    out[i] = make_double2(sr * norm, si * norm);
  }
  __syncthreads();
}

// One MLP target row per point: (Re a_k, Im a_k) for every k, then the
// density n = mean_p <|a_p|^2> - 1/2, with a_k the unitary DFT of the mean
// field <a_p>. Inputs are sums over `frames` frames (scale = 1 / frames).
__global__ void targets_kernel(const double* __restrict__ mean, const double* __restrict__ abs2, int nx, int ny,
                               double scale, float* __restrict__ rows, int64_t ld) {
  extern __shared__ __align__(16) double2 sm[];
  const int n = nx * ny;
  double2* a = sm;
  double2* tmp = sm + n;
  const int64_t pt = blockIdx.x;
  const double* mp = mean + pt * 2 * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = make_double2(mp[2 * i] * scale, mp[2 * i + 1] * scale);
  __syncthreads();
  dft2_shared(a, tmp, a, nx, ny, -1.0);
  float* r = rows + pt * ld;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    r[2 * i] = float(a[i].x);
    r[2 * i + 1] = float(a[i].y);
  }
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += abs2[pt * n + i] * scale;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < int(blockDim.x >> 5); ++i) t += red[i];
    r[2 * n] = float(t / double(n) - 0.5);
  }
}

// Initial fields from one MLP output row per point (de-standardised with
// mean / std when given, then un-squashed): beta_init = inverse unitary DFT
// of the predicted k-mode amplitudes; beta_sigma = sqrt((n_inc + 1/2) / 2)
// per quadrature with n_inc = min(max(n - |beta_init|^2, 0), max_inc), so
// that <|a|^2>_W - 1/2 starts at the predicted density n (vacuum: 1/2) unless
// the incoherent part is capped.
__global__ void fields_kernel(const float* __restrict__ rows, int64_t ld, const float* __restrict__ mu,
                              const float* __restrict__ sd, double squash, double max_inc, int nx, int ny,
                              double* __restrict__ binit, double* __restrict__ bsigma) {
  extern __shared__ __align__(16) double2 sm[];
  const int n = nx * ny;
  double2* a = sm;
  double2* tmp = sm + n;
  const int64_t pt = blockIdx.x;
  const float* r = rows + pt * ld;
  auto val = [&](int c) {
    const double v = mu ? double(r[c]) * double(sd[c]) + double(mu[c]) : double(r[c]);
    return unsquash_f(v, squash);
  };
  for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = make_double2(val(2 * i), val(2 * i + 1));
  __syncthreads();
  dft2_shared(a, tmp, a, nx, ny, 1.0);
  const double dens = val(2 * n);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double m2 = a[i].x * a[i].x + a[i].y * a[i].y;
    const double sg = sqrt((fmin(fmax(dens - m2, 0.0), max_inc) + 0.5) * 0.5);
    binit[(pt * n + i) * 2] = a[i].x;
    binit[(pt * n + i) * 2 + 1] = a[i].y;
    bsigma[(pt * n + i) * 2] = sg;
    bsigma[(pt * n + i) * 2 + 1] = 0.0;
  }
}

template <typename T>
struct DevArr {
  T* p = nullptr;
  ~DevArr() { if (p) cudaFree(p); }
  bool alloc(size_t n) {
    if (p) cudaFree(p);
    p = nullptr;
    return n == 0 || cudaMalloc(&p, n * sizeof(T)) == cudaSuccess;
  }
};

int grid_for(int64_t n, int cta) { return int(std::max<int64_t>(1, std::min<int64_t>((n + cta - 1) / cta, 4096))); }

}  // namespace

struct twmc_mlp {
  int device = 0;
  int nl = 0;
  std::vector<int> width;
  std::vector<int64_t> w_off, b_off;
  int64_t nparam = 0, max_batch = 0, step = 0;
  int max_width = 0;
  DevArr<float> w, g, m, v;
  DevArr<bf16> w16;
  LayerMap map{};
  std::vector<DevArr<bf16>> act;  // act[l]: input of layer l, [max_batch][pad8(width[l])]
  std::vector<DevArr<float>> z;   // z[l]: pre-activation output of layer l-1, [max_batch][width[l]] (l = 1..nl-1)
  DevArr<bf16> d0, d1;            // backward ping-pong, [max_batch][pad8(width)]
  DevArr<float> loss;
  int64_t launches = 0;
  std::string err;
};

namespace {

int mfail(twmc_mlp* m, int code, const std::string& s) {
  if (m) m->err = s;
  return code;
}

int64_t pad8(int64_t n) { return (n + 7) & ~int64_t(7); }

// One launch of one product, or of two that depend on the same input: 64 x 64
// tiles where they come to at least 96 CTAs and no sum is long, else 32 x 32
// with 64 of K at a time (on 64 x 64 tiles a sum over 2049 ran on 8 CTAs, 47 us
// of a training step's 119).
bool gemm(twmc_mlp* m, GemmArgs a, cudaStream_t s, const GemmArgs* b = nullptr) {
  GemmPair p{};
  auto tiles = [](GemmArgs& g, int t) {
    g.tiles_n = (g.N + t - 1) / t;
    g.tiles = ((g.M + t - 1) / t) * g.tiles_n;
    return int64_t(g.tiles);
  };
  p.g[0] = a;
  if (b) p.g[1] = *b;
  int64_t n = tiles(p.g[0], 64) + (b ? tiles(p.g[1], 64) : 0);
  if (n >= 96 && std::max(p.g[0].K, p.g[1].K) <= 512) {
    mlp_gemm_kernel<64, 64, 32><<<unsigned(n), 128, 0, s>>>(p);
  } else {
    n = tiles(p.g[0], 32) + (b ? tiles(p.g[1], 32) : 0);
    mlp_gemm_kernel<32, 32, 64><<<unsigned(n), 128, 0, s>>>(p);
  }
  ++m->launches;
  return cudaPeekAtLastError() == cudaSuccess;
}

// Forward pass of `batch` rows of x (device FP32 [batch][width[0]]), keeping
// activations for the backward. The output layer goes to yout (device FP32
// [batch][width[nl]]), or, with a target, to the loss and its gradient (d0).
bool forward_chunk(twmc_mlp* m, const float* x, int64_t batch, float* yout, cudaStream_t s,
                   const float* target = nullptr, const float* weight = nullptr) {
  const int64_t nin = batch * m->width[0];
  cast_input_kernel<<<grid_for(nin, 256), 256, 0, s>>>(x, batch, m->width[0], m->act[0].p, pad8(m->width[0]),
                                                       target ? m->loss.p : nullptr);
  ++m->launches;
  for (int l = 0; l < m->nl; ++l) {
    const int K = m->width[l], N = m->width[l + 1];
    GemmArgs g{};
    g.A = m->act[l].p; g.lda = pad8(K); g.a_kmajor = 1;
    g.B = m->w16.p + m->map.h[l]; g.ldb = m->map.ld[l]; g.b_kmajor = 1;
    g.M = int(batch); g.N = N; g.K = K;
    g.bias = m->w.p + m->b_off[l];
    g.ldf = N;
    if (l + 1 < m->nl) {
      g.epi = EPI_BIAS_GELU;
      g.outf = m->z[l + 1].p;
      g.outh = m->act[l + 1].p;
      g.ldh = pad8(N);
    } else if (target) {
      g.epi = EPI_MSE;
      g.target = target;
      g.weight = weight;
      g.loss = m->loss.p;
      g.outh = m->d0.p;
      g.ldh = pad8(N);
    } else {
      g.epi = EPI_BIAS;
      g.outf = yout;
    }
    if (!gemm(m, g, s)) return false;
  }
  return true;
}

bool fields_smem_ok(int64_t nx, int64_t ny, size_t* smem) {
  const int64_t n = nx * ny;
  if (nx < 1 || ny < 1 || n > 4096) return false;
  *smem = size_t(2 * n) * sizeof(double2);
  return true;
}

}  // namespace

extern "C" {

int twmc_mlp_create(int32_t n_layers, const int32_t* widths, int64_t max_batch, uint64_t seed, twmc_mlp** out) {
  if (!out || !widths || n_layers < 1 || n_layers > 16 || max_batch < 1 || max_batch > (int64_t(1) << 24))
    return TWMC_ERR_INVALID;
  *out = nullptr;
  for (int l = 0; l <= n_layers; ++l)
    if (widths[l] < 1 || widths[l] > 65536) return TWMC_ERR_INVALID;
  auto* m = new twmc_mlp;
  cudaGetDevice(&m->device);
  m->nl = n_layers;
  m->width.assign(widths, widths + n_layers + 1);
  m->max_batch = max_batch;
  int64_t off = 0;
  for (int l = 0; l < n_layers; ++l) {
    m->w_off.push_back(off);
    off += int64_t(widths[l + 1]) * widths[l];
    m->b_off.push_back(off);
    off += widths[l + 1];
  }
  m->nparam = off;
  int64_t h = 0;
  for (int l = 0; l < n_layers; ++l) {
    m->map.off[l] = m->w_off[l];
    m->map.n[l] = widths[l + 1];
    m->map.k[l] = widths[l];
    m->map.ld[l] = int(pad8(widths[l]));
    m->map.h[l] = h;
    h += int64_t(widths[l + 1]) * m->map.ld[l];
  }
  m->max_width = *std::max_element(m->width.begin(), m->width.end());
  m->act.resize(n_layers);
  m->z.resize(n_layers);
  bool ok = m->w.alloc(off) && m->g.alloc(off) && m->m.alloc(off) && m->v.alloc(off) && m->w16.alloc(h) &&
            m->d0.alloc(size_t(max_batch) * pad8(m->max_width)) && m->d1.alloc(size_t(max_batch) * pad8(m->max_width)) &&
            m->loss.alloc(1);
  for (int l = 0; l < n_layers && ok; ++l) {
    ok = m->act[l].alloc(size_t(max_batch) * pad8(widths[l]));
    if (ok && l > 0) ok = m->z[l].alloc(size_t(max_batch) * widths[l]);
  }
  if (!ok) {
    cudaGetLastError();
    delete m;
    return TWMC_ERR_NOMEM;
  }
  // Glorot-uniform weights, zero biases, from a seeded host generator.
  std::vector<float> p(size_t(off), 0.0f);
  std::mt19937_64 gen(seed);
  for (int l = 0; l < n_layers; ++l) {
    const double a = std::sqrt(6.0 / double(widths[l] + widths[l + 1]));
    std::uniform_real_distribution<double> u(-a, a);
    for (int64_t i = 0; i < int64_t(widths[l + 1]) * widths[l]; ++i) p[size_t(m->w_off[l] + i)] = float(u(gen));
  }
  *out = m;
  return twmc_mlp_set_params(m, p.data());
}

int64_t twmc_mlp_param_count(const twmc_mlp* m) { return m ? m->nparam : -1; }

int twmc_mlp_set_params(twmc_mlp* m, const float* host) {
  if (!m || !host) return TWMC_ERR_INVALID;
  cudaSetDevice(m->device);
  const size_t n = size_t(m->nparam);
  if (cudaMemcpy(m->w.p, host, n * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(m->m.p, 0, n * sizeof(float)) != cudaSuccess || cudaMemset(m->v.p, 0, n * sizeof(float)) != cudaSuccess ||
      cudaMemset(m->g.p, 0, n * sizeof(float)) != cudaSuccess)
    return mfail(m, TWMC_ERR_CUDA, "parameter upload failed");
  cast_params_kernel<<<dim3(unsigned(std::min(m->max_width, 4096)), unsigned(m->nl)), 256>>>(m->w.p, m->w16.p, m->map);
  ++m->launches;
  m->step = 0;
  const cudaError_t e = cudaDeviceSynchronize();
  return e == cudaSuccess ? TWMC_OK : mfail(m, TWMC_ERR_CUDA, cudaGetErrorString(e));
}

int twmc_mlp_get_params(twmc_mlp* m, float* host) {
  if (!m || !host) return TWMC_ERR_INVALID;
  cudaSetDevice(m->device);
  cudaDeviceSynchronize();
  return cudaMemcpy(host, m->w.p, size_t(m->nparam) * sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess
             ? TWMC_OK
             : mfail(m, TWMC_ERR_CUDA, "parameter download failed");
}

int twmc_mlp_get_grads(twmc_mlp* m, float* host) {
  if (!m || !host) return TWMC_ERR_INVALID;
  cudaSetDevice(m->device);
  cudaDeviceSynchronize();
  return cudaMemcpy(host, m->g.p, size_t(m->nparam) * sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess
             ? TWMC_OK
             : mfail(m, TWMC_ERR_CUDA, "gradient download failed");
}

int twmc_mlp_forward(twmc_mlp* m, const float* x, int64_t batch, float* y, void* stream) {
  if (!m || !x || !y || batch < 0) return TWMC_ERR_INVALID;
  cudaSetDevice(m->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (int64_t r = 0; r < batch; r += m->max_batch) {
    const int64_t b = std::min(m->max_batch, batch - r);
    if (!forward_chunk(m, x + r * m->width[0], b, y + r * m->width[m->nl], s)) {
      cudaGetLastError();
      return mfail(m, TWMC_ERR_CUDA, "forward launch failed");
    }
  }
  return TWMC_OK;
}

int twmc_mlp_backward(twmc_mlp* m, const float* x, const float* target, const float* weights, int64_t batch,
                      float* loss, void* stream) {
  if (!m || !x || !target || batch < 1 || batch > m->max_batch) return TWMC_ERR_INVALID;
  cudaSetDevice(m->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!forward_chunk(m, x, batch, nullptr, s, target, weights)) { cudaGetLastError(); return mfail(m, TWMC_ERR_CUDA, "forward launch failed"); }
  bf16* dcur = m->d0.p;
  bf16* dnext = m->d1.p;
  for (int l = m->nl - 1; l >= 0; --l) {
    const int K = m->width[l], N = m->width[l + 1];
    // dW_l[n][k] = sum_b dZ[b][n] act_l[b][k], db_l[n] = sum_b dZ[b][n]
    GemmArgs gw{};
    gw.A = dcur; gw.lda = pad8(N);
    gw.B = m->act[l].p; gw.ldb = pad8(K);
    gw.M = N; gw.N = K; gw.K = int(batch);
    gw.epi = EPI_DW;
    gw.outf = m->g.p + m->w_off[l];
    gw.ldf = K;
    gw.colsum = m->g.p + m->b_off[l];
    // dZ_{l-1}[b][k] = (sum_n dZ[b][n] W_l[n][k]) gelu'(z_l[b][k])
    GemmArgs gd{};
    if (l > 0) {
      gd.A = dcur; gd.lda = pad8(N); gd.a_kmajor = 1;
      gd.B = m->w16.p + m->map.h[l]; gd.ldb = m->map.ld[l];
      gd.M = int(batch); gd.N = K; gd.K = N;
      gd.epi = EPI_GELU_BWD;
      gd.z = m->z[l].p;
      gd.ldf = K;
      gd.outh = dnext;
      gd.ldh = pad8(K);
    }
    // the longer sum's tiles first
    const bool ok = l > 0 ? gemm(m, gd, s, &gw) : gemm(m, gw, s);
    if (!ok) { cudaGetLastError(); return mfail(m, TWMC_ERR_CUDA, "backward launch failed"); }
    std::swap(dcur, dnext);
  }
  if (loss) {
    if (cudaMemcpyAsync(loss, m->loss.p, sizeof(float), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return mfail(m, TWMC_ERR_CUDA, "loss download failed");
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TWMC_OK : mfail(m, TWMC_ERR_CUDA, cudaGetErrorString(e));
}

int twmc_mlp_adam(twmc_mlp* m, float lr, float beta1, float beta2, float eps, void* stream) {
  if (!m || !(lr >= 0.0f) || !(beta1 >= 0.0f && beta1 < 1.0f) || !(beta2 >= 0.0f && beta2 < 1.0f) || !(eps > 0.0f))
    return TWMC_ERR_INVALID;
  cudaSetDevice(m->device);
  ++m->step;
  const float c1 = float(1.0 / (1.0 - std::pow(double(beta1), double(m->step))));
  const float c2 = float(1.0 / (1.0 - std::pow(double(beta2), double(m->step))));
  const int per = m->nparam < kAdamWide ? 1 : 4;
  (per == 1 ? adam_kernel<1> : adam_kernel<4>)<<<grid_for((m->nparam + per - 1) / per, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      m->w.p, m->w16.p, m->g.p, m->m.p, m->v.p, m->nparam, m->map, m->nl, lr, beta1, beta2, eps, c1, c2);
  ++m->launches;
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TWMC_OK : mfail(m, TWMC_ERR_CUDA, cudaGetErrorString(e));
}

int twmc_mlp_last_loss(twmc_mlp* m, float* loss) {
  if (!m || !loss) return TWMC_ERR_INVALID;
  cudaSetDevice(m->device);
  cudaDeviceSynchronize();
  return cudaMemcpy(loss, m->loss.p, sizeof(float), cudaMemcpyDeviceToHost) == cudaSuccess
             ? TWMC_OK
             : mfail(m, TWMC_ERR_CUDA, "loss download failed");
}

const char* twmc_mlp_last_error(const twmc_mlp* m) { return m ? m->err.c_str() : "null network"; }
int64_t twmc_mlp_launch_count(const twmc_mlp* m) { return m ? m->launches : -1; }
void twmc_mlp_destroy(twmc_mlp* m) { delete m; }

int twmc_mlp_standardize(float* t, int64_t rows, int32_t cols, double squash, float floor_frac, float* mean,
                         float* stdv, float* weights, void* stream) {
  if (!t || !mean || !stdv || rows < 1 || cols < 1 || !(floor_frac >= 0.0f) || !(squash >= 0.0))
    return TWMC_ERR_INVALID;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (squash > 0.0) squash_kernel<<<grid_for(rows * cols, 256), 256, 0, s>>>(t, rows * cols, squash);
  colstats_kernel<<<(cols + 127) / 128, 128, 0, s>>>(t, rows, cols, mean, stdv);
  stdfloor_kernel<<<1, 1024, 0, s>>>(stdv, cols, floor_frac, weights);
  normalize_kernel<<<grid_for(rows * cols, 256), 256, 0, s>>>(t, rows, cols, mean, stdv);
  return cudaGetLastError() == cudaSuccess ? TWMC_OK : TWMC_ERR_CUDA;
}

int twmc_mlp_targets(const double* mean, const double* abs2, int64_t n_points, int64_t nx, int64_t ny,
                     int32_t frames, float* rows, int64_t ld, void* stream) {
  size_t smem = 0;
  if (!mean || !abs2 || !rows || n_points < 1 || frames < 1 || !fields_smem_ok(nx, ny, &smem) || ld < 2 * nx * ny + 1)
    return TWMC_ERR_INVALID;
  if (cudaFuncSetAttribute(targets_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) {
    cudaGetLastError();
    return TWMC_ERR_CUDA;
  }
  targets_kernel<<<unsigned(n_points), 256, smem, static_cast<cudaStream_t>(stream)>>>(
      mean, abs2, int(nx), int(ny), 1.0 / double(frames), rows, ld);
  return cudaGetLastError() == cudaSuccess ? TWMC_OK : TWMC_ERR_CUDA;
}

int twmc_mlp_fields(const float* rows, int64_t ld, int64_t n_points, const float* mean, const float* stdv,
                    double squash, double max_incoherent, int64_t nx, int64_t ny, double* beta_init,
                    double* beta_sigma, void* stream) {
  size_t smem = 0;
  if (!rows || !beta_init || !beta_sigma || n_points < 1 || !fields_smem_ok(nx, ny, &smem) ||
      ld < 2 * nx * ny + 1 || (!mean) != (!stdv) || !(squash >= 0.0) || !(max_incoherent >= 0.0))
    return TWMC_ERR_INVALID;
  if (cudaFuncSetAttribute(fields_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) {
    cudaGetLastError();
    return TWMC_ERR_CUDA;
  }
  fields_kernel<<<unsigned(n_points), 256, smem, static_cast<cudaStream_t>(stream)>>>(
      rows, ld, mean, stdv, squash, max_incoherent, int(nx), int(ny), beta_init, beta_sigma);
  return cudaGetLastError() == cudaSuccess ? TWMC_OK : TWMC_ERR_CUDA;
}

}  // extern "C"
