// twmc_mlp_map.h -- where the warm-start MLP's parameters lie: W_l [n][k] and
// then b_l [n] at `off` of the FP32 arrays, the BF16 copy of W_l at `h`, ld
// apart.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define TWMC_HD __host__ __device__ __forceinline__
#else
#define TWMC_HD inline
#endif

namespace twmc {

constexpr int kMaxLayers = 16;
struct LayerMap {
  int64_t off[kMaxLayers], h[kMaxLayers];
  int n[kMaxLayers], k[kMaxLayers], ld[kMaxLayers];
};

// Element of the BF16 copy that holds parameter i, of layer l, or -1 for a
// bias. n k is at most 2^32 (65536 x 65536), the biases lie beyond: the range
// is tested in 64 bits, and a weight's offset divided in 32.
TWMC_HD int64_t weight_slot(const LayerMap& m, int l, int64_t i) {
  const int64_t o = i - m.off[l];
  if (o >= int64_t(m.n[l]) * m.k[l]) return -1;
  const uint32_t at = uint32_t(o), r = at / uint32_t(m.k[l]);
  return m.h[l] + int64_t(r) * m.ld[l] + (at - r * uint32_t(m.k[l]));
}

}  // namespace twmc
