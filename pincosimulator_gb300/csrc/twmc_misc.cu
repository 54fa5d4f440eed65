// twmc_misc.cu -- one-off kernels: initial fields and disorder draws (FP64,
// Philox streams), the FP64 ensemble reduction, and the Philox self-check.
#include <algorithm>

#include "twmc_common.cuh"
#include "twmc_launch.h"
#include "twmc_moments.cuh"

namespace twmc {

namespace {

__device__ __forceinline__ double2 ld_c(const double* p, int64_t i) { return make_double2(p[2 * i], p[2 * i + 1]); }

// One trajectory-site of the initial state (TWMCBaseSolver.cpp:126-151 /
// TWMCLiebSolver.cpp:145-171 with the noise drawn from Philox streams).
// FP32 runs draw the normals with the FP32 Box-Muller of the Wiener noise,
// FP64 runs with the FP64 one; the sums with the base values are FP64 in
// both. (The FP64 logarithm and sine / cosine of two draws per site took
// 20 ms for 16384 trajectories of 64 x 64 on GB300's narrow FP64 pipe.)
template <int PREC>
__device__ __forceinline__ double2 init_normal(uint32_t a, uint32_t b) {
  if constexpr (PREC == 0) {
    const float2 z = normal_pair(a, b, 0.0f);
    return make_double2(widen(z.x), widen(z.y));
  } else {
    return normal_pair(a, b, 0.0);
  }
}
// One thread per pair of sites (p, p + half), which share each stream's Philox
// call. The FP64 pipe bounds it on FP32 runs too: what is zero (imaginary parts
// of spread and amplitude) or not asked for (matrices without disorder, array
// or realisation) is left out, and conversions are integer operations; 16.8 M
// sites with omega disorder took 0.74 ms with one thread per site and all three
// matrices formed, now 0.29.
template <int PREC>
__device__ __forceinline__ void store_c(void* p, int64_t i, double2 v) {
  if constexpr (PREC == 0) reinterpret_cast<float2*>(p)[i] = make_float2(narrow(v.x), narrow(v.y));
  else reinterpret_cast<double2*>(p)[i] = v;
}
template <int PREC>
__global__ void init_kernel(const InitArgs a) {
  const int64_t half = (a.nsites + 1) / 2, total = a.ntraj * half;
  const double half_gamma = a.gamma / 2.0;
  for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < total; k += int64_t(gridDim.x) * blockDim.x) {
    const int64_t tr = total <= 0xffffffffll ? int64_t(uint32_t(k) / uint32_t(half)) : k / half, c0 = k - tr * half;
    const uint32_t seed = a.seeds[tr], id = a.ids[tr];
    const int ns = c0 + half < a.nsites ? 2 : 1;
    u32x4 w{};
    if (a.ic_kind == 0) w = philox4x32_10(u32x4{uint32_t(c0), 0u, kStreamInit, 0u}, seed, id);
    for (int s = 0; s < ns; ++s) {
      const int64_t p = c0 + s * half, i = tr * a.nsites + p;
      double2 b;
      if (a.ic_kind == 2) {
        b = ld_c(a.given, i);
      } else {
        b = a.binit ? ld_c(a.binit, p) : make_double2(a.binit_s[0], a.binit_s[1]);
        if (a.ic_kind == 0) {
          const double2 z = s ? init_normal<PREC>(w.z, w.w) : init_normal<PREC>(w.x, w.y);
          const double2 sg = a.bsigma ? ld_c(a.bsigma, p) : make_double2(a.bsigma_s[0], a.bsigma_s[1]);
          double2 e = make_double2(__dmul_rn(sg.x, z.x), __dmul_rn(sg.x, z.y));
          if (!is_zero(sg.y)) e = make_double2(fma_rare(-sg.y, z.y, e.x), fma_rare(sg.y, z.x, e.y));
          b = cadd(b, e);
        }
      }
      store_c<PREC>(a.state, i, b);
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {  // U, omega (Lieb: E), F
      void* const dst = m == 0 ? a.iU : m == 1 ? a.rsl : a.iF;
      if (!dst && !a.real_out[m]) continue;
      const bool draw = !a.given_real[m] && a.kind[m] != 0;
      u32x4 u{};
      if (draw) u = philox4x32_10(u32x4{uint32_t(c0), 0u, a.stream[m], 0u}, seed, id);
      for (int s = 0; s < ns; ++s) {
        const int64_t p = c0 + s * half, i = tr * a.nsites + p;
        double2 v;
        if (a.given_real[m]) {
          v = ld_c(a.given_real[m], i);
        } else {
          v = a.base[m] ? ld_c(a.base[m], p) : make_double2(a.base_s[m][0], a.base_s[m][1]);
          if (draw) {
            uint32_t u0 = s ? u.z : u.x, u1 = s ? u.w : u.y;
            const double2 amp = ld_c(a.amp[m], p);
            if (a.kind[m] == 1) {
              const double2 z = init_normal<PREC>(u0, u1);
              v.x += z.x * amp.x;
              if (!is_zero(amp.y)) v.y = fma_rare(z.y, amp.y, v.y);
            } else {
              asm volatile("" : "+r"(u0), "+r"(u1));  // (stays in this branch)
              v.x += double(u0) * 0x1p-32 * amp.x;
              if (!is_zero(amp.y)) v.y = fma_rare(double(u1) * 0x1p-32, amp.y, v.y);
            }
          }
        }
        if (a.real_out[m]) { a.real_out[m][2 * i] = v.x; a.real_out[m][2 * i + 1] = v.y; }
        if (!dst) continue;
        if (m == 1) {  // rsl
          if (a.lattice == 0) v = make_double2(v.y - half_gamma, -v.x);  // -i omega - gamma/2
          else v = make_double2(-v.y - half_gamma, -(a.detuning - v.x));  // -i (detuning - E) - gamma/2
        } else {       // i U, i F
          v = make_double2(-v.y, v.x);
        }
        store_c<PREC>(dst, i, v);
      }
    }
  }
}

// Wiener increments of one trajectory exactly as the step kernels draw them
// in Philox mode: out[(step - step0) * n + p] (interleaved complex, widened
// to FP64 for an FP32 run), site p taking words (0,1) or (2,3) of call
// site_ctr(p).
__global__ void wiener_kernel(int prec, uint32_t seed, uint32_t id, uint32_t step0, int64_t nsteps, int64_t n,
                              double* out) {
  const int64_t total = nsteps * n;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < total; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t k = i / n, p = i % n;
    int hi;
    const uint32_t c0 = site_ctr(p, n, &hi);
    const u32x4 w = wiener_words(c0, step0 + uint32_t(k), seed, id);
    const uint32_t u0 = hi ? w.z : w.x, u1 = hi ? w.w : w.y;
    double2 z;
    if (prec == 0) {
      const float2 f = normal_pair(u0, u1, 0.0f);
      z = make_double2(double(f.x), double(f.y));
    } else {
      z = normal_pair(u0, u1, 0.0);
    }
    out[2 * i] = z.x;
    out[2 * i + 1] = z.y;
  }
}

__global__ void philox_kernel(const uint32_t* ctr, size_t n, uint32_t k0, uint32_t k1, uint32_t* out) {
  const size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const u32x4 r = philox4x32_10(u32x4{ctr[4 * i], ctr[4 * i + 1], ctr[4 * i + 2], ctr[4 * i + 3]}, k0, k1);
  out[4 * i] = r.x; out[4 * i + 1] = r.y; out[4 * i + 2] = r.z; out[4 * i + 3] = r.w;
}

// 8 independent FMA chains per thread; 2 flops per FMA.
__global__ void fma_kernel(float* out, int iters, float a, float b) {
  float x[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] = float(threadIdx.x + k);
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = fmaf(x[k], a, b);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += x[k];
  if (s == 1.2345f) out[0] = s;  // keeps the chains alive
}

bool check(cudaError_t e, std::string* err, const char* what) {
  if (e == cudaSuccess) return true;
  if (err) *err = std::string(what) + ": " + cudaGetErrorString(e);
  return false;
}

// FP32 -> FP64 widening of a field (complex64 -> complex128 as 2n reals),
// so that downloads copy the caller's type directly.
__global__ void widen_kernel(const float* __restrict__ in, double* __restrict__ out, int64_t n) {
  for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < n; k += int64_t(gridDim.x) * blockDim.x)
    out[k] = double(in[k]);
}

// One frame of a batch (n = trajectories x reals per trajectory values) into
// its place among a trajectory's frames, as doubles: row r of the batch at
// out + r * stride.
template <typename R>
__global__ void place_kernel(const R* __restrict__ in, double* __restrict__ out, int64_t n, int64_t row, int64_t stride) {
  for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < n; k += int64_t(gridDim.x) * blockDim.x)
    out[(k / row) * stride + k % row] = double(in[k]);
}

}  // namespace

bool init_launch(const InitArgs& a, cudaStream_t s, std::string* err) {
  const int64_t total = a.ntraj * ((a.nsites + 1) / 2);
  if (total <= 0) return true;
  const int64_t blocks = std::min<int64_t>((total + 255) / 256, 152 * 32);
  if (a.prec == 0) init_kernel<0><<<int(blocks), 256, 0, s>>>(a);
  else init_kernel<1><<<int(blocks), 256, 0, s>>>(a);
  return check(cudaGetLastError(), err, "init_kernel");
}

bool moments_launch(const MomentArgs& a, cudaStream_t s, std::string* err) {
  dim3 grid(unsigned((a.nsites + 127) / 128), unsigned(a.nblocks));
  if (a.prec == 0) moments_kernel<float><<<grid, 128, 0, s>>>(a);
  else moments_kernel<double><<<grid, 128, 0, s>>>(a);
  return check(cudaGetLastError(), err, "moments_kernel");
}

bool fp32_peak(double* tflops, std::string* err) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  float* out = nullptr;
  if (!check(cudaMalloc(&out, sizeof(float)), err, "fp32 peak alloc")) return false;
  const int threads = 512, blocks = sms * 4, iters = 1 << 16;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  double best = 0.0;
  for (int rep = 0; rep < 6; ++rep) {
    cudaEventRecord(e0);
    fma_kernel<<<blocks, threads>>>(out, iters, 0.999999f, 1e-7f);
    cudaEventRecord(e1);
    if (!check(cudaEventSynchronize(e1), err, "fp32 peak")) break;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    const double flops = 2.0 * 8.0 * double(iters) * double(threads) * double(blocks);
    if (rep > 0 && ms > 0) best = std::max(best, flops / (double(ms) * 1e-3) / 1e12);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  *tflops = best;
  return best > 0.0;
}

bool wiener_launch(int prec, uint32_t seed, uint32_t id, uint32_t step0, int64_t nsteps, int64_t n, double* d_out,
                   cudaStream_t s, std::string* err) {
  const int64_t total = nsteps * n;
  if (total <= 0) return true;
  const int grid = int(std::min<int64_t>((total + 255) / 256, 4096));
  wiener_kernel<<<grid, 256, 0, s>>>(prec, seed, id, step0, nsteps, n, d_out);
  return check(cudaGetLastError(), err, "wiener_kernel");
}

bool philox_launch(const uint32_t* d_ctr, size_t n, uint32_t k0, uint32_t k1, uint32_t* d_out, cudaStream_t s,
                   std::string* err) {
  if (n == 0) return true;
  philox_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(d_ctr, n, k0, k1, d_out);
  return check(cudaGetLastError(), err, "philox_kernel");
}

bool widen_launch(const void* in, double* out, int64_t n, cudaStream_t s, std::string* err) {
  if (n <= 0) return true;
  const int grid = int(std::min<int64_t>((n + 255) / 256, 152 * 16));
  widen_kernel<<<grid, 256, 0, s>>>(static_cast<const float*>(in), out, n);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { if (err) *err = std::string("widen: ") + cudaGetErrorString(e); return false; }
  return true;
}

bool place_launch(int prec, const void* in, double* out, int64_t rows, int64_t row, int64_t stride, cudaStream_t s,
                  std::string* err) {
  const int64_t n = rows * row;
  if (n <= 0) return true;
  const int grid = int(std::min<int64_t>((n + 255) / 256, 152 * 16));
  if (prec == 0) place_kernel<float><<<grid, 256, 0, s>>>(static_cast<const float*>(in), out, n, row, stride);
  else place_kernel<double><<<grid, 256, 0, s>>>(static_cast<const double*>(in), out, n, row, stride);
  return check(cudaGetLastError(), err, "place_kernel");
}

}  // namespace twmc
