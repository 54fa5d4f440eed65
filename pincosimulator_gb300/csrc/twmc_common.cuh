// twmc_common.cuh -- shared device helpers of the TWMC engine: complex
// arithmetic in FP32/FP64, Philox4x32-10 and the Box-Muller normal pairs.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>
#include <utility>

#include "bm_tables.inc"

namespace twmc {

template <typename R> struct C2;
template <> struct C2<float> { using type = float2; };
template <> struct C2<double> { using type = double2; };
template <typename R> using c2_t = typename C2<R>::type;

template <typename T> __device__ __forceinline__ T cmake(decltype(T::x) x, decltype(T::x) y) { T r; r.x = x; r.y = y; return r; }
template <typename T> __device__ __forceinline__ T cadd(T a, T b) { return cmake<T>(a.x + b.x, a.y + b.y); }
template <typename T> __device__ __forceinline__ T csub(T a, T b) { return cmake<T>(a.x - b.x, a.y - b.y); }
// FP32 complex add/sub as one packed FP32x2 instruction (sm_100+); same
// round-to-nearest results as the two scalar operations.
template <> __device__ __forceinline__ float2 cadd<float2>(float2 a, float2 b) { return __fadd2_rn(a, b); }
template <> __device__ __forceinline__ float2 csub<float2>(float2 a, float2 b) {
  return __fadd2_rn(a, make_float2(-b.x, -b.y));
}
template <typename T> __device__ __forceinline__ T cmul(T a, T b) { return cmake<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
// a * conj(b)
template <typename T> __device__ __forceinline__ T cmulc(T a, T b) { return cmake<T>(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y); }
// acc + y * conj(w) as four multiply-adds (one rounding per component step)
template <typename T> __device__ __forceinline__ T cmlac(T acc, T y, T w) {
  return cmake<T>(fma(y.x, w.x, fma(y.y, w.y, acc.x)), fma(y.y, w.x, fma(-y.x, w.y, acc.y)));
}
// 2 a - s: the difference a - u of a butterfly whose sum s = a + u is known
template <typename T> __device__ __forceinline__ T ctwice_minus(T a, T s) {
  using R = decltype(T::x);
  return cmake<T>(fma(R(2), a.x, -s.x), fma(R(2), a.y, -s.y));
}
// -i * a and +i * a
template <typename T> __device__ __forceinline__ T cmul_mi(T a) { return cmake<T>(a.y, -a.x); }
template <typename T> __device__ __forceinline__ T cmul_pi(T a) { return cmake<T>(-a.y, a.x); }

// Shared-memory access through 32-bit shared-window addresses (the
// real-space kernels compute their neighbour indices at run time; keeping the
// address arithmetic in 32 bits avoids 64-bit integer work per access).
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ float2 lds_c(uint32_t a, float2) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double2 lds_c(uint32_t a, double2) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  return v;
}
// Four consecutive reals from shared memory (16-byte aligned for FP32).
__device__ __forceinline__ void lds_r4(uint32_t a, float* w) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void lds_r4(uint32_t a, double* w) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(w[0]), "=d"(w[1]) : "r"(a) : "memory");
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(w[2]), "=d"(w[3]) : "r"(a + 16u) : "memory");
}
__device__ __forceinline__ void sts_c(uint32_t a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sts_c(uint32_t a, double2 v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
// The same address in the shared memory of cluster CTA `rank`, and a load
// through it (distributed shared memory).
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ float2 ldc_c(uint32_t a, float2) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}

// Compile-time loop: f(std::integral_constant<int, I>) for I = 0..N-1.
template <class F, int... Is>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, Is...>) {
  (f(std::integral_constant<int, Is>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl(f, std::make_integer_sequence<int, N>{});
}

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC'11): 10 rounds of two 32x32->64-bit
// multiplies with Weyl-sequence key bumps. Counter (c0,c1,c2,c3), key (k0,k1).
// ---------------------------------------------------------------------------
struct u32x4 { uint32_t x, y, z, w; };

template <int ROUNDS>
__host__ __device__ __forceinline__ u32x4 philox4x32(u32x4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
#ifdef __CUDA_ARCH__
    const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
    const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
#else
    const uint64_t p0 = uint64_t(0xD2511F53u) * c.x, p1 = uint64_t(0xCD9E8D57u) * c.z;
    const uint32_t lo0 = uint32_t(p0), hi0 = uint32_t(p0 >> 32);
    const uint32_t lo1 = uint32_t(p1), hi1 = uint32_t(p1 >> 32);
#endif
    c = u32x4{hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0};
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c;
}

__host__ __device__ __forceinline__ u32x4 philox4x32_10(u32x4 c, uint32_t k0, uint32_t k1) {
  return philox4x32<10>(c, k0, k1);
}

// Noise streams (counter word 2).
enum : uint32_t { kStreamWiener = 0, kStreamInit = 1, kStreamU = 2, kStreamOmega = 3, kStreamF = 4 };

// Wiener increments use a fixed key, kWienerKey0/1 (hex digits of pi), and
// carry the trajectory in the counter: (site pair, step, id, seed). The key
// schedule is then a compile-time constant that folds into the round's
// XORs instead of two adds per round on per-thread keys. The other streams
// keep the key (seed, id) and the counter (site pair, 0, stream, 0); with
// these constants the two families cannot share an input block.
constexpr uint32_t kWienerKey0 = 0x243F6A88u, kWienerKey1 = 0x85A308D3u;

__host__ __device__ __forceinline__ u32x4 wiener_words(uint32_t pair, uint32_t step, uint32_t seed, uint32_t id) {
  return philox4x32_10(u32x4{pair, step, id, seed}, kWienerKey0, kWienerKey1);
}

// The Wiener words of one site pair over many steps. Of the ten rounds' twenty
// 32 x 32 -> 64-bit products (10 of the packed steps' 21.7 instructions on the
// FMA pipe's wide half, per site) the first three rounds hold four
// that do not depend on the step and one that all pairs of a trajectory share:
// a thread keeps what they give per pair (WienerSite) and forms the shared one
// once per step (WienerStep). The compiler moves these products out of the step
// loop by itself too (the instruction count is the same), but holds more than
// these four registers per pair: 122 registers instead of 128 at 2 x 2 slots,
// a quarter fewer loads on clusters of four (spills). The same words as
// wiener_words.
struct WienerSite { uint32_t a, b, c, d; };
struct WienerStep { uint32_t hi, lo; };
constexpr uint32_t kPhiloxM0 = 0xD2511F53u, kPhiloxM1 = 0xCD9E8D57u, kPhiloxW0 = 0x9E3779B9u, kPhiloxW1 = 0xBB67AE85u;
__device__ __forceinline__ WienerSite wiener_site(uint32_t pair, uint32_t seed, uint32_t id) {
  const uint32_t y = __umulhi(kPhiloxM0, pair) ^ seed ^ kWienerKey1;
  const uint32_t s0 = __umulhi(kPhiloxM1, y) ^ (kPhiloxM1 * id) ^ (kWienerKey0 + kPhiloxW0);
  return WienerSite{(kPhiloxM0 * pair) ^ (kWienerKey1 + kPhiloxW1), (kPhiloxM1 * y) ^ (kWienerKey0 + 2u * kPhiloxW0),
                    __umulhi(kPhiloxM0, s0) ^ (kWienerKey1 + 2u * kPhiloxW1), kPhiloxM0 * s0};
}
__device__ __forceinline__ WienerStep wiener_step(uint32_t step, uint32_t id) {
  const uint32_t x = __umulhi(kPhiloxM1, id) ^ step ^ kWienerKey0;
  return WienerStep{__umulhi(kPhiloxM0, x), kPhiloxM0 * x};
}
__device__ __forceinline__ u32x4 wiener_words(WienerSite p, WienerStep t) {
  const uint32_t s2 = t.hi ^ p.a;
  const u32x4 c{__umulhi(kPhiloxM1, s2) ^ p.b, kPhiloxM1 * s2, p.c ^ t.lo, p.d};
  return philox4x32<7>(c, kWienerKey0 + 3u * kPhiloxW0, kWienerKey1 + 3u * kPhiloxW1);
}

// Box-Muller, FP32, scaled by s: s (r cos th, r sin th) with r = sqrt(-2 ln u1),
// u1 = fma(float(a), 2^-32, 2^-33) in (0, 1], th = 2 pi u2 - pi, u2 the same
// map of b. The radius is computed as sqrt(kn log2 u1) with kn = -2 ln(2) s^2
// (hardware log2 and square root), so a scale costs nothing; th is one FMA
// of float(b).
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kNegTwoLn2 = -1.38629436111989061883f;  // -2 ln 2: kn of the unscaled normals
__device__ __forceinline__ float2 scaled_normal_pair(uint32_t a, uint32_t b, float kn) {
  const float u1 = __fmaf_rn(__uint2float_rn(a), 0x1p-32f, 0x1p-33f);
  // 2 pi (float(b) 2^-32 + 2^-33) - pi
  const float th = __fmaf_rn(__uint2float_rn(b), 1.46291807926715968e-9f, -3.14159265285833420f);
  const float r = sqrt_approx(fmaxf(kn * lg2_approx(u1), 0.0f));
  float sn, cs;
  __sincosf(th, &sn, &cs);
  return make_float2(r * cs, r * sn);
}
__device__ __forceinline__ float2 normal_pair(uint32_t a, uint32_t b, float) {
  return scaled_normal_pair(a, b, kNegTwoLn2);
}

// float -> double and back (round to nearest even) by integer operations, the
// conversion instructions for subnormals, infinities and NaN only: those run
// on the FP64 pipe, two lanes per SM and cycle on GB300 (in functions of their
// own: the compiler would predicate them, and predicated instructions still
// take their turn on that pipe).
static __device__ __noinline__ double widen_rare(float x) { return double(x); }
static __device__ __noinline__ float narrow_rare(double x) { return float(x); }
static __device__ __noinline__ double fma_rare(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ double widen(float x) {
  const uint32_t b = __float_as_uint(x), e = b & 0x7f800000u;
  if (e == 0u || e == 0x7f800000u) return widen_rare(x);
  return __hiloint2double(int((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), int(b << 29));
}
__device__ __forceinline__ float narrow(double x) {
  const uint32_t hi = uint32_t(__double2hiint(x)), lo = uint32_t(__double2loint(x));
  const uint32_t e = (hi >> 20) & 0x7ffu;
  if (e - 897u > 252u) return narrow_rare(x);  // outside 2^-126 <= |x| < 2^127
  const uint32_t m = ((e - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29), rest = lo & 0x1fffffffu;
  const uint32_t up = rest > 0x10000000u || (rest == 0x10000000u && (m & 1u)) ? 1u : 0u;
  return __uint_as_float((hi & 0x80000000u) | (m + up));
}

// Whether x is +0 or -0, without a comparison on the FP64 pipe.
__device__ __forceinline__ bool is_zero(double x) { return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0; }

// Box-Muller, FP64: u = (w + 1/2) 2^-32, r = sqrt(-2 ln u1), th = 2 pi u2 - pi.
// The logarithm's reduction (the bit pattern less that of 0.6875, seven bits of
// it for the interval, an arithmetic shift for the exponent, one interval that
// ends at 1) is the one of log in Arm Optimized Routines (math/log.c, MIT);
// tables, polynomial and the rest are this file's and bm_tables.py's.
// The FP64 pipe of GB300 (two lanes per SM and cycle) bounds FP64 runs, and
// the general log, sincos and sqrt of a draw were about 70 of its 185
// instructions per site-update. Here 33: the words' structure makes both
// argument reductions exact integer work, tables (bm_tables.py) replace most
// of the polynomials, and the square root refines the FP32 reciprocal root:
// 500 trajectories of 16x16 over 100 steps take 3.07 ms, before 4.30 ms
// in all. Errors of the draws against 60 digits over 8192 pairs
// (tests/test_gpu_normals64.py): rms 0.95e-16, at most 7.7e-16 (with log, sincos
// and sqrt 1.41e-16 and 1.09e-15).
__device__ __forceinline__ double neg2_log_uniform(uint32_t w) {
  // 2 w + 1 as a double, by its leading bit
  const int lz = w ? __clz(int(w)) : 32;  // 33 - lz significant bits
  const uint64_t x = (uint64_t(w) << 1) | 1u;
  const uint64_t bits = (uint64_t(1023 + 32 - lz) << 52) + ((x << (20 + lz)) & 0xfffffffffffffull);
  const uint32_t tmp = uint32_t(bits >> 32) - 0x3fe60000u;  // from 0.6875
  const uint32_t i = (tmp >> 13) & 127u;
  const int k = int(tmp) >> 20;
  const double z = __longlong_as_double((long long)(bits - (uint64_t(uint32_t(k)) << 52)));
  const double2 t = kLogTable[i];
  const double s = fma(z, t.x, 2.0);
  double q = fma(s, 1.0 / 448.0, 1.0 / 192.0);
  q = fma(q, s, 1.0 / 80.0);
  q = fma(q, s, 1.0 / 32.0);
  q = fma(q, s, 1.0 / 12.0);
  q = fma(q, s, 0.25);
  return (kExpTable[k] + t.y) + fma(s * s, q, s);
}
__device__ __forceinline__ double2 normal_pair(uint32_t a, uint32_t b, double) {
  const double l = neg2_log_uniform(a);
  // sqrt(l), 2.3e-10 <= l <= 45.7: from y = l^-1/2 (1 + 2^-23) one coupled
  // Newton step for g = sqrt(l) and h = l^-1/2 / 2 (Markstein 1990), then a
  // correction of g by its residual
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(narrow(l)));
  const double yd = widen(y), h0 = widen(0.5f * y);
  double g = l * yd;
  const double e = fma(-g, h0, 0.5);
  const double h = fma(h0, e, h0);
  g = fma(g, e, g);
  const double r = fma(fma(-g, g, l), h, g);
  // the angle from the centre of its sector: (2 m + 1 - 2^24) pi 2^-32
  const double n = __hiloint2double(0x43300000, int(2u * (b & 0xffffffu) + 1u)) - 4503599644147712.0;  // 2^52 + 2^24
  const double d = n * 7.31459039633579843e-10, d2 = d * d;
  const double sd = fma(d2 * d, fma(d2, 1.0 / 120.0, -1.0 / 6.0), d);
  const double c1 = d2 * fma(d2, fma(d2, -1.0 / 720.0, 1.0 / 24.0), -0.5);
  const double2 t = kSectorTable[b >> 24];
  const double c = t.x + fma(-t.y, sd, t.x * c1), sn = t.y + fma(t.x, sd, t.y * c1);
  return make_double2(r * c, r * sn);
}

// Site pairing on Philox calls: half = ceil(n/2); site p < half uses words
// (0,1) of call p, site p >= half words (2,3) of call p - half.
__host__ __device__ __forceinline__ uint32_t site_ctr(int64_t p, int64_t n, int* hi) {
  const int64_t half = (n + 1) / 2;
  *hi = p >= half;
  return uint32_t(p >= half ? p - half : p);
}

}  // namespace twmc
