// FP64 values as fixed-point integers and back, and rounding to digits, for the
// digit planes of the tensor-core kernels.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

namespace hfg {
namespace {

// x 2^(bits - E) towards zero, two's complement, |x| < 2^E: by shifts of the
// significand (no FP64-pipe instructions); exponents far below E give 0
template <int BITS>
__device__ __forceinline__ uint64_t fixed_point(double x, int E) {
  const int h = __double2hiint(x);
  const int sh = min(max(E + 1083 - BITS - ((h >> 20) & 0x7FF), 0), 63);  // from a 61-bit significand
  const uint64_t m =
      ((((uint64_t)(uint32_t)((h & 0xFFFFF) | 0x100000)) << 32 | (uint32_t)__double2loint(x)) << 8) >> sh;
  const uint64_t sg = (uint64_t)(int64_t)(h >> 31);
  return (m ^ sg) - sg;
}

__device__ __forceinline__ double exp2d(int k) {  // 2^k, k clamped to the normal range
  return __hiloint2double((min(max(k, -1022), 1023) + 1023) << 20, 0);
}
// an integer below 2^51 in FP64
__device__ __forceinline__ double i2d(int64_t i) {
  return __longlong_as_double(0x4338000000000000ll + i) - 6755399441055744.0;
}

// float -> double times 2^k through the bit pattern (no FP64-pipe
// instructions); c = (896 + k) << 20, zero and subnormal floats give zero
__device__ __forceinline__ double f2d_scaled(float f, int c) {
  const uint32_t bits = __float_as_uint(f), t = bits & 0x7FFFFFFFu;
  const uint32_t hi = t < 0x00800000u ? 0u : ((t >> 3) + (uint32_t)c) | (bits & 0x80000000u);
  return __hiloint2double((int)hi, t < 0x00800000u ? 0 : (int)(bits << 29));
}

constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: x + M - M rounds |x| < 2^22 to an integer

__device__ __forceinline__ float rnd(float x) { return __fsub_rn(__fadd_rn(x, kMagic), kMagic); }
// rint(x * s) with one rounding of the product
__device__ __forceinline__ float rnd_mul(float x, float s) { return __fsub_rn(__fmaf_rn(x, s, kMagic), kMagic); }
__device__ __forceinline__ float exp2i(int k) {  // 2^k, k clamped to the normal range
  k = k < -126 ? -126 : (k > 127 ? 127 : k);
  return __int_as_float((k + 127) << 23);
}

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

constexpr int kBadExp = 1 << 20;  // exponent of a tile with a value that is not finite

}  // namespace
}  // namespace hfg
