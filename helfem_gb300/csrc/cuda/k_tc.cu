// Split-precision exchange on the tensor cores: the element-pair tiles of
// TwoDBasisT::exchange (src/atomic/TwoDBasis.cpp:879-999) with the FE
// assembly of assemble_K_FE_one_multipole_cached_chol
// (libhelfemqc/include/CoulombExchangeFE.h:484-530).
//
//   off-diagonal pairs a != b:  K_jk(a,b) -= sum_L A_L(a) X_jkL(a,b) B_L(b)^T,
//                               A/B = r_small/r_big by element order;
//   diagonal elements:          K_jk(a,a) -= sum_L Tk_L(a) vec X_jkL(a,a),
//                               Tk the exchange-ordered in-element tensor
//                               (the reference's sum_p M_p X M_p^T).
// X is the recoupled density tile.
//
// Arithmetic (an Ozaki-style slicing with exact integer sums):
//  * every operand is a fixed-point number below 1 written as balanced
//    digits, x = sum_k d_k b^-(k+1): integers, exact in the 16-bit operand
//    type. Element pairs: base 1024 (|d_0| <= 1024, the others <= 512) in f16,
//    six digits of the tables and of the intermediate, five of a density tile
//    (50 bits: a float pair has 48). Diagonal elements: base 256 (|d_0| <= 256,
//    |d_k| <= 128) in bf16, seven and six;
//  * the radial tables are digitised once per atom: a power of two per table
//    (L, element) brings its largest entry near 1, then one power of two per
//    row, shared by all multipoles, its absolute row sums to at most 1; Tk one
//    power of two per row;
//  * a recoupled density tile X_L (float pairs on the CUDA cores) of an element
//    pair is scaled by 2^(s_L - E), s_L the exponents of the pair's two tables
//    of multipole L and E one exponent per output block, from the largest
//    entries of the density tiles (taken in the norm pass): with tables of all
//    multipoles near 1 and one scale for all X_L of a block, the products of
//    all multipoles add up in tensor memory;
//  * the tensor core forms the digit products level by level,
//    acc_d = sum_{k+l=d} sum_p a_k b_l, in FP32 in tensor memory. The element
//    pairs' sums run over 16 terms and up to 8 multipoles: leading digits obey
//    the unit row sums and the others are spread over +-512, so that a level's
//    spread stays below 2^21, far from the 2^24 where FP32 sums of integers
//    would round;
//  * the levels of the first product (Y = A X, 128 rows = 8 output blocks x 16)
//    are carried into balanced digits on the CUDA cores and become the operand
//    of the second, which accumulates over the multipoles; its levels are
//    turned into a float pair, scaled, and converted to FP64 once per output
//    element and group.
// Truncation (48-bit density tiles, the levels dropped) leaves ~1e-14 of
// max|K| against the FP64 result. A row scale shared by the multipoles without
// the per-table power of two lost log2(1/r) L bits near the nucleus.
//
//
// FP64 form (F64): the same products from the FP64 density itself. The tiles
// are recoupled with FP64 FMAs (a thirteenth of the FP64 contraction's) and cut
// into fixed point by shifts of their significands, one digit more (58 bits
// below the tile's bound, 56 in the diagonal elements); the sums, integers,
// become FP64 numbers through exact integers. The contraction's own rounding is
// then below that of the FP64 sums it replaces: the error against the exact K
// is the tables' in both (4.120e-14 for Kr, l <= 3 dense 2.680e-14 and
// 2.679e-14), at 1.00 instead of 4.52 ms for Kr. A tile with a value that is
// not finite gives NaN throughout, as a product with FP64 NaNs does.
//
// Off-diagonal work unit = one element pair (a,b) and a range of groups of
// 8 active output angular blocks (listed by the density pass); per group and
// multipole L the group's entries with that L form one batch of M = 128 rows.
// For density digit kx the table planes kt = 0..5-kx are consecutive in shared
// memory and form one operand of N = 16 (6 - kx) rows whose block kt lands on
// the tensor-memory columns of level kx + kt, so a batch is 5 + 6 MMAs. The
// CUDA-core work on the digits is the bound (370 M warp instructions for the Kr
// basis at 58 % of the issue slots; the tensor pipe is some 6 % busy), so what
// matters is few instructions, warps that rarely wait and a loop that fits the
// instruction cache: one copy of every phase, nothing unrolled that need not
// be. Element pairs of the Kr basis (l <= 2, 40 elements): warps in step with
// their MMAs and the multipoles read back one by one 0.87 ms; multipoles summed
// in tensor memory, base 1024 0.79 ms; one arrival count instead of a warp that
// issues 0.68 ms; terms streamed through one register buffer by compact loops
// 0.57 ms.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <type_traits>

#include "devatom.cuh"
#include "smem_limit.hpp"
#include "ff.cuh"
#include "fixed.cuh"
#include "tc.cuh"

namespace hfg {
namespace {

constexpr int PD = TC_NDIGITS;  // element pairs: digits of the tables and the intermediate, levels
constexpr int PX = 5;           // digits of a density tile
constexpr int ND = 7;           // diagonal elements: digits of Tk, levels
constexpr int NDX = 6;          // digits of a density tile (48 bits)
constexpr int APLANE = 4096;    // bytes of one 128 x 16 bf16 operand plane
constexpr int TPLANE = 512;     // bytes of one 16 x 16 bf16 table plane

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// all 7 levels (16 columns apart) of 8 consecutive columns, one wait
__device__ __forceinline__ void tmem_ld_levels(uint32_t taddr, float (&v)[ND][8]) {
  static_assert(ND == 7, "level count of the load below");
  uint32_t r[56];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%56];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%57];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%58];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24,%25,%26,%27,%28,%29,%30,%31}, [%59];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%32,%33,%34,%35,%36,%37,%38,%39}, [%60];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%40,%41,%42,%43,%44,%45,%46,%47}, [%61];\n"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%48,%49,%50,%51,%52,%53,%54,%55}, [%62];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
        "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55])
      : "r"(taddr), "r"(taddr + 16), "r"(taddr + 32), "r"(taddr + 48), "r"(taddr + 64), "r"(taddr + 80),
        "r"(taddr + 96)
      : "memory");
#pragma unroll
  for (int d = 0; d < ND; ++d)
#pragma unroll
    for (int j = 0; j < 8; ++j) v[d][j] = __uint_as_float(r[8 * d + j]);
}

// carry the level sums (weights 256^-(d+2)) into balanced digits
// y_0..y_{ND-1} (weights 256^-(k+1)); the remainder of the last level is
// rounded into its neighbour and dropped
__device__ __forceinline__ void carry(float (&acc)[ND], float (&y)[ND]) {
#pragma unroll
  for (int d = ND - 1; d >= 1; --d) {
    const float c = rnd_mul(acc[d], 1.0f / 256.0f);
    acc[d] = __fmaf_rn(c, -256.0f, acc[d]);
    acc[d - 1] = __fadd_rn(acc[d - 1], c);
  }
  const float c0 = rnd_mul(acc[0], 1.0f / 256.0f);
  y[0] = c0;
  y[1] = __fmaf_rn(c0, -256.0f, acc[0]);
#pragma unroll
  for (int k = 2; k < ND; ++k) y[k] = acc[k - 1];
}

// the value of level sums as a float pair scaled by sc: carried into digits,
// an exact head and a rounded tail
__device__ __forceinline__ ffv levels_to_pair(float (&lv)[ND], float sc) {
  float z[ND];
  carry(lv, z);
  const float h = __fmaf_rn(z[1], 1.0f / 65536.0f, __fmul_rn(z[0], 1.0f / 256.0f));
  const float m2 = __fmul_rn(z[2], 1.0f / 16777216.0f);
  const float sh = __fadd_rn(h, m2);
  const float bb = __fsub_rn(sh, h);
  const float e = __fadd_rn(__fsub_rn(h, __fsub_rn(sh, bb)), __fsub_rn(m2, bb));
  float tail = 0.f;
#pragma unroll
  for (int k = ND - 1; k >= 3; --k) tail = __fmaf_rn(tail, 1.0f / 256.0f, z[k]);
  tail = __fmul_rn(tail, 1.0f / 4294967296.0f);  // z_3 weight 2^-32
  return {__fmul_rn(sh, sc), __fmul_rn(__fadd_rn(e, tail), sc)};
}

// the 6 balanced digits of 8 float-pair values against |X| < 2^E, packed in
// bf16 pairs: pk[k][j/2] holds elements j, j+1 of digit plane k
__device__ __forceinline__ void digits_of(const ffv (&x)[8], int E, uint32_t (&pk)[NDX][4]) {
  const float s = exp2i(24 - E);
#pragma unroll
  for (int jj = 0; jj < 8; jj += 2) {
    float dg[NDX][2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const int j = jj + w;
      const float h = __fmul_rn(x[j].hi, s);
      const float d0 = rnd_mul(h, 1.0f / 65536.0f);
      const float t1 = __fmaf_rn(d0, -65536.0f, h);
      const float d1 = rnd_mul(t1, 1.0f / 256.0f);
      const float t2 = __fmaf_rn(d1, -256.0f, t1);
      const float d2 = rnd(t2);
      float r = __fmaf_rn(x[j].lo, s, __fsub_rn(t2, d2));
      const float d3 = rnd_mul(r, 256.0f);
      r = __fmaf_rn(r, 256.0f, -d3);
      const float d4 = rnd_mul(r, 256.0f);
      r = __fmaf_rn(r, 256.0f, -d4);
      dg[0][w] = d0;
      dg[1][w] = d1;
      dg[2][w] = d2;
      dg[3][w] = d3;
      dg[4][w] = d4;
      dg[5][w] = rnd_mul(r, 256.0f);
    }
#pragma unroll
    for (int k = 0; k < NDX; ++k) pk[k][jj / 2] = pack_bf16(dg[k][0], dg[k][1]);
  }
}

// tile exponent from the biased float exponent of the largest high word:
// |X| < 2^E; tiles below 2^-100 keep fewer digits (their contribution is
// negligible)
__device__ __forceinline__ int tile_exponent(unsigned eb) { return max((int)max(eb, 1u) - 126, -100); }

// exact float -> double through the bit pattern (no FP64-pipe conversion);
// zero and subnormal floats map to zero, infinities and NaN to themselves
__device__ __forceinline__ double f2d_bits(float f) {
  const uint32_t bits = __float_as_uint(f);
  const uint32_t e = (bits >> 23) & 0xFFu;
  if (e == 0) return 0.0;
  const uint32_t e64 = e == 0xFFu ? 0x7FFu : e + 896u;
  const unsigned long long r = ((unsigned long long)(bits >> 31) << 63) | ((unsigned long long)e64 << 52) |
                               ((unsigned long long)(bits & 0x7FFFFFu) << 29);
  return __longlong_as_double((long long)r);
}
__device__ __forceinline__ double pair_to_d(ffv a) {
  const ffv n = ff_norm(a.hi, a.lo);
  return f2d_bits(n.hi) + f2d_bits(n.lo);
}

// ---- element pairs: base 1024 in f16 ----

// all six levels (16 columns apart) of 8 consecutive columns, one wait
__device__ __forceinline__ void tmem_ld_pairs(uint32_t taddr, float (&v)[PD][4]) {
  static_assert(PD == 6, "level count of the load below");
  uint32_t r[24];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%24];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%25];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%26];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12,%13,%14,%15}, [%27];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%16,%17,%18,%19}, [%28];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20,%21,%22,%23}, [%29];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23])
      : "r"(taddr), "r"(taddr + 16), "r"(taddr + 32), "r"(taddr + 48), "r"(taddr + 64), "r"(taddr + 80)
      : "memory");
#pragma unroll
  for (int d = 0; d < PD; ++d)
#pragma unroll
    for (int j = 0; j < 4; ++j) v[d][j] = __uint_as_float(r[4 * d + j]);
}

// carry the level sums (weights 1024^-(d+2)) so that every level but the
// first is a balanced digit; y0, y1 the first level's two digits
__device__ __forceinline__ void carry_pairs(float (&a)[PD], float& y0, float& y1) {
#pragma unroll
  for (int d = PD - 1; d >= 1; --d) {
    const float c = rnd_mul(a[d], 1.0f / 1024.0f);
    a[d] = __fmaf_rn(c, -1024.0f, a[d]);
    a[d - 1] = __fadd_rn(a[d - 1], c);
  }
  y0 = rnd_mul(a[0], 1.0f / 1024.0f);
  y1 = __fmaf_rn(y0, -1024.0f, a[0]);
}

// the value of the level sums (integers below 2^24, weights 1024^-(d+2)) times
// 2^k, c as above: the leading three with their rounding errors, the rest as
// they come
__device__ __forceinline__ double levels_to_d(const float (&a)[PD], int c) {
  auto two_sum = [](float x, float y, float& e) {
    const float s = __fadd_rn(x, y), bb = __fsub_rn(s, x);
    e = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bb)), __fsub_rn(y, bb));
    return s;
  };
  float e1, e2;
  const float s1 = two_sum(__fmul_rn(a[0], 1.0f / 1048576.0f), __fmul_rn(a[1], 1.0f / 1073741824.0f), e1);
  const float s2 = two_sum(s1, __fmul_rn(a[2], 1.0f / 1099511627776.0f), e2);
  float tail = __fmaf_rn(a[5], 1.0f / 1024.0f, a[4]);
  tail = __fmaf_rn(tail, 1.0f / 1024.0f, a[3]);
  tail = __fmaf_rn(tail, 8.8817841970012523e-16f, __fadd_rn(e1, e2));  // weight 2^-50
  return f2d_scaled(s2, c) + f2d_scaled(tail, c);
}

// the 5 balanced base-1024 digits of 8 float pairs scaled by 2^-30 s to below
// 1, packed in f16 pairs: pk[k][j/2] holds elements j, j+1 of digit plane k.
// The high word (24 bits) ends inside the third digit for the tile's largest
// entries, where the low word joins it exactly.
__device__ __forceinline__ void digits_pairs(const ffv (&x)[8], float s, uint32_t (&pk)[PX][4]) {
#pragma unroll
  for (int jj = 0; jj < 8; jj += 2) {
    float dg[PX][2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const float h = __fmul_rn(x[jj + w].hi, s), l = __fmul_rn(x[jj + w].lo, s);
      const float d0 = rnd_mul(h, 1.0f / 1048576.0f);
      const float t1 = __fmaf_rn(d0, -1048576.0f, h);
      const float d1 = rnd_mul(t1, 1.0f / 1024.0f);
      const float t2 = __fmaf_rn(d1, -1024.0f, t1);
      const float d2 = rnd(__fadd_rn(t2, l));
      float r = __fadd_rn(__fsub_rn(t2, d2), l);
      const float d3 = rnd_mul(r, 1024.0f);
      r = __fmaf_rn(r, 1024.0f, -d3);
      dg[0][w] = d0;
      dg[1][w] = d1;
      dg[2][w] = d2;
      dg[3][w] = d3;
      dg[4][w] = rnd_mul(r, 1024.0f);
    }
#pragma unroll
    for (int k = 0; k < PX; ++k) pk[k][jj / 2] = pack_f16(dg[k][0], dg[k][1]);
  }
}

// ---- FP64 density tiles ----

// the 6 balanced base-1024 digits of 8 values against |X| < 2^(E + 2), packed
// as in digits_pairs: with 512 added to every digit the digits are the 10-bit
// fields of the fixed-point number, and 1024 + field an f16 bit pattern
__device__ __forceinline__ void digits_fixed(const double (&x)[8], int E, uint32_t (&pk)[PD][4]) {
  static_assert(PD == 6, "two words of three fields");
#pragma unroll
  for (int jj = 0; jj < 8; jj += 2) {
    uint32_t hi[2], lo[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const uint64_t f = fixed_point<58>(x[jj + w], E) + 0x0802008020080200ull;
      lo[w] = (uint32_t)f & 0x3FFFFFFFu;
      hi[w] = (uint32_t)(f >> 30);
    }
    auto digit = [](uint32_t fields) {
      const uint32_t u = (fields & 0x03FF03FFu) | 0x64006400u;
      const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&u), __floats2half2_rn(1536.f, 1536.f));
      return *reinterpret_cast<const uint32_t*>(&d);
    };
    auto fields = [&](const uint32_t (&v)[2], int k) {
      pk[k + 2][jj / 2] = digit(__byte_perm(v[0], v[1], 0x5410));
      pk[k + 1][jj / 2] = digit(__byte_perm(v[0] << 6, v[1] << 6, 0x7632));
      pk[k][jj / 2] = digit(__byte_perm(v[0], v[1], 0x7632) >> 4);
    };
    fields(hi, 0);
    fields(lo, 3);
  }
}

// the 7 balanced base-256 digits of 8 values against |X| < 2^E, packed as in
// digits_of
__device__ __forceinline__ void digits_fixed256(const double (&x)[8], int E, uint32_t (&pk)[ND][4]) {
  static_assert(ND == 7, "a top digit and six bytes");
#pragma unroll
  for (int jj = 0; jj < 8; jj += 2) {
    float dg[ND][2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const uint64_t f = fixed_point<56>(x[jj + w], E) + 0x0000808080808080ull;
      const uint32_t hi = (uint32_t)(f >> 32), lo = (uint32_t)f;
      auto byte = [](uint32_t v, int b) {  // 2^23 + byte, as a float
        return __fsub_rn(__uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440u | b)), 8388736.f);
      };
      dg[0][w] = (float)((int)hi >> 16);
      dg[1][w] = byte(hi, 1);
      dg[2][w] = byte(hi, 0);
#pragma unroll
      for (int k = 3; k < 7; ++k) dg[k][w] = byte(lo, 6 - k);
    }
#pragma unroll
    for (int k = 0; k < ND; ++k) pk[k][jj / 2] = pack_bf16(dg[k][0], dg[k][1]);
  }
}

// level sums (integers) -> FP64 times 2^k: base 1024, weights 1024^-(d+2), and
// base 256, weights 256^-(d+2)
__device__ __forceinline__ double levels_to_f64(const float (&a)[PD], int k) {
  const int64_t u = ((int64_t)__float2int_rn(a[0]) << 20) + ((int64_t)__float2int_rn(a[1]) << 10) + __float2int_rn(a[2]);
  const int64_t v = ((int64_t)__float2int_rn(a[3]) << 20) + ((int64_t)__float2int_rn(a[4]) << 10) + __float2int_rn(a[5]);
  return fma(i2d(v), 9.313225746154785e-10, i2d(u)) * exp2d(k - 40);
}
__device__ __forceinline__ double levels_to_f64(const float (&a)[ND], int k) {
  const int64_t u = ((int64_t)__float2int_rn(a[0]) << 16) + ((int64_t)__float2int_rn(a[1]) << 8) + __float2int_rn(a[2]);
  const int64_t v = ((int64_t)__float2int_rn(a[3]) << 24) + ((int64_t)__float2int_rn(a[4]) << 16) +
                    ((int64_t)__float2int_rn(a[5]) << 8) + __float2int_rn(a[6]);
  return fma(i2d(v), 2.3283064365386963e-10, i2d(u)) * exp2d(k - 32);
}
// the 8 values y[j] of tile (a,b), block jk (-1: none), at row p and columns
// q0 + j: one pass over the columns with the block's base address computed
// once; owned entries go to K, the shared last row / column to the halo buffer
__device__ __forceinline__ void store_rows(const DevAtom& A, const DevScratch& S, double* K, int a, int b, int j,
                                           int k, int p, int q0, const double (&y)[4]) {
  const int nn = A.nn;
  const int gp = gfun(A, a, p), gq0 = gfun(A, b, q0);
  if (p >= nn || gp < 0 || gp >= A.nrad) return;
  const int lo = max(0, -gq0), hi = min(min(4, nn - q0), A.nrad - gq0);
  double* halo = S.khalo + ((size_t)(a * A.nel + b) * (A.nang * A.nang) + j + k * A.nang) * (2 * nn - 1);
  // the last row goes to the halo whole, of the others the last column
  const bool last = p == nn - 1;
  double* d = last ? halo + q0 : K + ((ptrdiff_t)k * A.nrad + gq0) * A.nbf + j * A.nrad + gp;
  const int step = last ? 1 : A.nbf, jl = last ? -1 : nn - 1 - q0;
  halo += nn + p;
#pragma unroll
  for (int jj = 0; jj < 4; ++jj, d += step)
    if (jj >= lo && jj < hi) *(jj == jl ? halo : d) = y[jj];
}

constexpr int PW = 8;                 // working warps
constexpr int PTHREADS = 32 * PW;
constexpr uint32_t kWait = TC_WAIT;  // limit of the waits of a CTA that gives up
constexpr int kNoFail = 0x7FFFFFFF;
constexpr int kGaveUp = 1 << 24;       // a warp's mark in the count of arrivals

// working warps q and q + 4 (named barriers 1-4)
__device__ __forceinline__ void pair_sync(int q) {
  if (q == 0) asm volatile("bar.sync 1, 64;" ::: "memory");
  else if (q == 1) asm volatile("bar.sync 2, 64;" ::: "memory");
  else if (q == 2) asm volatile("bar.sync 3, 64;" ::: "memory");
  else asm volatile("bar.sync 4, 64;" ::: "memory");
}

// shared-memory layout of k_tiles_tc past the operand planes
struct PairMeta {
  int alpha[16], beta[16];  // row exponents of the left and right tables
  int sL[8];                // table exponents of the pair
  // per group (four in flight), slot: exponent of the scaled density tiles,
  // multipoles present (bits), output block or -1
  int ex[4][8], mask[4][8], jk[4][8];  // jk: j | k << 16
  int fail;               // the first batch whose wait ran out, or kNoFail
  uint32_t tslot;
  int arrived;            // warps past their part of a batch, all batches (and kGaveUp)
  uint64_t done;          // a batch's second and the next one's first product
};
}  // namespace

// NaN in every result of a unit whose CTA gave up, the transposed partners' too
// (out of line and with plain arguments: inside k_tiles_tc it cost 1 % of Kr's K)
__device__ __noinline__ void mark_unit(int4 u, int end, int symmetric, int nn, int nel, int nrad, int nang, int nbf,
                                       const int* __restrict__ olist, double* khalo, double* K) {
  DevAtom A;
  A.nn = nn, A.nel = nel, A.nrad = nrad, A.nang = nang, A.nbf = nbf;
  DevScratch S;
  S.khalo = khalo;
  for (int x = 8 * u.z + (int)(threadIdx.x >> 5); x < end; x += PW) {
    const int jk = olist[x], kj = jk / nang + jk % nang * nang;
    for (int i = threadIdx.x & 31; i < nn * nn; i += 32) {
      const double bad = __longlong_as_double(0x7ff8000000000000ll);
      k_store_tile(A, S, K, u.x, u.y, jk, i % nn, i / nn, bad);
      if (symmetric) k_store_tile(A, S, K, u.y, u.x, kj, i / nn, i % nn, bad);
    }
  }
}

// Each of 8 warps, per batch: recouple and digitise slot w's density tile of
// the next batch into the other stage of the first operand, then read this
// batch's first product back (the lanes of slots 2 (w & 3) and the next one,
// half of the columns) and write its digits as the second operand; at the end
// of a group the second product into K. The last warp through issues the next
// first and this second product, which run while the warps recouple. One
// arrival count per batch is all the synchronisation between warps (a warp of
// its own that issues, with a barrier per role, cost 32 registers a thread).
template <bool F64>
__global__ void __launch_bounds__(PTHREADS, 2) k_tiles_tc(DevAtom A, DevScratch S, DevTC T,
                                                          const int4* __restrict__ units, int symmetric,
                                                          const double* __restrict__ P, double* __restrict__ K) {
  using Val = std::conditional_t<F64, double, float2>;
  constexpr int NX = F64 ? PD : PX;  // digits of a density tile
  const Val* src;
  if constexpr (F64) src = P; else src = S.p2;
  const int4 u = units[blockIdx.x];
  const int a = u.x, b = u.y;
  const int nn = A.nn, NL = A.NL, nang2 = A.nang * A.nang;
  const int count = S.ocount[0], g0 = u.z, g1 = min(u.w, (count + 7) / 8);
  if (g0 >= g1) return;  // uniform over the CTA
  extern __shared__ __align__(1024) unsigned char smraw[];
  unsigned char* A1 = smraw;                   // 2 stages x NX planes: rows (slot, q), K = p (MN-major)
  unsigned char* A2 = A1 + 2 * NX * APLANE;    // PD planes: rows (slot, i), K = q (MN-major)
  unsigned char* T1 = A2 + PD * APLANE;        // NL * PD planes of the left tables of element a
  unsigned char* T2 = T1 + NL * PD * TPLANE;   // NL * PD planes of the right tables of element b
  PairMeta& m = *reinterpret_cast<PairMeta*>(T2 + NL * PD * TPLANE);
  unsigned char* act = reinterpret_cast<unsigned char*>(&m + 1);  // [nang^2] density block above the screen
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;

  // ---- set-up once per unit: tables of this element pair, block flags ----
  const int kl = (a < b) ? 0 : 1, kr = (a < b) ? 1 : 0;  // left: r_small(a) if a < b
  {
    const int per = PD * TPLANE / 16;  // uint4 per (L, e)
    const uint4* s1 = reinterpret_cast<const uint4*>(T.digits) + (size_t)(kl * NL * A.nel) * per;
    const uint4* s2 = reinterpret_cast<const uint4*>(T.digits) + (size_t)(kr * NL * A.nel) * per;
    for (int idx = t; idx < NL * per; idx += blockDim.x) {
      const int L = idx / per, o = idx % per;
      reinterpret_cast<uint4*>(T1)[idx] = s1[((size_t)L * A.nel + a) * per + o];
      reinterpret_cast<uint4*>(T2)[idx] = s2[((size_t)L * A.nel + b) * per + o];
    }
    if (t < 16) {
      m.alpha[t] = T.rowexp[((size_t)kl * A.nel + a) * 16 + t];
      m.beta[t] = T.rowexp[((size_t)kr * A.nel + b) * 16 + t];
    }
    if (t < NL) m.sL[t] = T.texp[((size_t)kl * NL + t) * A.nel + a] + T.texp[((size_t)kr * NL + t) * A.nel + b];
    for (int idx = t; idx < nang2; idx += blockDim.x) act[idx] = S.act[idx];
    if (t == 0) {
      m.fail = kNoFail;
      m.arrived = 0;
      tc::mbar_init(&m.done, 1);
    }
  }
  if (warp == 0) {
    tc::tmem_alloc(&m.tslot, 256);
    tc::tmem_relinquish();
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tD1 = m.tslot, tD2 = m.tslot + 128;

  {
    // ---- producing: warp = slot, lane = (p, q-half), element j: column q =
    // 8 qh + j. Consecutive lanes load consecutive rows of a column (a lane
    // holding 8 rows of one column cost 32 cache lines per load, and the loads
    // bounded the kernel), and the lane's 8 columns are one 16-byte row of the
    // MN-major operand. ----
    int s_hi = m.sL[0];
    for (int L = 1; L < NL; ++L) s_hi = max(s_hi, m.sL[L]);
    const int rp = lane & 15, qh = lane >> 4;
    // Rows and columns past the tile repeat its last ones: finite digits, which
    // meet zero rows of the tables. Functions outside the basis (first and last
    // element) have table entries: their elements are zeroed.
    const int pa0 = max(gfun(A, a, 0), 0), pa1 = min(gfun(A, a, nn - 1), A.nrad - 1);
    const int qb0 = max(gfun(A, b, 0), 0), qb1 = min(gfun(A, b, nn - 1), A.nrad - 1);
    const bool edge = gfun(A, a, 0) < 0 || gfun(A, b, 0) < 0 || gfun(A, a, nn - 1) >= A.nrad || gfun(A, b, nn - 1) >= A.nrad;
    unsigned vm = 0;  // elements inside the basis
    int coff[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int gp = gfun(A, a, rp), gq = gfun(A, b, 8 * qh + j);
      if (gp >= pa0 && gp <= pa1 && gq >= qb0 && gq <= qb1) vm |= 1u << j;
      coff[j] = min(max(gq, qb0), qb1) * A.nbf + min(max(gp, pa0), pa1);
    }
    const uint32_t off1 = tc::off_mnmajor(warp * 16 + 8 * qh, rp);
    // the slot's terms of the group being produced, two per lane, multipoles
    // ascending: density offset, coefficient, multipole (-1: block below the
    // screen). Their
    // tiles stream through one register buffer: an element's next value is
    // loaded, for the next batch too, as soon as the last one is added.
    int toff[2], tL[2], E = 0, mask = 0;
    Val tc2[2];
    unsigned r0 = 0, r1 = 0;  // terms not yet loaded
    Val c{}, pv[8];  // coefficient and tile of the term in flight
    int off = 0;
    auto next_term = [&]() {  // its offset and coefficient; false: none left in the group
      if (!(r0 | r1)) return false;
      const bool lo = r0 != 0;
      const int at = __ffs(lo ? r0 : r1) - 1;
      if (lo) r0 &= r0 - 1; else r1 &= r1 - 1;
      off = __shfl_sync(0xffffffffu, lo ? toff[0] : toff[1], at);
      if constexpr (F64) {
        c = __shfl_sync(0xffffffffu, lo ? tc2[0] : tc2[1], at);
      } else {
        c.x = __shfl_sync(0xffffffffu, lo ? tc2[0].x : tc2[1].x, at);
        c.y = __shfl_sync(0xffffffffu, lo ? tc2[0].y : tc2[1].y, at);
      }
      return true;
    };
    // A group's terms come in three steps, each load's latency covered by a
    // part of the batch before: the block's range, its terms, the tile maxima.
    int4 next = 8 * g0 + warp < count ? S.oinfo[8 * g0 + warp] : make_int4(-1, 0, 0, -1);
    int tblk[2], pairjk = -1;
    unsigned bd[2];  // tile maxima: bits of a float, of a double's high word
    auto terms_of = [&](int g) {
      const int4 info = next;  // block, first term, terms, j | k << 16
      next = g + 1 < g1 && 8 * g + 8 + warp < count ? S.oinfo[8 * g + 8 + warp] : make_int4(-1, 0, 0, -1);
      pairjk = info.w;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        tblk[r] = -1;
        if (lane + 32 * r < info.z) {
          const int uu = info.y + lane + 32 * r;
          tblk[r] = A.kterm_blk[uu];
          if constexpr (F64) tc2[r] = A.kterm_coef[uu]; else tc2[r] = A.kterm_coef2[uu];
          toff[r] = A.kterm_off[uu];
          tL[r] = A.kterm_L[uu];
        }
      }
    };
    auto bounds_of = [&]() {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        bd[r] = 0u;
        if (tblk[r] >= 0 && act[tblk[r]])
          bd[r] = S.tmax[((size_t)tblk[r] * A.nel + a) * A.nel + b];
        else
          tL[r] = -1;
      }
    };
    // the scan of group g, and one exponent for its scaled tiles from the
    // largest entries of the density tiles
    auto enter = [&](int g) {
      unsigned any = 0;
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (tL[r] >= 0) any |= 1u << tL[r];
      r0 = __ballot_sync(0xffffffffu, tL[0] >= 0);
      r1 = __ballot_sync(0xffffffffu, tL[1] >= 0);
      mask = (int)__reduce_or_sync(0xffffffffu, any);
      if (next_term())
#pragma unroll
        for (int j = 0; j < 8; ++j) pv[j] = src[off + coff[j]];
      // |X_L| <= sum of |c| max|P| (high words and roundings: 2^-20), summed
      // upwards in units of 2^(e0 - 24): the largest multipole's, scaled by its
      // tables, gives E (s_hi - 96 at least: every scale stays a normal float)
      unsigned mx = 0, su[2], top = 0;
      int e0;
      if constexpr (F64) {
        double v[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          v[r] = tL[r] < 0 ? 0.0
                           : __hiloint2double((int)bd[r], -1) * (fabs(tc2[r]) * 1.000001) * exp2d(m.sL[tL[r]] - s_hi);
          mx = max(mx, (unsigned)__double2hiint(v[r]));
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        e0 = max((int)(mx >> 20) - 1022, -900);
#pragma unroll
        for (int r = 0; r < 2; ++r) su[r] = __double2uint_ru(v[r] * exp2d(24 - e0));
      } else {
        float v[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          v[r] = tL[r] < 0 ? 0.f : __uint_as_float(bd[r]) * (fabsf(tc2[r].x) * 1.000001f * exp2i(m.sL[tL[r]] - s_hi));
          mx = max(mx, __float_as_uint(v[r]));
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        e0 = max((int)(mx >> 23) - 126, -96);
#pragma unroll
        for (int r = 0; r < 2; ++r) su[r] = __float2uint_ru(v[r] * exp2i(24 - e0));
      }
      for (int L = 0; L < NL; ++L)
        top = max(top, __reduce_add_sync(0xffffffffu, (tL[0] == L ? su[0] : 0u) + (tL[1] == L ? su[1] : 0u)));
      E = max(s_hi + (F64 ? -900 : -96), s_hi + e0 + 8 - __clz(top));
      if (mx >= (F64 ? 0x7FF00000u : 0x7F800000u)) E = kBadExp;  // a value that is not finite
      if (lane == 0) {
        m.ex[g & 3][warp] = E;
        m.mask[g & 3][warp] = mask;
        m.jk[g & 3][warp] = pairjk;
      }
    };
    // slot's tile of multipole L into stage st
    auto produce = [&](int L, int st) {
      if ((mask >> L) & 1) {
        int left = __popc(__ballot_sync(0xffffffffu, tL[0] == L)) + __popc(__ballot_sync(0xffffffffu, tL[1] == L));
        std::conditional_t<F64, double, ffv> x[8];
        {  // an exact product: no sum to carry
          const Val cc = c;
          const bool more = next_term();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if constexpr (F64) {
              x[j] = cc * pv[j];
            } else {
              const float p = __fmul_rn(cc.x, pv[j].x);
              float pe = fmaf(cc.x, pv[j].x, -p);
              pe = fmaf(cc.x, pv[j].y, pe);
              x[j] = {p, fmaf(cc.y, pv[j].x, pe)};
            }
            if (more) pv[j] = src[off + coff[j]];
          }
        }
#pragma unroll 1
        while (--left > 0) {
          const Val cc = c;
          const bool more = next_term();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if constexpr (F64) x[j] = fma(cc, pv[j], x[j]); else x[j] = ff_fma(x[j], cc, pv[j]);
            if (more) pv[j] = src[off + coff[j]];
          }
        }
        if (edge)
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (!((vm >> j) & 1u)) x[j] = {};
        uint32_t pk[NX][4];
        if constexpr (F64) digits_fixed(x, E - m.sL[L], pk); else digits_pairs(x, exp2i(30 + m.sL[L] - E), pk);
        unsigned char* o = A1 + st * NX * APLANE + off1;
#pragma unroll
        for (int k = 0; k < NX; ++k)
          *reinterpret_cast<uint4*>(o + k * APLANE) = make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
      }
      // (operand rows of an idle slot keep their old digits: a tensor-core row
      // only feeds the same row of the result)
    };

    // the last warp through its part of batch n issues the second product of
    // batch n (L2 >= 0; start: the first of its group) and the first product of
    // batch n + 1 (L1 >= 0)
    auto issue = [&](int st, int L1, int L2, bool start) {
      tc::fence_before_sync();
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        uint32_t was;
        asm volatile("atom.acq_rel.cta.shared.add.u32 %0, [%1], 1;"
                     : "=r"(was)
                     : "r"(tc::smem_u32(&m.arrived))
                     : "memory");
        // (not after a warp gave up, which it says before it arrives)
        if ((was & (PW - 1)) == PW - 1 && was < kGaveUp) {
          tc::fence_after_sync();
          if (L1 >= 0) {
            const uint64_t dA = tc::smem_desc(tc::smem_u32(A1 + st * NX * APLANE));
            const uint64_t dT = tc::smem_desc(tc::smem_u32(T1 + L1 * PD * TPLANE));
#pragma unroll
            for (int kx = 0; kx < NX; ++kx)
              tc::mma_bf16(tD1 + 16 * kx, dA + (uint64_t)(kx * APLANE >> 4), dT, tc::idesc_f16(128, 16 * (PD - kx), 1, 0),
                           kx > 0 ? 1u : 0u);
          }
          if (L2 >= 0) {
            const uint64_t dA = tc::smem_desc(tc::smem_u32(A2)), dT = tc::smem_desc(tc::smem_u32(T2 + L2 * PD * TPLANE));
#pragma unroll
            for (int ky = 0; ky < PD; ++ky)
              tc::mma_bf16(tD2 + 16 * ky, dA + (uint64_t)(ky * APLANE >> 4), dT, tc::idesc_f16(128, 16 * (PD - ky), 1, 0),
                           (!start || ky > 0) ? 1u : 0u);
          }
          tc::mma_commit(&m.done);
        }
      }
      __syncwarp();
    };

    // ---- read-back: tensor-memory lanes 32 (w & 3) .. (two slots), columns
    // 8 half ..; lane = (slot, q) in the first product, (slot, i) in the second ----
    const int qw = warp & 3, half = warp >> 2;
    const uint32_t lane_off = (uint32_t)(32 * qw) << 16;
    const int oslot = 2 * qw + (lane >> 4), oi = lane & 15;
    const uint32_t off2 = tc::off_mnmajor(oslot * 16 + 8 * half, oi);
    int E2 = 0, mask2 = 0, jk = -1;  // of the group being read back
    // a group's sums -> FP64: rows p = oi, columns q = 8 half + j; staged in
    // this warp's part of the (free) second operand for the transposed partner
    auto store_group = [&]() {
      // entry (slot, r, c): 1 KB of each of four planes per pair of slots
      auto stage = [&](int r, int cc) {
        const int idx = (lane >> 4) * 256 + r * 16 + (cc ^ r);  // ^ r: spread over the banks
        return reinterpret_cast<double*>(A2 + (idx >> 7) * APLANE + qw * 1024) + (idx & 127);
      };
      const int ea = m.alpha[oi] + E2;  // (FP64 tiles are scaled to below 1/4)
#pragma unroll 1
      for (int h = 8 * half; h < 8 * half + 8; h += 4) {
        float v[PD][4];
        tmem_ld_pairs(tD2 + lane_off + h, v);
        double y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float lv[PD];
#pragma unroll
          for (int d = 0; d < PD; ++d) lv[d] = v[d][j];
          if constexpr (F64)
            y[j] = -levels_to_f64(lv, ea + m.beta[h + j] + 2);
          else
            y[j] = -levels_to_d(lv, (max(ea + m.beta[h + j], -800) + 896) << 20);
          if (E2 == kBadExp) y[j] = __longlong_as_double(0x7ff8000000000000ll);
          if (symmetric) *stage(oi, h + j) = y[j];
        }
        if (jk >= 0) store_rows(A, S, K, a, b, jk & 0xFFFF, jk >> 16, oi, h, y);
      }
      if (symmetric) {
        // both column halves are staged: warps w and w + 4
        pair_sync(qw);
#pragma unroll 1
        for (int h = 8 * half; h < 8 * half + 8; h += 4) {
          double y[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) y[j] = *stage(h + j, oi);
          if (jk >= 0) store_rows(A, S, K, b, a, jk >> 16, jk & 0xFFFF, oi, h, y);
        }
        // read before the next batch's digits overwrite it
        pair_sync(qw);
      }
    };
    // iteration n produces batch n + 1 and reads batch n back
    uint32_t limit = T.wait;  // of this warp's next wait
    int g = g0 - 1, cur = 0;  // multipoles left of group g
    bool start = false;       // the first of its group
    terms_of(g0);
    bounds_of();
    for (int n = -1;; ++n) {
      // ---- the batch after this one ----
      int gn = g;
      int nxt = cur & (cur - 1);
      const bool begin = !nxt && ++gn < g1;
      if (begin) {
        nxt = S.gmask[gn];
        enter(gn);
      }
      if (nxt) produce(__ffs(nxt) - 1, (n + 1) & 1);
      const bool ahead = nxt && !(nxt & (nxt - 1)) && gn + 1 < g1;  // the one after that starts a group
      if (ahead) terms_of(gn + 1);
      const int L = __ffs(cur) - 1;
      if (n >= 0) {
        // this batch's first product, the last one's second. Where a wait runs
        // out nothing more is issued and the unit is marked below, but the warp
        // stays in the loop: its partner meets it at barriers without a limit.
        if (!__all_sync(0xffffffffu, tc::mbar_wait(&m.done, (uint32_t)(n & 1), limit))) {
          if (lane == 0) {
            atomicMin(&m.fail, n);
            atomicOr(&m.arrived, kGaveUp);
          }
          limit = 0;
          jk = -1;
        }
        tc::fence_after_sync();
        if (start || !cur) {
          if (n > 0) store_group();
          if (!cur) break;
          E2 = m.ex[g & 3][oslot];
          mask2 = m.mask[g & 3][oslot];
          // (the warps that gave up no longer meet the others at every batch: what
          // those say of a group may not be there yet, so nothing is stored)
          jk = limit ? m.jk[g & 3][oslot] : -1;
        }
        // ---- levels -> balanced digits of Y = A X, the second product's
        // MN-major operand: rows (slot, i), K = q ----
        // the second product accumulates over the multipoles: a slot that is
        // idle in this one adds zeros
        const bool idle = !((mask2 >> L) & 1);
        const bool none = __all_sync(0xffffffffu, idle);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {  // 4 columns at a time: registers
          uint32_t pk[PD][2];
          if (!none) {
            float v[PD][4];
            tmem_ld_pairs(tD1 + lane_off + 8 * half + 4 * h, v);
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
              float y[PD][2];
#pragma unroll
              for (int w = 0; w < 2; ++w) {
                float lv[PD];
#pragma unroll
                for (int d = 0; d < PD; ++d) lv[d] = v[d][2 * jj + w];
                carry_pairs(lv, y[0][w], y[1][w]);
#pragma unroll
                for (int k = 2; k < PD; ++k) y[k][w] = lv[k - 1];
              }
#pragma unroll
              for (int k = 0; k < PD; ++k) pk[k][jj] = pack_f16(y[k][0], y[k][1]);
            }
          }
#pragma unroll
          for (int k = 0; k < PD; ++k)
            *reinterpret_cast<uint2*>(A2 + k * APLANE + off2 + 8 * h) =
                idle ? make_uint2(0, 0) : make_uint2(pk[k][0], pk[k][1]);
        }
      }
      if (ahead) bounds_of();
      issue((n + 1) & 1, nxt ? __ffs(nxt) - 1 : -1, L, start);
      g = gn;
      cur = nxt;
      start = begin;
    }
  }
  __syncthreads();
  if (m.fail != kNoFail) {  // uniform over the CTA
    if (t == 0) {
      atomicExch(T.err, 1);
      // the products of that batch may still be running (none came after them):
      // the tensor memory is released after them
      if (!tc::mbar_wait(&m.done, (uint32_t)(m.fail & 1), kWait))
        for (int i = 0; i < 100; ++i) __nanosleep(1000);
    }
    const int4 v = units[blockIdx.x];
    mark_unit(v, min(8 * v.w, S.ocount[0]), symmetric, A.nn, A.nel, A.nrad, A.nang, A.nbf, S.olist, S.khalo, K);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tD1, 256);
}

// ------------------------------------------------------------------------
// Diagonal element tiles. Per element a, group of up to 16 output blocks
// and row tile of 128 rows t of Tk, one batch per multipole L:
//     D[t, 16 level + slot] = sum_{kt+kx=level} sum_v Tk_kt[t, v] X_kx[slot, v],
// v = p + q nn. Tk's digit planes are streamed through shared memory one K
// step (16 columns v) at a time by bulk asynchronous copies, four steps in
// flight; the density digits of all 16 slots are resident, those of the next
// multipole beside those in use. For table digit kt the density planes kx =
// 0..6-kt are consecutive and form one operand of N = 16 (7 - kt). The level
// sums here run over up to nn^2 products: the leading levels stay exact, and a
// rounding in the deepest ones is below 2^-60 of max|K|.
// A chain of short steps, so bound by latency: copies, products and the digit
// work each have their own warps and run a multipole ahead of one another. Two
// CTAs per SM with one thread that copied, issued and waited in turn took 148
// us for Kr and 61 us for Ne (FP64 form, cold), this 115 and 29.

namespace {
constexpr int DSLOT = 16;  // output blocks per diagonal group
}

__global__ void tc_tk_digits_kernel(const double* __restrict__ tk, int NL, int nel, int n2, int mtiles, int ksteps,
                                    unsigned char* __restrict__ out, int* __restrict__ rowexp) {
  const int mt = blockIdx.x, le = blockIdx.y, m = threadIdx.x;  // le = L * nel + e
  const int t = 128 * mt + m;
  const double* Tm = tk + (size_t)le * n2 * n2;
  int ex = 0;
  if (t < n2) {
    double rs = 0.0;
    for (int v = 0; v < n2; ++v) rs += fabs(Tm[t + (size_t)v * n2]);
    if (rs > 0.0) frexp(rs, &ex);  // rs <= 2^ex
  }
  rowexp[((size_t)le * mtiles + mt) * 128 + m] = ex;
  unsigned char* base = out + ((size_t)le * mtiles + mt) * ksteps * ND * APLANE;
  for (int v = 0; v < 16 * ksteps; ++v) {
    double r = (t < n2 && v < n2) ? ldexp(Tm[t + (size_t)v * n2], -ex) : 0.0;
    unsigned char* plane = base + (size_t)(v >> 4) * ND * APLANE;
    const uint32_t off = tc::off_kmajor(m, v & 15);
#pragma unroll
    for (int k = 0; k < ND; ++k) {
      r *= 256.0;
      const double dg = rint(r);
      r -= dg;
      *reinterpret_cast<__nv_bfloat16*>(plane + k * APLANE + off) = __float2bfloat16_rn((float)dg);
    }
  }
}

constexpr int DST = 4;                   // stages of the table stream (at most)
constexpr int DW = 8;                    // working warps
constexpr int DTHREADS = 32 * (DW + 2);  // a copying and an issuing one

// warps 0-7: recouple and digitise the density vectors of one multipole while
// the products of the one before run, then read those back; warp 8 streams the
// tables' digits, warp 9 issues
// NC: chunks of eight density entries per thread (2: up to 16 nodes, 3: 17)
template <bool F64, int NC>
__global__ void __launch_bounds__(DTHREADS, 1) k_diag_tc(DevAtom A, DevScratch S, DevTC T, int symmetric,
                                                         const double* __restrict__ P, double* __restrict__ K) {
  using Val = std::conditional_t<F64, double, float2>;
  using Sum = std::conditional_t<F64, double, ffv>;
  constexpr int NX = F64 ? ND : NDX;  // digits of the density vectors
  const Val* src;
  if constexpr (F64) src = P; else src = S.p2;
  const int nn = A.nn, n2 = nn * nn, NL = A.NL, nang2 = A.nang * A.nang;
  const int ksteps = T.dksteps, mtiles = T.dmtiles, nst = T.dstages;
  // unit = (element, row tile, group of 16 active output blocks); the list is
  // made by the density pass (j <= k only in symmetric mode)
  const int count = symmetric ? S.ocount[1] : S.ocount[0];
  const int* list = symmetric ? S.olist + nang2 : S.olist;
  const int ngr = (count + DSLOT - 1) / DSLOT;
  const int g = blockIdx.x % T.dgroups, mt = (blockIdx.x / T.dgroups) % mtiles, a = blockIdx.x / (T.dgroups * mtiles);
  if (g >= ngr) return;  // uniform over the CTA
  extern __shared__ __align__(1024) unsigned char smraw[];
  unsigned char* Abuf = smraw;                  // nst x ND planes of 128 x 16
  unsigned char* Bx = Abuf + nst * ND * APLANE;  // 2 x ksteps x ND planes of 16 x 16
  const size_t bsize = (size_t)ksteps * ND * TPLANE;
  int* exs = reinterpret_cast<int*>(Bx + 2 * bsize);  // [4][16] slot exponents (bits) of four multipoles
  int* sact = exs + 4 * DSLOT;                        // [NL][16]
  int* gent = sact + NL * DSLOT;                      // [16][NL]
  int* gjk = gent + NL * DSLOT;                       // [16]
  int* fail = gjk + DSLOT;                            // [2]: flag, number of multipoles
  int* actL = fail + 2;                               // [NL] the multipoles of the group's entries
  uint64_t* full = reinterpret_cast<uint64_t*>(actL + NL + (NL & 1));
  uint64_t* empty = full + DST;
  uint64_t* bfull = empty + DST;  // [2] density digits there
  uint64_t* done = bfull + 2;     // [2] products finished
  uint64_t* drain = done + 2;     // every product finished (of a CTA that gives up)
  uint32_t* tslot = reinterpret_cast<uint32_t*>(drain + 1);
  unsigned char* act = reinterpret_cast<unsigned char*>(tslot + 2);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int qw = warp & 3, half = warp >> 2;

  if (t < DSLOT) {
    const int jk = g * DSLOT + t < count ? list[g * DSLOT + t] : -1;
    gjk[t] = jk;
    for (int L = 0; L < NL; ++L) {
      gent[t * NL + L] = -1;
      sact[L * DSLOT + t] = 0;
    }
    if (jk >= 0)
      for (int e = A.kjk_ptr[jk]; e < A.kjk_ptr[jk + 1]; ++e) {
        gent[t * NL + A.kent_L[e]] = e;
        sact[A.kent_L[e] * DSLOT + t] = S.ent_act[e] ? 1 : 0;
      }
  }
  for (int idx = t; idx < nang2; idx += blockDim.x) act[idx] = S.act[idx];
  // the zero seventh plane of float-pair densities in every K step (operands of N = 112)
  for (int idx = t; NX < ND && idx < 2 * ksteps * (TPLANE / 16); idx += blockDim.x) {
    const int ks = idx / (TPLANE / 16), o = idx % (TPLANE / 16);
    reinterpret_cast<uint4*>(Bx + ((size_t)ks * ND + NDX) * TPLANE)[o] = make_uint4(0, 0, 0, 0);
  }
  if (t < 4 * DSLOT) exs[t] = F64 ? 64 : 0;  // (FP64: so far above a zero that its significand is shifted out)
  if (t == 0) {
    fail[0] = 0;
    for (int i = 0; i < DST; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&bfull[i], DW);
      tc::mbar_init(&done[i], 1);
    }
    tc::mbar_init(drain, 1);
  }
  if (warp == DW + 1) {
    tc::tmem_alloc(tslot, 256);
    tc::tmem_relinquish();
  }
  __syncthreads();
  if (t == 0) {
    int n = 0;
    for (int L = 0; L < NL; ++L) {
      int any = 0;
      for (int s = 0; s < DSLOT; ++s) any |= sact[L * DSLOT + s];
      if (any) actL[n++] = L;
    }
    fail[1] = n;
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tD = *tslot;
  const int na = fail[1];
  const int row = 32 * qw + lane, trow = 128 * mt + row;  // a working thread's tensor-memory lane
  Sum acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = {};

  int copied = 0;  // copies started (by the copying thread)
  if (warp == DW) {
    if (lane == 0) {
      bool ok = true;
      int& it = copied;
      for (int n = 0; n < na && ok; ++n) {
        const unsigned char* Ag =
            T.tk_digits + (((size_t)actL[n] * A.nel + a) * mtiles + mt) * ksteps * ND * APLANE;
        for (int ks = 0; ks < ksteps; ++ks, ++it) {
          const int s = it % nst;
          if (it >= nst && !tc::mbar_wait(&empty[s], (uint32_t)((it / nst - 1) & 1), T.wait)) {
            ok = false;
            break;
          }
          tc::mbar_expect_tx(&full[s], ND * APLANE);
          tc::bulk_g2s(Abuf + s * ND * APLANE, Ag + (size_t)ks * ND * APLANE, ND * APLANE, &full[s]);
        }
      }
      if (!ok) atomicExch(fail, 1);
    }
  } else if (warp == DW + 1) {
    if (lane == 0) {
      bool ok = true;
      int it = 0;
      for (int n = 0; n < na && ok; ++n) {
        const int bf = n & 1;
        // (the working warps arrive after reading batch n - 2 back)
        if (!(ok = tc::mbar_wait(&bfull[bf], (uint32_t)((n >> 1) & 1), T.wait))) break;
        tc::fence_after_sync();
        const uint64_t dB = tc::smem_desc(tc::smem_u32(Bx + bf * bsize));
        for (int ks = 0; ks < ksteps; ++ks, ++it) {
          const int s = it % nst;
          if (!(ok = tc::mbar_wait(&full[s], (uint32_t)((it / nst) & 1), T.wait))) break;
          tc::fence_after_sync();
          const uint64_t dA = tc::smem_desc(tc::smem_u32(Abuf + s * ND * APLANE));
#pragma unroll
          for (int kt = 0; kt < ND; ++kt)
            tc::mma_bf16(tD + 128 * bf + 16 * kt, dA + (uint64_t)(kt * APLANE >> 4),
                         dB + (uint64_t)((size_t)ks * ND * TPLANE >> 4), tc::idesc_bf16(128, 16 * (ND - kt), 0, 0),
                         (ks > 0 || kt > 0) ? 1u : 0u);
          tc::mma_commit(&empty[s]);
        }
        if (ok) tc::mma_commit(&done[bf]);
      }
      if (!ok) atomicExch(fail, 1);
    }
  } else {
    const int nchunk = DSLOT * 2 * ksteps;  // chunks of 8 consecutive v per slot
    for (int n = 0; n <= na; ++n) {
      if (n < na) {
        const int L = actL[n];
        int* ex = exs + (n & 3) * DSLOT;
        // ---- recouple the 16 density vectors and take each slot's exponent ----
        Sum xs[NC][8];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int ch = t + c * 256;
#pragma unroll
          for (int j = 0; j < 8; ++j) xs[c][j] = {};
          if (ch >= nchunk) continue;
          const int s = ch / (2 * ksteps), v0 = 8 * (ch % (2 * ksteps));
          if (!sact[L * DSLOT + s]) continue;
          const int ent = gent[s * NL + L];
          int eo[8];  // density offsets of the 8 elements (nbf^2 < 2^31), -1: outside the basis
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int v = v0 + j, p = v % nn, q = v / nn;
            const int gp = gfun(A, a, p), gq = gfun(A, a, q);
            eo[j] = (v < n2 && gp >= 0 && gp < A.nrad && gq >= 0 && gq < A.nrad) ? gq * A.nbf + gp : -1;
          }
          // two terms' loads in flight together
          const int u1 = A.kent_ptr[ent + 1];
          for (int uu = A.kent_ptr[ent]; uu < u1; uu += 2) {
            Val cf[2], pv[2][8];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
              const bool on = uu + w < u1 && act[A.kterm_blk[uu + w]];
              cf[w] = {};
              if constexpr (F64) {
                if (on) cf[w] = A.kterm_coef[uu + w];
              } else {
                if (on) cf[w] = A.kterm_coef2[uu + w];
              }
              const Val* pb = src + (on ? A.kterm_off[uu + w] : 0);
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                pv[w][j] = {};
                if (on && eo[j] >= 0) pv[w][j] = pb[eo[j]];
              }
            }
#pragma unroll
            for (int w = 0; w < 2; ++w)
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                if constexpr (F64) xs[c][j] = fma(cf[w], pv[w][j], xs[c][j]); else xs[c][j] = ff_fma(xs[c][j], cf[w], pv[w][j]);
              }
          }
          unsigned eb = 0;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if constexpr (F64) {
              eb = max(eb, ((unsigned)__double2hiint(xs[c][j]) >> 20) & 0x7FFu);
            } else {
              xs[c][j] = ff_norm(xs[c][j].hi, xs[c][j].lo);
              eb = max(eb, (__float_as_uint(xs[c][j].hi) >> 23) & 0xFFu);
            }
          }
          atomicMax(&ex[s], (int)eb);
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (t < DSLOT) exs[((n + 2) & 3) * DSLOT + t] = F64 ? 64 : 0;  // last read for batch n - 2
        // ---- digits: B[ks][kx][row slot, k = v mod 16]; batch n - 2 has been
        // read back, its products are over ----
        unsigned char* Bn = Bx + (n & 1) * bsize;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int ch = t + c * 256;
          if (ch >= nchunk) continue;
          const int s = ch / (2 * ksteps), kk = ch % (2 * ksteps), ks = kk >> 1, h = kk & 1;
          uint32_t pk[NX][4];
          if constexpr (F64) digits_fixed256(xs[c], ex[s] - 1022, pk); else digits_of(xs[c], tile_exponent((unsigned)ex[s]), pk);
          const uint32_t off = tc::off_kmajor(s, 8 * h);
#pragma unroll
          for (int k = 0; k < NX; ++k)
            *reinterpret_cast<uint4*>(Bn + ((size_t)ks * ND + k) * TPLANE + off) =
                make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
        }
        tc::fence_before_sync();
        tc::fence_async_smem();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&bfull[n & 1]);
      }
      if (n == 0) continue;
      // ---- the batch before: levels scaled by 2^(alpha_t + E_slot), summed
      // over the multipoles; columns [8 half, 8 half + 8) = slots ----
      const int m = n - 1, L = actL[m];
      const int* ex = exs + (m & 3) * DSLOT;
      const int ea = T.tk_rowexp[(((size_t)L * A.nel + a) * mtiles + mt) * 128 + row];
      const bool ok = tc::mbar_wait(&done[m & 1], (uint32_t)((m >> 1) & 1), T.wait);
      if (!__all_sync(0xffffffffu, ok)) {
        // (the other working warps meet at barrier 1: all give up in turn)
        if (lane == 0) atomicExch(fail, 1);
        if (n < na) continue;
        break;
      }
      tc::fence_after_sync();
      float v[ND][8];
      tmem_ld_levels(tD + 128 * (m & 1) + ((uint32_t)(32 * qw) << 16) + 8 * half, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int s = 8 * half + j;
        if (!sact[L * DSLOT + s]) continue;
        float lv[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d) lv[d] = v[d][j];
        if constexpr (F64)
          acc[j] += ex[s] == 0x7FF ? __longlong_as_double(0x7ff8000000000000ll) : levels_to_f64(lv, ea + ex[s] - 1022);
        else
          acc[j] = ff_add(acc[j], levels_to_pair(lv, exp2i(ea + tile_exponent((unsigned)ex[s]))));
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();

  // ---- store K_jk(a,a)[p, q], t = p + q nn; with a symmetric density also
  // the transposed partner K_kj(a,a)[q, p] (j != k) ----
  const bool failed = fail[0] != 0;
  if (warp < DW && trow < n2) {
    const int p = trow % nn, q = trow / nn;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int jk = gjk[8 * half + j];
      if (jk < 0) continue;
      double y;
      if constexpr (F64) y = -acc[j]; else y = -pair_to_d(acc[j]);
      if (failed) y = __longlong_as_double(0x7ff8000000000000ll);
      k_store_tile(A, S, K, a, a, jk, p, q, y);
      const int j0 = jk % A.nang, k0 = jk / A.nang;
      if (symmetric && j0 != k0) k_store_tile(A, S, K, a, a, k0 + j0 * A.nang, q, p, y);
    }
  }
  // the copies in flight must land before the CTA leaves
  if (failed && copied > 0)
    for (int i = max(0, copied - nst); i < copied; ++i)
      tc::mbar_wait(&full[i % nst], (uint32_t)((i / nst) & 1), kWait);
  if (failed && warp == DW + 1 && lane == 0) {
    atomicExch(T.err, 1);
    // products may still be running: the tensor memory is released after them
    tc::mma_commit(drain);
    tc::mbar_wait(drain, 0, kWait);
  }
  __syncthreads();
  if (warp == DW + 1) tc::tmem_dealloc(tD, 256);
}

size_t tc_smem_bytes(int NL, int nang, bool f64) {
  return (size_t)(2 * (f64 ? PD : PX) + PD) * APLANE + (size_t)2 * NL * PD * TPLANE + sizeof(PairMeta) +
         (size_t)nang * nang + 16;
}

size_t tc_diag_smem_bytes(int NL, int ksteps, int nang, int stages) {
  return (size_t)stages * ND * APLANE + (size_t)2 * ksteps * ND * TPLANE +
         sizeof(int) * (4 * DSLOT + NL * DSLOT * 2 + DSLOT + 2 + NL + 1) + 8 * (2 * DST + 5) + 8 + (size_t)nang * nang + 64;
}

// P: the FP64 form (from the density itself), nullptr: the split form (from S.p2)
cudaError_t launch_k_tiles_tc(const DevAtom& A, const DevScratch& S, const DevTC& T, bool symmetric, const double* P,
                              double* K, cudaStream_t st) {
  const int n = symmetric ? T.n_sym : T.n_all;
  if (n == 0) return cudaSuccess;
  const size_t smem = tc_smem_bytes(A.NL, A.nang, P != nullptr);
  auto kern = P ? k_tiles_tc<true> : k_tiles_tc<false>;
  const cudaError_t e = smem_limit(kern, smem);
  if (e != cudaSuccess) return e;
  kern<<<n, PTHREADS, smem, st>>>(A, S, T, symmetric ? T.units_sym : T.units_all, symmetric ? 1 : 0, P, K);
  return cudaGetLastError();
}

cudaError_t launch_tk_digits(const DevAtom& A, int mtiles, int ksteps, unsigned char* out, int* rowexp,
                             cudaStream_t st) {
  const int n2 = A.nn * A.nn;
  cudaError_t e = cudaMemsetAsync(out, 0, (size_t)A.NL * A.nel * mtiles * ksteps * ND * APLANE, st);
  if (e != cudaSuccess) return e;
  tc_tk_digits_kernel<<<dim3(mtiles, A.NL * A.nel), 128, 0, st>>>(A.tk, A.NL, A.nel, n2, mtiles, ksteps, out, rowexp);
  return cudaGetLastError();
}

cudaError_t launch_k_diag_tc(const DevAtom& A, const DevScratch& S, const DevTC& T, bool symmetric, const double* P,
                             double* K, cudaStream_t st) {
  DevTC Td = T;
  const int nblk = symmetric ? A.nang * (A.nang + 1) / 2 : A.nang * A.nang;
  Td.dgroups = (nblk + DSLOT - 1) / DSLOT;
  const int n = A.nel * T.dmtiles * Td.dgroups;
  // as many stages as fit (four up to 16 nodes, three for 17) and there are steps
  // for: with less shared memory element-pair tiles run on the same SM
  int dev = 0, most = 0;
  cudaError_t e0 = cudaGetDevice(&dev);
  if (e0 == cudaSuccess) e0 = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e0 != cudaSuccess) return e0;
  Td.dstages = std::min(DST, A.NL * T.dksteps);
  while (Td.dstages > 2 && tc_diag_smem_bytes(A.NL, T.dksteps, A.nang, Td.dstages) > (size_t)most) --Td.dstages;
  const size_t smem = tc_diag_smem_bytes(A.NL, T.dksteps, A.nang, Td.dstages);
  const bool wide = DSLOT * 2 * T.dksteps > 512;
  auto kern = P ? (wide ? k_diag_tc<true, 3> : k_diag_tc<true, 2>) : (wide ? k_diag_tc<false, 3> : k_diag_tc<false, 2>);
  const cudaError_t e = smem_limit(kern, smem);
  if (e != cudaSuccess) return e;
  kern<<<n, DTHREADS, smem, st>>>(A, S, Td, symmetric ? 1 : 0, P, K);
  return cudaGetLastError();
}

}  // namespace hfg
