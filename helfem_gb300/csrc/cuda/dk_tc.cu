// Split-precision diatomic exchange, in-element (diagonal) tiles on the tensor
// cores: for every element e and active output block (j, k)
//   K_jk(e,e)[t] -= sum_lm fac_lm sum_ab sum_v tx_ab(lm, e)[t, v] X_ab(lm, jk)[v]
// (src/diatomic/basis.cpp:1960-2061 with the factor contracted into the
// exchange-ordered kernel tx; X_ab the four recoupled channel tiles, t = p +
// q nn, v = i + l nn), a matrix product of M = output blocks, N = tile entries
// t and K = 4 nn^2 per multipole and element.
//
// Arithmetic (as in k_tc.cu): fixed-point operands as balanced base-512 digits
// (integers up to 512, exact in f16), seven of the kernel, six of a tile; the kernel rows t are scaled
// so that their absolute row sum (all channels, with the multipole's factor)
// is at most 1, the recoupled tiles so that their largest entry is below 1.
// The tensor core sums the digit products level by level (acc_d = sum over
// digit pairs with k + l = d) in FP32 tensor memory. The 4 nn^2-term sums of
// digit products stay far below 2^24: the leading digits of a row obey its
// unit row sum, and the others are spread over +-256, so that a level's sum of
// 900 products has a spread below 2^21. The levels are carried into three
// floats and summed in FP64 over the multipoles.
//
// FP64 form (F64): the tiles are recoupled in FP64 and cut into seven digits by
// shifts of their significands (59 bits below the largest entry), the level
// sums (integers) added up in FP64: the error against the exact K is that of the
// FP64 kernels (H2 6.2e-15 and 6.4e-15, CO 1.005e-14 and 1.010e-14 of |K|). Whole
// K, FP64 kernels for these tiles and this form: H2 on 3 elements, l <= 4 0.55 and 0.29
// ms; N2 on 9 elements, l <= 10, m <= 3 132 and 87 ms.
//
// In both forms a tile with a value that is not finite gives NaN in its rows.
//
// Two passes: dk_tc_x recouples each (element, output block, multipole) once
// (sharing the sums over l between the output rows of one k) and writes its
// digits in the operand layout; dk_tc_gemm streams those and the table's
// digits through shared memory with bulk copies, one producer and one issuing
// warp beside eight warps that read the sums back. The table is read once per
// 128 output blocks (it was read once per 8 by the float-pair kernel this
// replaced). Whole split K, before and after: N2 on 3 elements, l <= 5, m <= 1
// 7.65 -> 0.41 ms; on 6 elements, l <= 10, m = 0 6.82 -> 1.17 ms; on 12
// elements, l <= 10, m <= 3 84.2 -> 44.2 ms (with the shared recoupling of the
// element pairs). Digits of as many (element, tile of
// 128 blocks) units as a fixed scratch holds are made at a time.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "dk_recouple.cuh"
#include "fixed.cuh"
#include "smem_limit.hpp"
#include "tc.cuh"

namespace hfg {
namespace {

constexpr int XD = DTC_XDIGITS;   // digits of a float-pair tile (54 bits: a float pair has 48)
constexpr int TD = DTC_TDIGITS;   // digits of the table, and levels kept
constexpr int APL = 4096;             // bytes of a 128 x 16 f16 plane
constexpr int TT = DTC_TT;            // tile entries t per CTA
constexpr int BPL = TT * 32;          // bytes of a TT x 16 f16 plane
constexpr int NSTAGE = 5;
constexpr int kNoRow = (int)0x80808080;
constexpr uint32_t kWait = DTC_WAIT;  // limit of the waits of a CTA that gives up

// six balanced base-512 digits of a float pair |x| < 2^E (weights 512^-(k+1))
__device__ __forceinline__ void digits512(float2 x, float s27, float (&d)[XD]) {
  const float h = __fmul_rn(x.x, s27), l = __fmul_rn(x.y, s27);  // scaled to |h| < 2^27
  d[0] = rnd_mul(h, 1.0f / 262144.0f);
  const float t1 = __fmaf_rn(d[0], -262144.0f, h);
  d[1] = rnd_mul(t1, 1.0f / 512.0f);
  const float t2 = __fmaf_rn(d[1], -512.0f, t1);
  d[2] = rnd(__fadd_rn(t2, l));
  float r = __fadd_rn(__fsub_rn(t2, d[2]), l);
#pragma unroll
  for (int k = 3; k < XD; ++k) {
    d[k] = rnd_mul(r, 512.0f);
    r = __fmaf_rn(r, 512.0f, -d[k]);
  }
}

// seven balanced base-512 digits (weights 512^-(k+1)) of 8 values |x| < 2^(E+2):
// with 256 added to every digit the digits are the 9-bit fields of the
// fixed-point number, and 1024 + field an f16 bit pattern
__device__ __forceinline__ void digits512_fixed(const double (&x)[8], int E, uint32_t (&pk)[TD][4]) {
  static_assert(TD == 7, "three fields in each of two words and one on top");
#pragma unroll
  for (int jj = 0; jj < 8; jj += 2) {
    uint32_t w[3][2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint64_t f = fixed_point<61>(x[jj + i], E) + 0x4020100804020100ull;
      w[0][i] = (uint32_t)f & 0x7FFFFFFu;
      w[1][i] = (uint32_t)(f >> 27) & 0x7FFFFFFu;
      w[2][i] = (uint32_t)(f >> 54);
    }
    auto digit = [](uint32_t a, uint32_t b) {
      const uint32_t u = (__byte_perm(a, b, 0x5410) & 0x01FF01FFu) | 0x64006400u;
      const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&u), __floats2half2_rn(1280.f, 1280.f));
      return *reinterpret_cast<const uint32_t*>(&d);
    };
    pk[0][jj / 2] = digit(w[2][0], w[2][1]);
#pragma unroll
    for (int k = 1; k < TD; ++k) {
      const int v = k <= 3 ? 1 : 0, sh = 9 * ((6 - k) % 3);
      pk[k][jj / 2] = digit(w[v][0] >> sh, w[v][1] >> sh);
    }
  }
}

// level sums (integers) -> FP64 times 2^k
__device__ __forceinline__ double levels512_f64(const float (&a)[TD], int k) {
  const int64_t u = ((int64_t)__float2int_rn(a[0]) << 18) + ((int64_t)__float2int_rn(a[1]) << 9) + __float2int_rn(a[2]);
  const int64_t v = ((int64_t)__float2int_rn(a[3]) << 27) + ((int64_t)__float2int_rn(a[4]) << 18) +
                    ((int64_t)__float2int_rn(a[5]) << 9) + __float2int_rn(a[6]);
  return fma(i2d(v), 1.4551915228366852e-11, i2d(u)) * exp2d(k - 36);  // 2^-36
}

// the value of the level sums (weights 512^-(d+2)) as three floats. The first
// two are exact where the value is far below the bound that scales it: with one
// float for the tail its rounding, 2^-51 of the bound, was the form's error
// (3.0e-14 of |K| for H2, 1.0e-14 now).
__device__ __forceinline__ void levels512(float (&a)[TD], float& head, float& mid, float& tail) {
#pragma unroll
  for (int d = TD - 1; d >= 1; --d) {
    const float c = rnd_mul(a[d], 1.0f / 512.0f);
    a[d] = __fmaf_rn(c, -512.0f, a[d]);
    a[d - 1] = __fadd_rn(a[d - 1], c);
  }
  const float y0 = rnd_mul(a[0], 1.0f / 512.0f), y1 = __fmaf_rn(y0, -512.0f, a[0]);
  const float h = __fmaf_rn(y1, 1.0f / 262144.0f, __fmul_rn(y0, 1.0f / 512.0f));
  const float m2 = __fmul_rn(a[1], 1.0f / 134217728.0f);
  const float sh = __fadd_rn(h, m2), bb = __fsub_rn(sh, h);
  const float e = __fadd_rn(__fsub_rn(h, __fsub_rn(sh, bb)), __fsub_rn(m2, bb));
  head = sh;
  mid = __fmaf_rn(__fmaf_rn(a[3], 1.0f / 512.0f, a[2]), 1.0f / 68719476736.0f, e);  // weight 2^-36 of a[2]
  tail = __fmul_rn(__fmaf_rn(__fmaf_rn(a[6], 1.0f / 512.0f, a[5]), 1.0f / 512.0f, a[4]), 5.551115123125783e-17f);
}

// all seven levels (TT columns apart) of 8 consecutive columns, one wait
__device__ __forceinline__ void ld_levels(uint32_t taddr, float (&v)[TD][8]) {
  static_assert(TD == 7 && TT == 64, "level count and stride of the load below");
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
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55])
      : "r"(taddr), "r"(taddr + 64), "r"(taddr + 128), "r"(taddr + 192), "r"(taddr + 256), "r"(taddr + 320), "r"(taddr + 384)
      : "memory");
#pragma unroll
  for (int d = 0; d < TD; ++d)
#pragma unroll
    for (int j = 0; j < 8; ++j) v[d][j] = __uint_as_float(r[8 * d + j]);
}

// the active output blocks of the call, and the units that they make
struct Blocks {
  const int* list;
  int count, ntile;
};
__device__ __forceinline__ Blocks blocks_of(const DevDiatomic& D, const DevDiatomicScratch& S, int symmetric) {
  Blocks b;
  b.list = symmetric ? S.jk_list + (size_t)D.nang * D.nang : S.jk_list;
  b.count = symmetric ? S.counts[1] : S.counts[0];
  b.ntile = (b.count + 127) / 128;
  return b;
}

}  // namespace

// ---- the table's column exponents, once per handle: grid (nlm*nel), threads
// over the columns (channel ab, v) ----
__global__ void dk_tc_colexp(DevDiatomic D, int* __restrict__ cexp) {
  const size_t le = blockIdx.x;
  const int n2 = D.nn * D.nn, nv = 4 * n2;
  const double* tx = D.tx + le * 4 * n2 * n2;
  for (int v = threadIdx.x; v < nv; v += blockDim.x) {
    double m = 0.0;
    for (int t = 0; t < n2; ++t) m = fmax(m, fabs(tx[t + (size_t)v * n2]));
    int ex = 0;
    if (m > 0.0) frexp(m, &ex);  // m < 2^ex
    cexp[le * nv + v] = ex;
  }
}

// ---- its digits: grid (t tiles, nlm*nel), one thread per (row t, quarter of
// the columns) ----
__global__ void __launch_bounds__(4 * TT) dk_tc_table(DevDiatomic D, DevDiaTC T, unsigned char* __restrict__ out,
                                                      int* __restrict__ rowexp) {
  __shared__ double part[4][TT];
  const int tt = blockIdx.x, ilm = blockIdx.y / D.nel;
  const size_t le = blockIdx.y;
  const int r = threadIdx.x % TT, c = threadIdx.x / TT, n2 = D.nn * D.nn, nv = 4 * n2;
  const int t = tt * TT + r;
  const double fac = (D.lmM[ilm] & 1) ? -D.lmfac[ilm] : D.lmfac[ilm];
  const double* tx = D.tx + le * 4 * n2 * n2;  // channel ab, column v: offset (ab n2 + v) n2
  const int* ce = T.cexp + le * nv;
  double rs = 0.0;
  if (t < n2)
    for (int v = c; v < nv; v += 4) rs += fabs(fac * tx[t + (size_t)v * n2] * exp2d(-ce[v]));
  part[c][r] = rs;
  __syncthreads();
  rs = part[0][r] + part[1][r] + part[2][r] + part[3][r];
  int ex = 0;
  if (rs > 0.0) frexp(rs, &ex);  // rs < 2^ex
  ex = max(ex, -900);  // (a zero's significand is shifted out)
  if (c == 0) rowexp[(le * T.ntt + tt) * TT + r] = ex + 2;  // the digits are of values below 1/4
  unsigned char* base = out + (le * T.ntt + tt) * T.ksteps * TD * BPL;
  for (int v8 = c; v8 < 2 * T.ksteps; v8 += 4) {
    double x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int v = 8 * v8 + j;
      x[j] = (t < n2 && v < nv) ? fac * tx[t + (size_t)v * n2] * exp2d(-ce[v]) : 0.0;
    }
    uint32_t pk[TD][4];
    digits512_fixed(x, ex, pk);
    unsigned char* p = base + (size_t)(v8 >> 1) * TD * BPL + tc::off_kmajor(r, 8 * (v8 & 1));
#pragma unroll
    for (int k = 0; k < TD; ++k)
      *reinterpret_cast<uint4*>(p + k * BPL) = make_uint4(pk[k][0], pk[k][1], pk[k][2], pk[k][3]);
  }
}

// ---- recoupled tiles of the units [u0, u0 + cap) as digits: items (element,
// active (k, group of rows), range of multipoles), or with `itemwise` one
// output block per item (the same operations per block) ----
template <int NN, bool F64>
__global__ void __launch_bounds__(NN == 15 ? 256 : 320, 2) dk_tc_x(DevDiatomic D, DevDiatomicScratch S, DevDiaTC T,
                                                                   const double* __restrict__ Pd, int symmetric,
                                                                   int itemwise, int u0, int nchunk) {
  using AR = std::conditional_t<F64, ArD, ArF>;
  using V = typename AR::V;
  constexpr int NX = F64 ? TD : XD;  // digits of a tile
  const int nn = NN > 0 ? NN : D.nn, n2 = nn * nn;
  extern __shared__ __align__(16) unsigned char smraw[];
  Chunk<AR, JC_DIAG>& C = *reinterpret_cast<Chunk<AR, JC_DIAG>*>(smraw);
  V* Xs = reinterpret_cast<V*>(smraw + sizeof(Chunk<AR, JC_DIAG>));  // [2][16 ksteps]
  __shared__ int s_js[JC_DIAG], s_row[JC_DIAG], s_unit[JC_DIAG], s_nj, s_use;
  __shared__ unsigned s_eb[JC_DIAG];
  const Blocks B = blocks_of(D, S, symmetric);
  if (B.count == 0) return;
  const int e_lo = u0 / B.ntile, e_hi = min(D.nel - 1, (u0 + T.cap - 1) / B.ntile);
  if (e_lo > e_hi) return;
  const Src<AR> Sr = src_of<AR>(D, S, Pd);
  const int nitem = itemwise ? B.count : S.counts[3];
  const int* kgl = S.kg_list + (size_t)D.nang * D.ngrp;
  const long total = (long)(e_hi - e_lo + 1) * nitem * nchunk;
  const int t = threadIdx.x, lane = t & 31;
  const bool live = t < n2;
  const int p = live ? t % nn : 0, q = live ? t / nn : 0;
  const int nv = 4 * n2, nv8 = 2 * T.ksteps;
  for (long w = blockIdx.x; w < total; w += gridDim.x) {
    const int e = e_lo + (int)(w / ((long)nitem * nchunk)), c = (int)(w % nchunk),
              it = (int)((w / nchunk) % nitem);
    int k;
    __syncthreads();
    if (itemwise) {
      const int jk = B.list[it];
      k = jk / D.nang;
      if (t == 0) {
        s_js[0] = jk % D.nang;
        s_nj = 1;
      }
    } else {
      k = kgl[it] / D.ngrp8;
      const int g = kgl[it] % D.ngrp8;
      if (t == 0) {
        int n = 0;
        for (int x = D.grp8_ptr[g]; x < D.grp8_ptr[g + 1]; ++x)
          if (S.jk_pos[D.msh[x] + k * D.nang] >= 0) s_js[n++] = D.msh[x];
        s_nj = n;
      }
    }
    __syncthreads();
    const int nj = s_nj;
    if (t == 0) s_use = 0;
    __syncthreads();
    if (t < nj) {
      const int pos = S.jk_pos[s_js[t] + k * D.nang], u = e * B.ntile + pos / 128 - u0;
      s_row[t] = pos % 128;
      s_unit[t] = (u >= 0 && u < T.cap) ? u : -1;
      if (s_unit[t] >= 0) s_use = 1;
    }
    __syncthreads();
    if (!s_use) continue;  // uniform over the CTA
    const int mj = D.mval[s_js[0]];
    const int gp = sgf(D, e, p), gq = sgf(D, e, q);
    const bool vpq = live && gp < D.nrad && gq < D.nrad;
    const V* pb = Sr.P + (size_t)gq * D.nd + gp;
    const int l0 = (int)((long)D.nlm * c / nchunk), l1 = (int)((long)D.nlm * (c + 1) / nchunk);
    int par = 0;
    for (int ilm = l0; ilm < l1; ++ilm) {
      const int L = D.lmL[ilm], Ma = D.lmM[ilm];
      typename AR::A x[JC_DIAG][4];
#pragma unroll
      for (int jj = 0; jj < JC_DIAG; ++jj)
#pragma unroll
        for (int ab = 0; ab < 4; ++ab) x[jj][ab] = AR::zero();
      bool any = false;
      for (int sgn = 0; sgn < (Ma ? 2 : 1); ++sgn) {
        const int M = sgn ? -Ma : Ma, mi = mj - M;
        if (mi < -D.mmax || mi > D.mmax) continue;
        const int xk = sal(D, k, L, M);
        if (D.al_ptr[xk] == D.al_ptr[xk + 1]) continue;
        const int* is = D.msh + D.msh_ptr[mi + D.mmax];
        const int ni_all = D.msh_ptr[mi + D.mmax + 1] - D.msh_ptr[mi + D.mmax];
        bool first = true;
        for (int i0 = 0; i0 < ni_all; i0 += IC) {
          const int ni = min(IC, ni_all - i0);
          par ^= 1;
          const int nl = chunk_fill<AR, JC_DIAG>(D, S, Sr, C, s_js, nj, k, L, M, is + i0, ni, par, first);
          first = false;
          if (nl == 0) continue;
          any = true;
          typename AR::A v0[IC], v2[IC];
          recouple_k<AR, JC_DIAG>(D, C, pb, vpq, is + i0, ni, nl, par, v0, v2);
          V a0[IC], a2[IC];
#pragma unroll
          for (int ii = 0; ii < IC; ++ii) {
            a0[ii] = AR::val(v0[ii]);
            a2[ii] = AR::val(v2[ii]);
          }
#pragma unroll
          for (int jj = 0; jj < JC_DIAG; ++jj) {
            if (jj >= nj) break;  // uniform
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) {
              const V c0 = C.j0[par][jj][ii], c2 = C.j2[par][jj][ii];
              if (AR::nz(c0) || AR::nz(c2)) {  // uniform
                x[jj][0] = AR::fma(x[jj][0], c0, a0[ii]);
                x[jj][1] = AR::fma(x[jj][1], c0, a2[ii]);
                x[jj][2] = AR::fma(x[jj][2], c2, a0[ii]);
                x[jj][3] = AR::fma(x[jj][3], c2, a2[ii]);
              }
            }
          }
          __syncthreads();  // the chunk's lists are read until here
        }
      }
      if (!any) continue;  // uniform over the CTA
      if (t < JC_DIAG) s_eb[t] = 0;
      // the column scaling of the table, inverted
      std::conditional_t<F64, double, float> cs[4];
#pragma unroll
      for (int ab = 0; ab < 4; ++ab) {
        const int ce = live ? T.cexp[((size_t)ilm * D.nel + e) * nv + ab * n2 + t] : 0;
        if constexpr (F64) cs[ab] = live ? exp2d(ce) : 0.0; else cs[ab] = live ? exp2i(ce) : 0.f;
      }
      __syncthreads();
#pragma unroll
      for (int jj = 0; jj < JC_DIAG; ++jj) {
        if (jj >= nj) break;
        unsigned eb = 0;
#pragma unroll
        for (int ab = 0; ab < 4; ++ab) {
          if constexpr (F64) {
            x[jj][ab] *= cs[ab];
            if (live) eb = max(eb, ((unsigned)__double2hiint(x[jj][ab]) >> 20) & 0x7FFu);
          } else {
            x[jj][ab] = ff_norm(x[jj][ab].hi * cs[ab], x[jj][ab].lo * cs[ab]);
            if (live) eb = max(eb, (__float_as_uint(x[jj][ab].hi) >> 23) & 0xFFu);
          }
        }
        eb = __reduce_max_sync(0xffffffffu, eb);
        if (lane == 0) atomicMax(&s_eb[jj], eb);
      }
      // two rows at a time: values to shared memory, then 8 columns per thread
#pragma unroll
      for (int j2 = 0; j2 < JC_DIAG; j2 += 2) {
        if (j2 >= nj) break;
        __syncthreads();
        if (live)
#pragma unroll
          for (int w2 = 0; w2 < 2; ++w2)
#pragma unroll
            for (int ab = 0; ab < 4; ++ab) {
              V y;
              if constexpr (F64) y = x[j2 + w2][ab]; else y = make_float2(x[j2 + w2][ab].hi, x[j2 + w2][ab].lo);
              Xs[w2 * 16 * T.ksteps + ab * n2 + t] = (ab == 1 || ab == 2) ? AR::neg(y) : y;
            }
        if (t < 2 * (16 * T.ksteps - nv)) {  // columns beyond 4 nn^2
          const int pad = 16 * T.ksteps - nv;
          Xs[(t / pad) * 16 * T.ksteps + nv + t % pad] = V{};
        }
        __syncthreads();
        for (int ch = t; ch < 2 * nv8; ch += blockDim.x) {
          const int w2 = ch / nv8, v8 = ch % nv8, jj = j2 + w2;
          if (jj >= nj || s_unit[jj] < 0) continue;
          uint32_t pk[NX][4];
          int E;
          if constexpr (F64) {
            E = (int)max(s_eb[jj], 64u) - 1022;  // (64: a zero's significand is shifted out)
            double xv[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) xv[j] = Xs[w2 * 16 * T.ksteps + 8 * v8 + j];
            digits512_fixed(xv, E, pk);
            E = s_eb[jj] == 0x7FFu ? kBadExp : E + 2;
          } else {
            E = max((int)max(s_eb[jj], 1u) - 126, -100);
            const float s27 = exp2i(27 - E);
            if (s_eb[jj] == 0xFFu) E = kBadExp;
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              float d0[XD], d1[XD];
              digits512(Xs[w2 * 16 * T.ksteps + 8 * v8 + j], s27, d0);
              digits512(Xs[w2 * 16 * T.ksteps + 8 * v8 + j + 1], s27, d1);
#pragma unroll
              for (int kk = 0; kk < XD; ++kk) pk[kk][j / 2] = pack_f16(d0[kk], d1[kk]);
            }
          }
          unsigned char* o = T.x + (((size_t)s_unit[jj] * D.nlm + ilm) * T.ksteps + (v8 >> 1)) * NX * APL +
                             tc::off_kmajor(s_row[jj], 8 * (v8 & 1));
#pragma unroll
          for (int kk = 0; kk < NX; ++kk)
            *reinterpret_cast<uint4*>(o + kk * APL) = make_uint4(pk[kk][0], pk[kk][1], pk[kk][2], pk[kk][3]);
          if (v8 == 0) T.xexp[((size_t)s_unit[jj] * D.nlm + ilm) * 128 + s_row[jj]] = E;
        }
      }
    }
  }
}

// ---- the products: CTA = (unit, tile of TT entries t, part of the
// multipoles); warps 0-7 read back, warp 8 copies, warp 9 issues ----
template <bool F64>
__global__ void __launch_bounds__(320, 1) dk_tc_gemm(DevDiatomic D, DevDiatomicScratch S, DevDiaTC T, int symmetric,
                                                     int u0) {
  constexpr int NX = F64 ? TD : XD;
  const Blocks B = blocks_of(D, S, symmetric);
  const int tt = blockIdx.x % T.ntt, lp = (blockIdx.x / T.ntt) % T.lparts, lu = blockIdx.x / (T.ntt * T.lparts);
  const int u = u0 + lu;
  if (u >= D.nel * B.ntile) return;  // uniform over the CTA
  const int e = u / B.ntile;
  extern __shared__ __align__(1024) unsigned char smg[];
  unsigned char* Abuf = smg;                                        // NSTAGE x NX planes of 128 x 16
  unsigned char* Bbuf = Abuf + NSTAGE * NX * APL;                     // NSTAGE x TD planes of TT x 16
  uint64_t* full = reinterpret_cast<uint64_t*>(Bbuf + NSTAGE * TD * BPL);
  uint64_t* empty = full + NSTAGE;
  uint64_t* done = empty + NSTAGE;
  uint64_t* fre = done + 1;
  uint64_t* drain = fre + 1;  // every product finished (of a CTA that gives up)
  uint32_t* tslot = reinterpret_cast<uint32_t*>(drain + 1);
  int* fail = reinterpret_cast<int*>(tslot + 1);
  int* nact = fail + 1;
  int* act = nact + 1;  // [nlm] multipoles with a row in this tile
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int l0 = (int)((long)D.nlm * lp / T.lparts), l1 = (int)((long)D.nlm * (lp + 1) / T.lparts);
  for (int ilm = l0 + warp; ilm < l1; ilm += 10) {
    const int* x = T.xexp + ((size_t)lu * D.nlm + ilm) * 128;
    bool any = false;
    for (int r = lane; r < 128; r += 32) any |= x[r] != kNoRow;
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) act[ilm - l0] = any ? 1 : 0;
  }
  if (warp == 9) {
    tc::tmem_alloc(tslot, 512);
    tc::tmem_relinquish();
  }
  if (t == 0) {
    for (int i = 0; i < NSTAGE; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], 1);
    }
    tc::mbar_init(done, 1);
    tc::mbar_init(fre, 8);
    tc::mbar_init(drain, 1);
    fail[0] = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  if (t == 0) {
    int n = 0;
    for (int i = 0; i < l1 - l0; ++i)
      if (act[i]) act[n++] = l0 + i;
    nact[0] = n;
  }
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tD = *tslot;
  const int na = nact[0];
  double acc[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) acc[j] = 0.0;

  bool bad = false;  // this row's tile has a value that is not finite
  int copied = 0;  // K steps whose copies were started (by the copying thread)
  if (warp == 8) {
    if (lane == 0) {
      bool ok = true;
      int& it = copied;
      for (int a = 0; a < na && ok; ++a) {
        const unsigned char* xs = T.x + ((size_t)lu * D.nlm + act[a]) * T.ksteps * NX * APL;
        const unsigned char* ts = T.tx + (((size_t)act[a] * D.nel + e) * T.ntt + tt) * T.ksteps * TD * BPL;
        for (int ks = 0; ks < T.ksteps; ++ks, ++it) {
          const int s = it % NSTAGE;
          if (it >= NSTAGE && !tc::mbar_wait(&empty[s], (uint32_t)((it / NSTAGE - 1) & 1), T.wait)) {
            ok = false;
            break;
          }
          tc::mbar_expect_tx(&full[s], NX * APL + TD * BPL);
          tc::bulk_g2s(Abuf + s * NX * APL, xs + (size_t)ks * NX * APL, NX * APL, &full[s]);
          tc::bulk_g2s(Bbuf + s * TD * BPL, ts + (size_t)ks * TD * BPL, TD * BPL, &full[s]);
        }
      }
      if (!ok) atomicExch(fail, 1);
    }
  } else if (warp == 9) {
    if (lane == 0) {
      bool ok = true;
      int it = 0;
      for (int a = 0; a < na && ok; ++a) {
        // the sums of the previous multipole have been read back
        if (a > 0 && !tc::mbar_wait(fre, (uint32_t)((a - 1) & 1), T.wait)) { ok = false; break; }
        tc::fence_after_sync();
        for (int ks = 0; ks < T.ksteps; ++ks, ++it) {
          const int s = it % NSTAGE;
          if (!tc::mbar_wait(&full[s], (uint32_t)((it / NSTAGE) & 1), T.wait)) { ok = false; break; }
          tc::fence_after_sync();
          const uint64_t da = tc::smem_desc(tc::smem_u32(Abuf + s * NX * APL));
          const uint64_t db = tc::smem_desc(tc::smem_u32(Bbuf + s * TD * BPL));
          // digit kx of the tiles against the table digits 0..6-kx, which are
          // consecutive: levels kx.. at columns TT kx.. (at most 256 per MMA)
#pragma unroll 1
          for (int kx = 0; kx < NX; ++kx) {
            const int n = TT * (TD - kx);
            const uint64_t ad = da + (uint64_t)(kx * APL >> 4);
            const uint32_t on = (ks > 0 || kx > 0) ? 1u : 0u;
            const int n0 = n > 256 ? 256 : n;
            tc::mma_bf16(tD + TT * kx, ad, db, tc::idesc_f16(128, n0, 0, 0), on);
            if (n > 256)
              tc::mma_bf16(tD + TT * kx + 256, ad, db + (uint64_t)(256 / TT * BPL >> 4),
                           tc::idesc_f16(128, n - 256, 0, 0), on);
          }
          tc::mma_commit(&empty[s]);
        }
        if (ok) tc::mma_commit(done);
      }
      if (!ok) atomicExch(fail, 1);
    }
  } else {
    const int qw = warp & 3, half = warp >> 2, row = 32 * qw + lane;
    const uint32_t col0 = tD + ((uint32_t)(32 * qw) << 16) + 32 * half;
    for (int a = 0; a < na; ++a) {
      const int ilm = act[a];
      const int E = T.xexp[((size_t)lu * D.nlm + ilm) * 128 + row];
      bad |= E == kBadExp;
      const int* te = T.txexp + (((size_t)ilm * D.nel + e) * T.ntt + tt) * TT + 32 * half;
      const bool ok = tc::mbar_wait(done, (uint32_t)(a & 1), T.wait);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(fail, 1);
        break;
      }
      tc::fence_after_sync();
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        float v[TD][8];
        ld_levels(col0 + 8 * g, v);
        if (E != kNoRow && E != kBadExp) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float lv[TD];
#pragma unroll
            for (int d = 0; d < TD; ++d) lv[d] = v[d][j];
            if constexpr (F64) {
              acc[8 * g + j] += levels512_f64(lv, te[8 * g + j] + E);
            } else {
              float z0, z1, z2;
              levels512(lv, z0, z1, z2);
              const int c = (max(te[8 * g + j] + E, -800) + 896) << 20;
              acc[8 * g + j] += f2d_scaled(z0, c);
              acc[8 * g + j] += f2d_scaled(z1, c);
              acc[8 * g + j] += f2d_scaled(z2, c);
            }
          }
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(fre);
    }
  }
  __syncthreads();
  if (warp < 8) {
    const int row = 32 * (warp & 3) + lane, half = warp >> 2;
    bad |= fail[0] != 0;
    double* o = T.part + ((((size_t)lp * T.cap + lu) * T.ntt + tt) * TT + 32 * half) * 128 + row;
#pragma unroll
    for (int j = 0; j < 32; ++j)
      o[(size_t)j * 128] = bad ? __longlong_as_double(0x7ff8000000000000ll) : acc[j];
  }
  // the copies in flight must land before the CTA leaves
  if (fail[0] && copied > 0)
    for (int i = max(0, copied - NSTAGE); i < copied; ++i)
      tc::mbar_wait(&full[i % NSTAGE], (uint32_t)((i / NSTAGE) & 1), kWait);
  if (warp == 9 && lane == 0 && fail[0]) {
    atomicExch(T.err, 1);
    // products may still be running: the tensor memory is released after them
    tc::mma_commit(drain);
    tc::mbar_wait(drain, 0, kWait);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 9) tc::tmem_dealloc(tD, 512);
}

// ---- the parts of every tile entry summed in order and written to K (and
// to the transposed partner of a symmetric density); grid (units, parts of the tile) ----
__global__ void dk_tc_store(DevDiatomic D, DevDiatomicScratch S, DevDiaTC T, int symmetric, int u0,
                            double* __restrict__ Kd) {
  const Blocks B = blocks_of(D, S, symmetric);
  const int lu = blockIdx.x, u = u0 + lu;
  if (u >= D.nel * B.ntile) return;
  const int e = u / B.ntile, tile = u % B.ntile, n2 = D.nn * D.nn;
  for (int idx = blockIdx.y * blockDim.x + threadIdx.x; idx < n2 * 128; idx += gridDim.y * blockDim.x) {
    const int row = idx % 128, t = idx / 128, pos = tile * 128 + row;
    if (pos >= B.count) continue;
    double s = 0.0;
#pragma unroll 8
    for (int lp = 0; lp < T.lparts; ++lp) s += T.part[((((size_t)lp * T.cap + lu) * T.ntt) * TT + t) * 128 + row];
    const int jk = B.list[pos], j = jk % D.nang, k = jk / D.nang, p = t % D.nn, q = t / D.nn;
    share_store(D, S, Kd, e, e, jk, p, q, -s);
    if (symmetric && j != k) share_store(D, S, Kd, e, e, k + j * D.nang, q, p, -s);
  }
}

cudaError_t launch_dk_tc_table(const DevDiatomic& D, const DevDiaTC& T, unsigned char* tx, int* txexp, int* cexp,
                               cudaStream_t st) {
  dk_tc_colexp<<<D.nlm * D.nel, 256, 0, st>>>(D, cexp);
  dk_tc_table<<<dim3(T.ntt, D.nlm * D.nel), 4 * TT, 0, st>>>(D, T, tx, txexp);
  return cudaGetLastError();
}

static size_t dtc_gemm_smem(const DevDiatomic& D, bool f64) {
  return (size_t)NSTAGE * ((f64 ? TD : XD) * APL + TD * BPL) + 8 * (2 * NSTAGE + 3) + 4 * (4 + (size_t)D.nlm);
}

// Pd: the FP64 form (from the density itself), nullptr: the split form (S.pd2)
cudaError_t launch_dk_tc_diag(const DevDiatomic& D, const DevDiatomicScratch& S, const DevDiaTC& T, const double* Pd,
                              double* Kd, bool symmetric, bool itemwise, cudaStream_t st) {
  const int n2 = D.nn * D.nn, th = ((n2 + 31) / 32) * 32;
  int dev = 0, nsm = 152, per = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  auto xk = Pd ? (D.nn == 15 ? dk_tc_x<15, true> : dk_tc_x<0, true>)
               : (D.nn == 15 ? dk_tc_x<15, false> : dk_tc_x<0, false>);
  auto gk = Pd ? dk_tc_gemm<true> : dk_tc_gemm<false>;
  const size_t xsm = sizeof(Chunk<ArF, JC_DIAG>) + sizeof(float2) * 2 * 16 * (size_t)T.ksteps;
  cudaError_t e = smem_limit(xk, xsm);
  if (e != cudaSuccess) return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, xk, th, xsm);
  if (e != cudaSuccess) return e;
  const size_t gsm = dtc_gemm_smem(D, Pd != nullptr);
  if ((e = smem_limit(gk, gsm)) != cudaSuccess) return e;
  const int slots = nsm * std::max(per, 1);
  const long nblk = symmetric ? (long)D.nang * (D.nang + 1) / 2 : (long)D.nang * D.nang;
  const int units = (int)(D.nel * ((nblk + 127) / 128));
  // multipoles in parts where there are few (element, k) items: parts share
  // nothing, so the count follows the items alone
  const int items = D.nel * D.nang;
  const int nchunk = std::max(1, std::min(D.nlm, (4 * slots + items - 1) / items));
  for (int u0 = 0; u0 < units; u0 += T.cap) {
    e = cudaMemsetAsync(T.xexp, 0x80, sizeof(int) * (size_t)T.cap * D.nlm * 128, st);
    if (e != cudaSuccess) return e;
    xk<<<slots, th, xsm, st>>>(D, S, T, Pd, symmetric ? 1 : 0, itemwise ? 1 : 0, u0, nchunk);
    const int nu = std::min(T.cap, units - u0);
    gk<<<nu * T.ntt * T.lparts, 320, gsm, st>>>(D, S, T, symmetric ? 1 : 0, u0);
    dk_tc_store<<<dim3(nu, 64), 256, 0, st>>>(D, S, T, symmetric ? 1 : 0, u0, Kd);
  }
  return cudaGetLastError();
}

}  // namespace hfg
