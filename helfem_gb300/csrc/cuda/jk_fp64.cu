// Plain-FP64 Coulomb (J) and exchange (K) builds for the atomic FE basis.
//
// J restates TwoDBasisT::coulomb (src/atomic/TwoDBasis.cpp:773-877) with the
// per-multipole FE assembly of assemble_J_FE_one_multipole_cached_chol
// (libhelfemqc/include/CoulombExchangeFE.h:432-482):
//   j_contract : per (L,M) channel and element, the Gaunt-weighted ket
//                contraction restricted to the element-diagonal tile (the only
//                part of Paux the assembly reads), the two disjoint traces
//                and the in-element Cholesky contraction L (L^T vec P).
//   j_scatter  : per output angular block and element, the O(Nel) prefix
//                sums of the disjoint traces (the reference's O(Nel^2) double
//                loop) and the Gaunt-weighted bra scatter.
// K restates TwoDBasisT::exchange (TwoDBasis.cpp:879-999) with
// assemble_K_FE_one_multipole_cached_chol (CoulombExchangeFE.h:484-530):
//   k_block_norms : density-block screening, ||P_il||_F < 10 eps skipped, and
//                   the split copy of the density.
//   k_tiles       : work units of (element pair, range of output angular
//                   blocks). Off-diagonal pairs: recouple the (a,b) tiles of
//                   P, then A_L X B_L^T with A/B = r_small/r_big by element
//                   order. Diagonal elements: the exchange-ordered
//                   in-element tensor (equal to sum_p M_p X M_p^T). With a
//                   symmetric density only half of the tiles are computed and
//                   each is also written transposed (K_kj(b,a) = K_jk(a,b)^T).
//   k_fixup       : adds the contributions of neighbouring tiles on the
//                   shared boundary functions, in a fixed order (no atomics,
//                   bitwise reproducible).
#include <algorithm>
#include <cfloat>

#include "devatom.cuh"
#include "ff.cuh"
#include "smem_limit.hpp"

namespace hfg {
namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-wide sum, result valid in every thread; red needs >= 32 doubles
__device__ double block_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  for (int i = 0; i < nw; ++i) s += red[i];
  return s;
}

__device__ __forceinline__ bool gvalid(const DevAtom& A, int g) { return g >= 0 && g < A.nrad; }

// ------------------------------------------------------------------ Coulomb
__global__ void j_contract(DevAtom A, DevScratch S, const double* __restrict__ P) {
  const int ch = blockIdx.x, e = blockIdx.y;
  const int nn = A.nn, n2 = nn * nn, L = A.chanL[ch];
  extern __shared__ double sm[];
  double* X = sm;
  double* sc = X + n2;
  double* red = sc + A.rmax;
  const int k0 = A.jket_ptr[ch], k1 = A.jket_ptr[ch + 1];
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int p = idx % nn, q = idx / nn;
    const int gp = gfun(A, e, p), gq = gfun(A, e, q);
    double x = 0.0;
    if (gvalid(A, gp) && gvalid(A, gq))
      for (int u = k0; u < k1; ++u) {
        const int blk = A.jket_blk[u], k = blk % A.nang, l = blk / A.nang;
        x += A.jket_coef[u] * P[(size_t)(l * A.nrad + gq) * A.nbf + (size_t)k * A.nrad + gp];
      }
    X[idx] = x;
  }
  __syncthreads();
  const size_t le = (size_t)L * A.nel + e;
  const double* rs = A.rs + le * n2;
  const double* rb = A.rb + le * n2;
  double ts = 0.0, tb = 0.0;
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int p = idx % nn, q = idx / nn;
    const double xt = X[q + p * nn];
    ts += rs[idx] * xt;
    tb += rb[idx] * xt;
  }
  ts = block_sum(ts, red);
  tb = block_sum(tb, red);
  if (threadIdx.x == 0) {
    S.jscal[((size_t)ch * A.nel + e) * 2 + 0] = ts;
    S.jscal[((size_t)ch * A.nel + e) * 2 + 1] = tb;
  }
  const int r = A.rank[le];
  const double* C = A.cholp + le * n2 * A.rmax;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  for (int j = w; j < r; j += nw) {
    double s = 0.0;
    for (int q = lane; q < n2; q += 32) s += C[q + (size_t)j * n2] * X[q];
    s = warp_sum(s);
    if (lane == 0) sc[j] = s;
  }
  __syncthreads();
  double* jin = S.jin + ((size_t)ch * A.nel + e) * n2;
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    double s = 0.0;
    for (int j = 0; j < r; ++j) s += C[idx + (size_t)j * n2] * sc[j];
    jin[idx] = s;
  }
}

constexpr int JMAXTERMS = 64;

// ---- Coulomb, split form: the contraction above in float pairs (the FP64
// pipe bounds the FP64 form on GB300: 2 n2 r multiply-adds per channel and
// element for the in-element factor alone). The density is split with
// integer operations, the in-element factor and the radial tables come as
// float-pair copies, sums of n2 or r terms are renormalised every step; the
// in-element part goes to the scratch as float pairs, the two scalars per
// (channel, element) as FP64.
__device__ __forceinline__ ffv ff_warp_sum(ffv v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = ff_add(v, ffv{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
  return v;
}

// block-wide float-pair sum, valid in thread 0; red needs >= 32 entries
__device__ ffv ff_block_sum(ffv v, ffv* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = ff_warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  ffv s{0.f, 0.f};
  if (threadIdx.x == 0)
    for (int i = 0; i < nw; ++i) s = ff_add(s, red[i]);
  return s;
}

__global__ void j_contract_split(DevAtom A, DevScratch S, const double* __restrict__ P,
                                 const float2* __restrict__ C2) {
  const int ch = blockIdx.x, e = blockIdx.y;
  const int nn = A.nn, n2 = nn * nn, L = A.chanL[ch];
  extern __shared__ float2 smf[];
  float2* X = smf;       // [n2]
  float2* sc = X + n2;   // [rmax]
  __shared__ ffv red[32];
  const int k0 = A.jket_ptr[ch], k1 = A.jket_ptr[ch + 1];
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int p = idx % nn, q = idx / nn;
    const int gp = gfun(A, e, p), gq = gfun(A, e, q);
    ffv x{0.f, 0.f};
    if (gvalid(A, gp) && gvalid(A, gq))
      for (int u = k0; u < k1; ++u) {
        const int blk = A.jket_blk[u], k = blk % A.nang, l = blk / A.nang;
        x = ff_fma(x, A.jket_coef2[u], split_bits(P[(size_t)(l * A.nrad + gq) * A.nbf + (size_t)k * A.nrad + gp]));
      }
    X[idx] = ff2(x);
  }
  __syncthreads();
  const size_t le = (size_t)L * A.nel + e;
  const float2* rs = A.rs2 + le * n2;
  const float2* rb = A.rb2 + le * n2;
  ffv ts{0.f, 0.f}, tb{0.f, 0.f};
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int p = idx % nn, q = idx / nn;
    const float2 xt = X[q + p * nn];
    ts = ff_fma_n(ts, rs[idx], xt);
    tb = ff_fma_n(tb, rb[idx], xt);
  }
  ts = ff_block_sum(ts, red);
  tb = ff_block_sum(tb, red);
  if (threadIdx.x == 0) {
    S.jscal[((size_t)ch * A.nel + e) * 2 + 0] = ff_to_d(ts);
    S.jscal[((size_t)ch * A.nel + e) * 2 + 1] = ff_to_d(tb);
  }
  const int r = A.rank[le];
  const float2* C = C2 + le * n2 * A.rmax;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  for (int j = w; j < r; j += nw) {
    ffv v{0.f, 0.f};
    for (int q = lane; q < n2; q += 32) v = ff_fma_n(v, C[q + (size_t)j * n2], X[q]);
    v = ff_warp_sum(v);
    if (lane == 0) sc[j] = make_float2(v.hi, v.lo);
  }
  __syncthreads();
  float2* jin = reinterpret_cast<float2*>(S.jin) + ((size_t)ch * A.nel + e) * n2;
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    ffv v{0.f, 0.f};
    for (int j = 0; j < r; ++j) v = ff_fma_n(v, C[idx + (size_t)j * n2], sc[j]);
    jin[idx] = ff2(v);
  }
}

__global__ void j_scatter_split(DevAtom A, DevScratch S, double* __restrict__ J, int accumulate) {
  const int ij = blockIdx.x, e = blockIdx.y;
  const int i = ij % A.nang, j = ij / A.nang;
  const int b0 = A.jbra_ptr[ij], b1 = A.jbra_ptr[ij + 1];
  const int nt = b1 - b0;
  if (nt == 0) return;
  const int nn = A.nn, n2 = nn * nn;
  __shared__ float2 Ab[JMAXTERMS], As[JMAXTERMS], Ab1[JMAXTERMS], As1[JMAXTERMS];
  for (int u = threadIdx.x; u < nt; u += blockDim.x) {
    const int ch = A.jbra_chan[b0 + u];
    const double* sc = S.jscal + (size_t)ch * A.nel * 2;
    double big = 0.0, small = 0.0;
    for (int e2 = e + 1; e2 < A.nel; ++e2) big += sc[2 * e2 + 1];
    for (int e2 = 0; e2 < e; ++e2) small += sc[2 * e2 + 0];
    Ab[u] = split_bits(big);
    As[u] = split_bits(small);
    if (e > 0) {
      Ab1[u] = split_bits(big + sc[2 * e + 1]);
      As1[u] = split_bits(small - sc[2 * (e - 1) + 0]);
    }
  }
  __syncthreads();
  const float2* jin2 = reinterpret_cast<const float2*>(S.jin);
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int p = idx % nn, q = idx / nn;
    // J has element-diagonal tiles only: the single entry two tiles share is
    // the corner on the common boundary function, owned by the later tile
    if (p == nn - 1 && q == nn - 1) continue;
    const int gp = gfun(A, e, p), gq = gfun(A, e, q);
    if (!gvalid(A, gp) || !gvalid(A, gq)) continue;
    ffv v{0.f, 0.f};
    for (int u = 0; u < nt; ++u) {
      const int ch = A.jbra_chan[b0 + u], L = A.chanL[ch];
      const size_t le = (size_t)L * A.nel + e;
      ffv t{0.f, 0.f};
      t = ff_fma(t, Ab[u], A.rs2[le * n2 + idx]);
      t = ff_fma(t, As[u], A.rb2[le * n2 + idx]);
      const float2 ji = jin2[((size_t)ch * A.nel + e) * n2 + idx];
      t = ff_add(t, ffv{ji.x, ji.y});
      v = ff_fma_n(v, A.jbra_coef2[b0 + u], ff2(t));
    }
    if (p == 0 && q == 0 && e > 0) {
      const int c = (nn - 1) + (nn - 1) * nn;
      for (int u = 0; u < nt; ++u) {
        const int ch = A.jbra_chan[b0 + u], L = A.chanL[ch];
        const size_t le = (size_t)L * A.nel + (e - 1);
        ffv t{0.f, 0.f};
        t = ff_fma(t, Ab1[u], A.rs2[le * n2 + c]);
        t = ff_fma(t, As1[u], A.rb2[le * n2 + c]);
        const float2 ji = jin2[((size_t)ch * A.nel + (e - 1)) * n2 + c];
        t = ff_add(t, ffv{ji.x, ji.y});
        v = ff_fma_n(v, A.jbra_coef2[b0 + u], ff2(t));
      }
    }
    double* out = J + (size_t)(j * A.nrad + gq) * A.nbf + (size_t)i * A.nrad + gp;
    const double y = ff_to_d(v);
    if (accumulate) *out += y; else *out = y;
  }
}

__global__ void j_scatter(DevAtom A, DevScratch S, double* __restrict__ J, int accumulate) {
  const int ij = blockIdx.x, e = blockIdx.y;
  const int i = ij % A.nang, j = ij / A.nang;
  const int b0 = A.jbra_ptr[ij], b1 = A.jbra_ptr[ij + 1];
  const int nt = b1 - b0;
  if (nt == 0) return;
  const int nn = A.nn, n2 = nn * nn;
  __shared__ double Ab[JMAXTERMS], As[JMAXTERMS], Ab1[JMAXTERMS], As1[JMAXTERMS];
  for (int u = threadIdx.x; u < nt; u += blockDim.x) {
    const int ch = A.jbra_chan[b0 + u];
    const double* sc = S.jscal + (size_t)ch * A.nel * 2;
    double big = 0.0, small = 0.0;
    for (int e2 = e + 1; e2 < A.nel; ++e2) big += sc[2 * e2 + 1];
    for (int e2 = 0; e2 < e; ++e2) small += sc[2 * e2 + 0];
    Ab[u] = big;
    As[u] = small;
    if (e > 0) {
      Ab1[u] = big + sc[2 * e + 1];
      As1[u] = small - sc[2 * (e - 1) + 0];
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < n2; idx += blockDim.x) {
    const int p = idx % nn, q = idx / nn;
    // J has element-diagonal tiles only: the single entry two tiles share is
    // the corner on the common boundary function, owned by the later tile
    if (p == nn - 1 && q == nn - 1) continue;
    const int gp = gfun(A, e, p), gq = gfun(A, e, q);
    if (!gvalid(A, gp) || !gvalid(A, gq)) continue;
    double v = 0.0;
    for (int u = 0; u < nt; ++u) {
      const int ch = A.jbra_chan[b0 + u], L = A.chanL[ch];
      const size_t le = (size_t)L * A.nel + e;
      const double* jin = S.jin + ((size_t)ch * A.nel + e) * n2;
      v += A.jbra_coef[b0 + u] * (Ab[u] * A.rs[le * n2 + idx] + As[u] * A.rb[le * n2 + idx] + jin[idx]);
    }
    if (p == 0 && q == 0 && e > 0) {
      const int c = (nn - 1) + (nn - 1) * nn;
      for (int u = 0; u < nt; ++u) {
        const int ch = A.jbra_chan[b0 + u], L = A.chanL[ch];
        const size_t le = (size_t)L * A.nel + (e - 1);
        const double* jin = S.jin + ((size_t)ch * A.nel + (e - 1)) * n2;
        v += A.jbra_coef[b0 + u] * (Ab1[u] * A.rs[le * n2 + c] + As1[u] * A.rb[le * n2 + c] + jin[c]);
      }
    }
    double* out = J + (size_t)(j * A.nrad + gq) * A.nbf + (size_t)i * A.nrad + gp;
    if (accumulate) *out += v; else *out = v;
  }
}

// ----------------------------------------------------------------- exchange
// Density pass, grid (nang^2, nel), thread = row: the columns of one element of
// one angular block. Squared norms of the columns that the element owns (the
// shared last one is the next element's), and in the split form (p2) the
// float-pair copy and the largest high word of every density tile of the
// element's columns. The last CTA adds the norms up in a fixed order, applies
// the reference's 10*DBL_EPSILON screen and marks the exchange entries that
// see an active block (its own launch took 6 us for Kr and 30 us for l <= 3,
// every entry summing its blocks' partial norms again).
// Bound by HBM (202 MB read, 202 MB written for Kr in the split form, 320 and
// 320 MB for the l <= 3 atom of 33 elements); up to eight loads in flight per
// thread. With the flags 82 us (Kr) and 144 us; without the last CTA's part 75
// and 117 us; the norms without the tiles' maxima plus the flags' own launch
// took 90 and 137 us.
// NORM_PLAIN: norms and flags; NORM_COPY: with the float-pair copy; NORM_SPLIT:
// with the copy and what the tensor-core form needs (the tiles' maxima, the
// lists); NORM_LISTS: the latter for an FP64 density (maxima as the high words of
// the doubles)
// entries: the last CTA marks the exchange entries too; otherwise (their flags
// do not fit its shared memory) k_flags does.
enum { NORM_PLAIN, NORM_COPY, NORM_SPLIT, NORM_LISTS };
template <int MODE>
__global__ void k_block_norms(DevAtom A, DevScratch S, const double* __restrict__ P, float2* __restrict__ p2,
                              int symmetric, int entries) {
  constexpr bool SPLIT = MODE == NORM_COPY || MODE == NORM_SPLIT, LISTS = MODE == NORM_SPLIT || MODE == NORM_LISTS;
  __shared__ double red[32];
  __shared__ bool last;
  __shared__ int cnt[64];
  extern __shared__ unsigned int emax[];  // [nel] (list forms); flags of the last CTA
  const int blk = blockIdx.x, i = blk % A.nang, l = blk / A.nang, b = blockIdx.y, nn = A.nn;
  const int c0 = max(gfun(A, b, 0), 0), c1 = min(gfun(A, b, nn - 1), A.nrad - 1);
  const int nc = c1 - c0 + 1, nown = b == A.nel - 1 ? nc : nc - 1;  // columns, those owned
  if (LISTS) {
    for (int e = threadIdx.x; e < A.nel; e += blockDim.x) emax[e] = 0u;
    __syncthreads();
  }
  double s = 0.0;
  float sf = 0.f;
  const size_t base = (size_t)l * A.nrad * A.nbf + (size_t)i * A.nrad + (size_t)c0 * A.nbf;
  constexpr int NU = 8;  // loads in flight: the columns in equal passes of at most that many
  const int nu = (nown + (nown + NU - 1) / NU - 1) / ((nown + NU - 1) / NU);
  for (int r = threadIdx.x; r < A.nrad; r += blockDim.x) {
    unsigned int mx = 0u;
    const double* p = P + base + r;
    float2* q = SPLIT ? p2 + base + r : nullptr;
    auto add = [&](double v) {
      if (SPLIT) {
        // integer-only split (no FP64-pipe instructions) and an FP32 norm of
        // the high words for the screen
        const float2 h = split_bits(v);
        mx = max(mx, __float_as_uint(h.x) & 0x7FFFFFFFu);
        *q = h;
        q += A.nbf;
        sf = fmaf(h.x, h.x, sf);
      } else {
        if (LISTS) mx = max(mx, (unsigned)__double2hiint(v) & 0x7FFFFFFFu);
        s += v * v;
      }
    };
    const double vb = LISTS && nown < nc ? p[(size_t)nown * A.nbf] : 0.0;  // the next element's first column
    for (int c = 0; c < nown; c += nu) {
      const int len = min(nu, nown - c);
      double v[NU];
#pragma unroll
      for (int w = 0; w < NU; ++w)
        if (w < len) v[w] = p[(size_t)w * A.nbf];
#pragma unroll
      for (int w = 0; w < NU; ++w)
        if (w < len) add(v[w]);
      p += (size_t)nu * A.nbf;
    }
    if (LISTS) mx = max(mx, (SPLIT ? __float_as_uint(split_bits(vb).x) : (unsigned)__double2hiint(vb)) & 0x7FFFFFFFu);
    if (LISTS) {
      // row r is function r + 1 - a (nn - 1) of element a, and the last of the one before
      const int a = (r + 1) / (nn - 1), f = (r + 1) - a * (nn - 1);
      if (a < A.nel) atomicMax(&emax[a], mx);
      if (a > 0 && f == 0) atomicMax(&emax[a - 1], mx);
    }
  }
  if (SPLIT) {  // float sums by warp, in a fixed order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sf += __shfl_xor_sync(0xffffffffu, sf, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = (double)sf;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int v = 0; v < (int)blockDim.x >> 5; ++v) s += red[v];
  } else {
    s = block_sum(s, red);
  }
  if (LISTS)  // (both sums end after a barrier)
    for (int e = threadIdx.x; e < A.nel; e += blockDim.x) S.tmax[((size_t)blk * A.nel + e) * A.nel + b] = emax[e];
  // ---- the last CTA: flags (bnorm alone is read here: the copy and the
  // maxima are the next kernels' and need no fence) ----
  const int nang2 = A.nang * A.nang;
  if (threadIdx.x == 0) {
    S.bnorm[(size_t)b * nang2 + blk] = s;
    __threadfence();
    last = atomicAdd(S.count, 1u) == gridDim.x * gridDim.y - 1;
    if (last) __threadfence();
  }
  __syncthreads();
  if (!last) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // (dynamic shared memory past emax: block, entry and output-block flags)
  unsigned char* sact = reinterpret_cast<unsigned char*>(emax + (LISTS ? A.nel + nang2 : 0));
  unsigned char* sent = sact + nang2;
  int* sout = reinterpret_cast<int*>(emax) + A.nel;  // multipoles of a block's active entries (bits)
  for (int x = threadIdx.x; x < nang2; x += blockDim.x) {
    double q = 0.0;
#pragma unroll 16
    for (int e = 0; e < A.nel; ++e) q += __ldcg(&S.bnorm[(size_t)e * nang2 + x]);
    const unsigned char f = !(sqrt(q) < 10.0 * DBL_EPSILON);
    if (entries) sact[x] = f;
    S.act[x] = f;
  }
  if (threadIdx.x == 0) *S.count = 0u;  // for the next call
  if (!entries) return;
  __syncthreads();
  // entries: every term marks its entry. (One CTA alone: each loop loads a
  // batch before it stores, or the latencies of its loads add up.)
  for (int ent = threadIdx.x; ent < A.nent; ent += blockDim.x) sent[ent] = 0;
  __syncthreads();
  constexpr int NB = 8;
  const int nterm = A.kent_ptr[A.nent], step = blockDim.x;
  for (int u0 = threadIdx.x; u0 < nterm; u0 += NB * step) {
    int blk[NB], ent[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int u = min(u0 + i * step, nterm - 1);
      blk[i] = A.kterm_blk[u];
      ent[i] = A.kterm_ent[u];
    }
#pragma unroll
    for (int i = 0; i < NB; ++i)
      if (sact[blk[i]]) sent[ent[i]] = 1;
  }
  if (LISTS)
    for (int x = threadIdx.x; x < nang2; x += step) sout[x] = 0;
  __syncthreads();
  for (int e0 = threadIdx.x; e0 < A.nent; e0 += NB * step) {
    int sig[NB];
    if (LISTS)
#pragma unroll
      for (int i = 0; i < NB; ++i) sig[i] = A.kent_sig[min(e0 + i * step, A.nent - 1)];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int e = e0 + i * step;
      if (e >= A.nent) break;
      S.ent_act[e] = sent[e];
      if (LISTS && sent[e]) atomicOr(&sout[sig[i] & 0xFFFFFF], 1 << (sig[i] >> 24));
    }
  }
  if (!LISTS) return;
  // ---- list forms: the active output blocks in jk_order. A symmetric
  // density's transposed partner tile is written too: (j, k) counts as active
  // where (k, j) is ----
  for (int x = threadIdx.x; x < 64; x += blockDim.x) cnt[x] = 0;
  __syncthreads();
  // positions: warps count their parts of the order, then place them
  const int part = ((nang2 + nw - 1) / nw + 31) / 32 * 32;
  for (int pass = 0; pass < 2; ++pass) {
    int n = 0, nh = 0;
    if (pass) {
      for (int v = 0; v < w; ++v) n += cnt[v], nh += cnt[32 + v];
    }
    for (int x0 = w * part; x0 < min((w + 1) * part, nang2); x0 += 32) {
      const int x = x0 + lane;
      const int4 info = x < nang2 ? A.jk_order[x] : make_int4(0, 0, 0, 0);
      const int jk = info.x, j = info.w & 0xFFFF, k = info.w >> 16;
      const bool on = x < nang2 && (sout[jk] || (symmetric && sout[k + j * A.nang])), half = on && j <= k;
      const unsigned mo = __ballot_sync(0xffffffffu, on), mh = __ballot_sync(0xffffffffu, half);
      const unsigned below = (1u << lane) - 1u;
      if (pass && on) {
        S.olist[n + __popc(mo & below)] = jk;
        S.oinfo[n + __popc(mo & below)] = info;
      }
      if (pass && half) S.olist[nang2 + nh + __popc(mh & below)] = jk;
      if (pass && x < nang2) S.jk_on[jk] = on;
      n += __popc(mo);
      nh += __popc(mh);
    }
    if (!pass && lane == 0) {
      cnt[w] = n;
      cnt[32 + w] = nh;
    }
    __syncthreads();
  }
  int n = 0, nh = 0;
  for (int v = 0; v < nw; ++v) n += cnt[v], nh += cnt[32 + v];
  if (threadIdx.x == 0) {
    S.ocount[0] = n;
    S.ocount[1] = nh;
  }
  for (int g = threadIdx.x; g < (n + 7) / 8; g += blockDim.x) {
    int m = 0;
#pragma unroll
    for (int x = 8 * g; x < 8 * g + 8; ++x)
      if (x < n) m |= sout[S.olist[x]];
    S.gmask[g] = m ? m : 1;
  }
}

// K of the output blocks without an active entry (the tensor-core tiles run
// over the active ones alone); grid (nang^2, column bands)
__global__ void k_zero_inactive(DevAtom A, DevScratch S, double* __restrict__ K, int symmetric) {
  __shared__ int on;
  const int jk = blockIdx.x, j = jk % A.nang, k = jk / A.nang, kj = k + j * A.nang;
  if (threadIdx.x == 0) on = 0;
  __syncthreads();
  for (int e = A.kjk_ptr[jk] + threadIdx.x; e < A.kjk_ptr[jk + 1]; e += blockDim.x)
    if (S.ent_act[e]) on = 1;
  if (symmetric)
    for (int e = A.kjk_ptr[kj] + threadIdx.x; e < A.kjk_ptr[kj + 1]; e += blockDim.x)
      if (S.ent_act[e]) on = 1;
  __syncthreads();
  if (on) return;
  for (int c = blockIdx.y * 8 + (threadIdx.x >> 5); c < A.nrad; c += 8 * gridDim.y) {
    double* Kc = K + (size_t)(k * A.nrad + c) * A.nbf + (size_t)j * A.nrad;
#pragma unroll 4
    for (int r = threadIdx.x & 31; r < A.nrad; r += 32) Kc[r] = 0.0;
  }
}

// the entries that see an active block, where the density pass leaves them out
__global__ void k_flags(DevAtom A, DevScratch S) {
  for (int ent = blockIdx.x * blockDim.x + threadIdx.x; ent < A.nent; ent += gridDim.x * blockDim.x) {
    bool any = false;
    for (int u = A.kent_ptr[ent]; u < A.kent_ptr[ent + 1] && !any; ++u) any = S.act[A.kterm_blk[u]];
    S.ent_act[ent] = any ? 1 : 0;
  }
}

// threads of k_block_norms: the rows in equal passes of at most 224, so that
// several CTAs share an SM and one's sums and count overlap another's loads
inline int norm_threads(const DevAtom& A) {
  const int passes = (A.nrad + 223) / 224;
  return std::max(64, ((A.nrad + passes - 1) / passes + 31) / 32 * 32);
}

// The density pass. Its last CTA keeps a flag per block and entry in shared
// memory where that fits the default limit, as for every basis of distinct (l, m)
// functions (at most 1.7 KB); a basis that repeats them often has more entries,
// and a CTA would take long over them.
template <int MODE>
cudaError_t launch_norms(const DevAtom& A, const DevScratch& S, const double* P, float2* p2, bool symmetric,
                         cudaStream_t st) {
  constexpr bool lists = MODE == NORM_SPLIT || MODE == NORM_LISTS;
  const size_t nang2 = (size_t)A.nang * A.nang, flags = nang2 + A.nent;
  const bool entries = lists || flags <= 48 * 1024;
  const size_t smem = (lists ? sizeof(int) * (A.nel + nang2) : 0) + (entries ? flags : 0);
  const cudaError_t e = smem_limit(k_block_norms<MODE>, smem);
  if (e != cudaSuccess) return e;
  k_block_norms<MODE><<<dim3((int)nang2, A.nel), norm_threads(A), smem, st>>>(A, S, P, p2, symmetric ? 1 : 0,
                                                                            entries ? 1 : 0);
  if (!entries) k_flags<<<std::min(152 * 4, (A.nent + 255) / 256), 256, 0, st>>>(A, S);
  return cudaGetLastError();
}

__device__ __forceinline__ void load_active(const DevAtom& A, const DevScratch& S, unsigned char* act) {
  const int nang2 = A.nang * A.nang;
  for (int idx = threadIdx.x; idx < nang2; idx += blockDim.x) act[idx] = S.act[idx];
}

__device__ __forceinline__ size_t halo_idx(const DevAtom& A, int a, int b, int jk, int h) {
  return ((size_t)(a * A.nel + b) * (A.nang * A.nang) + jk) * (2 * A.nn - 1) + h;
}

// store the finished contribution y of tile (a,b), angular block jk, at
// local position (p,q): owned entries go to K, the shared last row/column to
// the halo buffer (added by k_fixup)
__device__ __forceinline__ void k_store(const DevAtom& A, const DevScratch& S, double* K, int a, int b,
                                        int jk, int p, int q, double y) {
  const int nn = A.nn;
  const int gp = gfun(A, a, p), gq = gfun(A, b, q);
  if (!gvalid(A, gp) || !gvalid(A, gq)) return;
  const int j = jk % A.nang, k = jk / A.nang;
  if (p <= nn - 2 && q <= nn - 2)
    K[(size_t)(k * A.nrad + gq) * A.nbf + (size_t)j * A.nrad + gp] = y;
  else if (p == nn - 1)
    S.khalo[halo_idx(A, a, b, jk, q)] = y;
  else
    S.khalo[halo_idx(A, a, b, jk, nn + p)] = y;
}

// recoupled tile value for thread (p,q) of element pair (a,b), entry ent
// P_base = P + gq*nbf + gp for this thread's tile entry
__device__ __forceinline__ double k_recouple(const DevAtom& A, const double* __restrict__ Pbase,
                                             const unsigned char* act, int ent) {
  double x = 0.0;
  const int u0 = A.kent_ptr[ent], u1 = A.kent_ptr[ent + 1];
  for (int u = u0; u < u1; ++u) {
    if (!act[A.kterm_blk[u]]) continue;
    x += A.kterm_coef[u] * Pbase[A.kterm_off[u]];
  }
  return x;
}

// Range-separated exchange with the erfc kernel (TwoDBasisT::rs_exchange,
// src/atomic/TwoDBasis.cpp:1001-1131, with the pairwise assembly of
// CoulombExchangeFE.h:396-422): the kernel does not separate into r< / r>
// factors, so every element pair (a,b) carries a dense exchange-ordered
// table per multipole, K_jk(a,b)[t] = -sum_L sum_v T_L(a,b)[t, v] X_L(a,b)[v]
// (t = p + q nn, v = p' + q' nn). One CTA per (element pair, output block),
// one thread per tile entry t; FP64.
__global__ void k_erfc_tiles(DevAtom A, DevScratch S, const double* __restrict__ tk,
                             const double* __restrict__ P, double* __restrict__ K) {
  const int a = blockIdx.x % A.nel, b = blockIdx.x / A.nel, jk = blockIdx.y;
  const int nn = A.nn, n2 = nn * nn, t = threadIdx.x;
  extern __shared__ double xs[];  // [n2]
  unsigned char* act = reinterpret_cast<unsigned char*>(xs + n2);
  for (int idx = t; idx < A.nang * A.nang; idx += blockDim.x) act[idx] = S.act[idx];
  __syncthreads();
  double y = 0.0;
  for (int e = A.kjk_ptr[jk]; e < A.kjk_ptr[jk + 1]; ++e) {
    if (!S.ent_act[e]) continue;  // uniform over the CTA
    for (int v = t; v < n2; v += blockDim.x) {
      const int gp = gfun(A, a, v % nn), gq = gfun(A, b, v / nn);
      xs[v] = (gvalid(A, gp) && gvalid(A, gq)) ? k_recouple(A, P + (size_t)gq * A.nbf + gp, act, e) : 0.0;
    }
    __syncthreads();
    if (t < n2) {
      const double* T = tk + (((size_t)A.kent_L[e] * A.nel + a) * A.nel + b) * n2 * n2;
      for (int v = 0; v < n2; ++v) y += T[t + (size_t)v * n2] * xs[v];
    }
    __syncthreads();
  }
  if (t < n2) k_store(A, S, K, a, b, jk, t % nn, t / nn, -y);
}

// One work unit = one element pair (a,b) and a range of output angular
// blocks. a != b: off-diagonal pair, jk over [lo,hi) in natural order,
// contribution A_L X B_L^T. a == b: diagonal element, jk = diag_jk[lo..hi),
// contribution Tk X. In symmetric mode (P = P^T) only a < b pairs and j <= k
// diagonal blocks are units; each also writes the transposed partner tile
// (k,j,b,a), since K_kj(b,a) = K_jk(a,b)^T.
__global__ void __launch_bounds__(320) k_tiles(DevAtom A, DevScratch S, const int4* __restrict__ units,
                                               const int* __restrict__ diag_jk, int symmetric,
                                               const double* __restrict__ P, double* __restrict__ K) {
  const int4 u = units[blockIdx.x];
  const int a = u.x, b = u.y;
  const int nn = A.nn, n2 = nn * nn, NL = A.NL, nang2 = A.nang * A.nang;
  extern __shared__ double sm[];
  double* X = sm;
  double* T = X + n2;
  double* Am = T + n2;
  double* Bm = Am + NL * n2;
  unsigned char* act = reinterpret_cast<unsigned char*>(Bm + NL * n2);
  const bool diag = (a == b);
  if (!diag) {
    const double* srcA = (a < b) ? A.rs : A.rb;
    const double* srcB = (a < b) ? A.rb : A.rs;
    for (int idx = threadIdx.x; idx < NL * n2; idx += blockDim.x) {
      const int L = idx / n2, o = idx % n2;
      Am[idx] = srcA[((size_t)L * A.nel + a) * n2 + o];
      Bm[idx] = srcB[((size_t)L * A.nel + b) * n2 + o];
    }
  }
  load_active(A, S, act);
  __syncthreads();
  const int t = threadIdx.x;
  const bool live = t < n2;
  const int p = live ? t % nn : 0, q = live ? t / nn : 0;
  const int gp = gfun(A, a, p), gq = gfun(A, b, q);
  const bool vpq = live && gvalid(A, gp) && gvalid(A, gq);
  for (int w = u.z; w < u.w; ++w) {
    const int jk = diag ? diag_jk[w] : w;
    double y = 0.0;
    const double* Pbase = P + (size_t)gq * A.nbf + gp;
    for (int ent = A.kjk_ptr[jk]; ent < A.kjk_ptr[jk + 1]; ++ent) {
      if (!S.ent_act[ent]) continue;  // uniform over the CTA
      const int L = A.kent_L[ent];
      if (live) X[t] = vpq ? k_recouple(A, Pbase, act, ent) : 0.0;
      __syncthreads();
      if (diag) {
        if (live) {
          const double* Tk = A.tk + ((size_t)L * A.nel + a) * n2 * n2;
          double s = 0.0;
          for (int v = 0; v < n2; ++v) s += Tk[t + (size_t)v * n2] * X[v];
          y += s;
        }
      } else {
        if (live) {
          const double* Bl = Bm + L * n2;
          double s = 0.0;
          for (int c = 0; c < nn; ++c) s += X[p + c * nn] * Bl[q + c * nn];
          T[t] = s;
        }
        __syncthreads();
        if (live) {
          const double* Al = Am + L * n2;
          double s = 0.0;
          for (int c = 0; c < nn; ++c) s += Al[p + c * nn] * T[c + q * nn];
          y += s;
        }
      }
      __syncthreads();
    }
    if (live) k_store(A, S, K, a, b, jk, p, q, -y);
    const int j = jk % A.nang, k = jk / A.nang;
    if (symmetric && (!diag || j != k)) {
      // transposed partner: stage through shared memory so that consecutive
      // threads write consecutive rows of the column-major output
      if (live) X[t] = -y;
      __syncthreads();
      if (live) k_store(A, S, K, b, a, k + j * A.nang, p, q, X[q + p * nn]);
      __syncthreads();
    }
  }
}

// p2base = S.p2 + gq*nbf + gp for this thread's tile entry
__device__ __forceinline__ ffv k_recouple_ff(const DevAtom& A, const float2* __restrict__ p2base,
                                             const unsigned char* act, int ent) {
  ffv x = {0.f, 0.f};
  const int u0 = A.kent_ptr[ent], u1 = A.kent_ptr[ent + 1];
  for (int u = u0; u < u1; ++u) {
    if (!act[A.kterm_blk[u]]) continue;
    x = ff_fma(x, A.kterm_coef2[u], p2base[A.kterm_off[u]]);
  }
  return x;
}


// NN > 0: element order fixed at compile time (the element-pair contractions
// unroll with immediate shared-memory offsets); NN = 0: any order
template <int NN>
__global__ void __launch_bounds__(320) k_tiles_split(DevAtom A, DevScratch S, const int4* __restrict__ units,
                                                     const int* __restrict__ diag_jk, int symmetric,
                                                     double* __restrict__ K) {
  const int4 u = units[blockIdx.x];
  const int a = u.x, b = u.y;
  const int nn = NN > 0 ? NN : A.nn, n2 = nn * nn, NL = A.NL;
  extern __shared__ float2 sm2[];
  float2* X = sm2;
  float2* T = X + n2;
  float2* Am = T + n2;
  float2* Bm = Am + NL * n2;
  double* Y = reinterpret_cast<double*>(Bm + NL * n2);
  unsigned char* act = reinterpret_cast<unsigned char*>(Y + n2);
  const bool diag = (a == b);
  if (!diag) {
    const float2* srcA = (a < b) ? A.rs2 : A.rb2;
    const float2* srcB = (a < b) ? A.rb2 : A.rs2;
    for (int idx = threadIdx.x; idx < NL * n2; idx += blockDim.x) {
      const int L = idx / n2, o = idx % n2;
      Am[idx] = srcA[((size_t)L * A.nel + a) * n2 + o];
      Bm[idx] = srcB[((size_t)L * A.nel + b) * n2 + o];
    }
  }
  load_active(A, S, act);
  __syncthreads();
  const int t = threadIdx.x;
  const bool live = t < n2;
  const int p = live ? t % nn : 0, q = live ? t / nn : 0;
  const int gp = gfun(A, a, p), gq = gfun(A, b, q);
  const bool vpq = live && gvalid(A, gp) && gvalid(A, gq);
  const float2* p2base = S.p2 + (size_t)gq * A.nbf + gp;
  for (int w = u.z; w < u.w; ++w) {
    const int jk = diag ? diag_jk[w] : w;
    ffv yacc = {0.f, 0.f};
    // the recoupled density tile of the next active entry is loaded while the
    // current one is contracted (its global loads overlap the FP32 work)
    const int ent_end = A.kjk_ptr[jk + 1];
    int ent = A.kjk_ptr[jk];
    while (ent < ent_end && !S.ent_act[ent]) ++ent;  // uniform over the CTA
    float2 xcur = make_float2(0.f, 0.f);
    if (ent < ent_end && vpq) xcur = ff2(k_recouple_ff(A, p2base, act, ent));
    while (ent < ent_end) {
      const int L = A.kent_L[ent];
      if (live) X[t] = xcur;
      __syncthreads();
      int ent_next = ent + 1;
      while (ent_next < ent_end && !S.ent_act[ent_next]) ++ent_next;
      float2 xnext = make_float2(0.f, 0.f);
      if (ent_next < ent_end && vpq) xnext = ff2(k_recouple_ff(A, p2base, act, ent_next));
      ffv acc = {0.f, 0.f};
      if (diag) {
        if (live) {
          // lazy low-word accumulation, renormalised every nn terms
          const float2* Tk = A.tk2 + ((size_t)L * A.nel + a) * n2 * n2;
          for (int v0 = 0; v0 < n2; v0 += nn) {
#pragma unroll
            for (int c = 0; c < (NN > 0 ? NN : 1); ++c) {
              if (NN == 0) break;
              acc = ff_fma(acc, Tk[t + (size_t)(v0 + c) * n2], X[v0 + c]);
            }
            if (NN == 0)
              for (int v = v0; v < v0 + nn; ++v) acc = ff_fma(acc, Tk[t + (size_t)v * n2], X[v]);
            acc = ff_norm(acc.hi, acc.lo);
          }
        }
      } else {
        if (live) {
          const float2* Bl = Bm + L * n2;
          ffv s = {0.f, 0.f};
          if (NN > 0) {
#pragma unroll
            for (int c = 0; c < (NN > 0 ? NN : 1); ++c) s = ff_fma(s, X[p + c * nn], Bl[q + c * nn]);
          } else {
            for (int c = 0; c < nn; ++c) s = ff_fma(s, X[p + c * nn], Bl[q + c * nn]);
          }
          T[t] = ff2(s);
        }
        __syncthreads();
        if (live) {
          const float2* Al = Am + L * n2;
          if (NN > 0) {
#pragma unroll
            for (int c = 0; c < (NN > 0 ? NN : 1); ++c) acc = ff_fma(acc, Al[p + c * nn], T[c + q * nn]);
          } else {
            for (int c = 0; c < nn; ++c) acc = ff_fma(acc, Al[p + c * nn], T[c + q * nn]);
          }
        }
      }
      yacc = ff_add(yacc, ff_norm(acc.hi, acc.lo));
      __syncthreads();
      ent = ent_next;
      xcur = xnext;
    }
    const double y = ff_to_d(yacc);  // FP64 recombination, once per output element
    if (live) k_store(A, S, K, a, b, jk, p, q, -y);
    const int j = jk % A.nang, k = jk / A.nang;
    if (symmetric && (!diag || j != k)) {
      if (live) Y[t] = -y;
      __syncthreads();
      if (live) k_store(A, S, K, b, a, k + j * A.nang, p, q, Y[q + p * nn]);
      __syncthreads();
    }
  }
}

// one CTA per element pair (a,b), all output blocks: the first row/column of
// each tile receives its neighbours' halo entries in a fixed order. After the
// tensor-core tiles, which leave out the inactive output blocks: the active
// ones (FIX_ACTIVE), or all, those without an entry zeroed (FIX_ZERO).
enum { FIX_ALL, FIX_ACTIVE, FIX_ZERO };
template <int MODE>
__global__ void k_fixup(DevAtom A, DevScratch S, double* __restrict__ K) {
  const int a = blockIdx.x % A.nel, b = blockIdx.x / A.nel;
  const int nn = A.nn, per = 2 * nn - 3, nang2 = A.nang * A.nang, nblk = MODE == FIX_ACTIVE ? S.ocount[0] : nang2;
  for (int w = threadIdx.x; w < per * nblk; w += blockDim.x) {
    const int idx = w % per, jk = MODE == FIX_ACTIVE ? S.olist[w / per] : w / per;
    if (MODE == FIX_ZERO && !S.jk_on[jk]) continue;
    const int j = jk % A.nang, k = jk / A.nang;
    int p, q;
    double v;
    if (idx < nn - 1) {  // first row of tile (a,b), q in [0, nn-2]
      if (a == 0) continue;
      p = 0;
      q = idx;
      v = S.khalo[halo_idx(A, a - 1, b, jk, q)];
      if (q == 0) {
        if (b == 0) continue;
        v += S.khalo[halo_idx(A, a, b - 1, jk, nn + 0)];
        v += S.khalo[halo_idx(A, a - 1, b - 1, jk, nn - 1)];
      }
    } else {  // first column, p in [1, nn-2]
      if (b == 0) continue;
      p = idx - (nn - 1) + 1;
      q = 0;
      v = S.khalo[halo_idx(A, a, b - 1, jk, nn + p)];
    }
    const int gp = gfun(A, a, p), gq = gfun(A, b, q);
    if (!gvalid(A, gp) || !gvalid(A, gq)) continue;
    K[(size_t)(k * A.nrad + gq) * A.nbf + (size_t)j * A.nrad + gp] += v;
  }
  if (MODE != FIX_ZERO) return;
  for (int jk = 0; jk < nang2; ++jk) {
    if (S.jk_on[jk]) continue;
    const int j = jk % A.nang, k = jk / A.nang;
    for (int w = threadIdx.x; w < (nn - 1) * (nn - 1); w += blockDim.x) {
      const int gp = gfun(A, a, w % (nn - 1)), gq = gfun(A, b, w / (nn - 1));
      if (gvalid(A, gp) && gvalid(A, gq)) K[(size_t)(k * A.nrad + gq) * A.nbf + (size_t)j * A.nrad + gp] = 0.0;
    }
  }
}

// Inactive output blocks: zeroed in the fix-up where K is small, otherwise by a
// kernel of their own beside the tiles. A launch after the diagonal tiles is 3 to 4
// us of a small build's time (l = 0, 5 elements of 6 nodes, tile stage 18.1 us
// with it, 14.1 without; l <= 1, 10 elements of 15 nodes, whole K 62.5 and 59.2),
// while Rn's 240 inactive blocks are 300 MB of writes.
inline bool zero_in_fixup(const DevAtom& A) { return A.nang <= 4 && A.nbf <= 1024; }

inline int threads_for(int n2) { return ((n2 + 31) / 32) * 32; }

struct Mark {
  Profiler* p;
  int slot = -1;
  cudaStream_t s;
  Mark(Profiler* p_, int k, cudaStream_t s_) : p(p_), s(s_) {
    if (p && p->on && ((p->mask >> k) & 1u) && p->n < p->cap) {
      slot = p->n++;
      p->cls[slot] = k;
      cudaEventRecord(p->ev[2 * slot], s);
    }
  }
  ~Mark() {
    if (slot >= 0) cudaEventRecord(p->ev[2 * slot + 1], s);
  }
};

}  // namespace

cudaError_t launch_coulomb_fp64(const DevAtom& A, const DevScratch& S, const double* P, double* J,
                                bool zero_output, cudaStream_t st, Profiler* prof) {
  const int n2 = A.nn * A.nn, th = threads_for(n2);
  if (zero_output) {
    cudaError_t err = cudaMemsetAsync(J, 0, sizeof(double) * (size_t)A.nbf * A.nbf, st);
    if (err != cudaSuccess) return err;
  }
  const size_t sm1 = sizeof(double) * (n2 + A.rmax + 32);
  {
    Mark m(prof, KC_J_CONTRACT, st);
    j_contract<<<dim3(A.nchan, A.nel), th, sm1, st>>>(A, S, P);
  }
  {
    Mark m(prof, KC_J_SCATTER, st);
    j_scatter<<<dim3(A.nang * A.nang, A.nel), th, 0, st>>>(A, S, J, zero_output ? 0 : 1);
  }
  return cudaGetLastError();
}

cudaError_t launch_coulomb_split(const DevAtom& A, const DevScratch& S, const double* P, double* J,
                                 bool zero_output, cudaStream_t st, Profiler* prof) {
  if (!A.cholp2 || !A.jket_coef2 || !A.jbra_coef2 || !A.rs2 || !A.rb2) return cudaErrorInvalidValue;
  const int n2 = A.nn * A.nn, th = threads_for(n2);
  if (zero_output) {
    cudaError_t err = cudaMemsetAsync(J, 0, sizeof(double) * (size_t)A.nbf * A.nbf, st);
    if (err != cudaSuccess) return err;
  }
  const size_t sm1 = sizeof(float2) * (n2 + A.rmax);
  {
    Mark m(prof, KC_J_CONTRACT, st);
    const cudaError_t e = smem_limit(j_contract_split, sm1);
    if (e != cudaSuccess) return e;
    j_contract_split<<<dim3(A.nchan, A.nel), th, sm1, st>>>(A, S, P, A.cholp2);
  }
  {
    Mark m(prof, KC_J_SCATTER, st);
    j_scatter_split<<<dim3(A.nang * A.nang, A.nel), th, 0, st>>>(A, S, J, zero_output ? 0 : 1);
  }
  return cudaGetLastError();
}

cudaError_t launch_exchange_erfc(const DevAtom& A, const DevScratch& S, const double* tk, const double* P, double* K,
                                 cudaStream_t st, Profiler* prof) {
  const int n2 = A.nn * A.nn, nang2 = A.nang * A.nang;
  {
    Mark m(prof, KC_K_NORMS, st);
    const cudaError_t e = launch_norms<NORM_PLAIN>(A, S, P, nullptr, false, st);
    if (e != cudaSuccess) return e;
  }
  {
    Mark m(prof, KC_K_TILES, st);
    const size_t smem = sizeof(double) * n2 + nang2;
    const cudaError_t e = smem_limit(k_erfc_tiles, smem);
    if (e != cudaSuccess) return e;
    k_erfc_tiles<<<dim3(A.nel * A.nel, nang2), threads_for(n2), smem, st>>>(A, S, tk, P, K);
  }
  {
    Mark m(prof, KC_K_FIXUP, st);
    k_fixup<FIX_ALL><<<A.nel * A.nel, 256, 0, st>>>(A, S, K);
  }
  return cudaGetLastError();
}

// The diagonal elements on the tensor cores, through the exchange-ordered
// tensor, and the element pairs by pairs(st): on the tensor cores too, or, for
// elements they do not take (17 nodes), by the FP64 or float-pair kernel. Blocks
// without an active entry are zeroed. P: FP64 form.
template <class Pairs>
static cudaError_t launch_tiles_tc(const DevAtom& A, const DevScratch& S, const DevTC& tc, bool symmetric,
                                   const double* P, double* K, cudaStream_t st, const SideStream* side, Pairs&& pairs) {
  const int nang2 = A.nang * A.nang;
  const bool apart = !zero_in_fixup(A);
  cudaError_t e = cudaSuccess;
  if (side && side->s) {
    // the diagonal stage (a chain of dependent steps in 0.8 of a wave)
    // beside the issue-bound off-diagonal tiles, joined before the fix-up
    e = cudaEventRecord(side->fork, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side->s, side->fork, 0);
    // (the FP64 and float-pair kernels first: a diagonal CTA takes an SM whole)
    if (e == cudaSuccess && !tc.digits) e = pairs();
    if (e == cudaSuccess) e = launch_k_diag_tc(A, S, tc, symmetric, P, K, side->s);
    if (e == cudaSuccess && apart) k_zero_inactive<<<dim3(nang2, 8), 256, 0, side->s>>>(A, S, K, symmetric ? 1 : 0);
    const cudaError_t j = cudaEventRecord(side->join, side->s);
    if (e == cudaSuccess) e = j;
    if (e == cudaSuccess && tc.digits) e = pairs();
    const cudaError_t w = cudaStreamWaitEvent(st, side->join, 0);  // (joined whatever failed)
    if (e == cudaSuccess) e = w;
  } else {
    e = pairs();
    if (e == cudaSuccess) e = launch_k_diag_tc(A, S, tc, symmetric, P, K, st);
    if (e == cudaSuccess && apart) k_zero_inactive<<<dim3(nang2, 8), 256, 0, st>>>(A, S, K, symmetric ? 1 : 0);
  }
  return e;
}

cudaError_t launch_exchange_fp64(const DevAtom& A, const DevScratch& S, const KUnits& U, const double* P,
                                 double* K, bool symmetric, cudaStream_t st, Profiler* prof, const DevTC* tc,
                                 const SideStream* side) {
  const int n2 = A.nn * A.nn, th = threads_for(n2), nang2 = A.nang * A.nang;
  if (tc) {
    {
      Mark m(prof, KC_K_NORMS, st);
      const cudaError_t e = launch_norms<NORM_LISTS>(A, S, P, nullptr, symmetric, st);
      if (e != cudaSuccess) return e;
    }
    {
      Mark m(prof, KC_K_TILES, st);
      const cudaError_t e = launch_tiles_tc(A, S, *tc, symmetric, P, K, st, side, [&]() -> cudaError_t {
        if (tc->digits) return launch_k_tiles_tc(A, S, *tc, symmetric, P, K, st);
        const size_t smem = sizeof(double) * (2 * n2 + 2 * A.NL * n2) + nang2;
        const int nunits = symmetric ? U.n_off_sym : U.n_off_all;
        const cudaError_t l = smem_limit(k_tiles, smem);
        if (l != cudaSuccess) return l;
        if (nunits > 0)
          k_tiles<<<nunits, th, smem, st>>>(A, S, symmetric ? U.sym : U.all, U.diag_jk_src(symmetric), symmetric ? 1 : 0, P,
                                            K);
        return cudaGetLastError();
      });
      if (e != cudaSuccess) return e;
    }
    {
      Mark m(prof, KC_K_FIXUP, st);
      (zero_in_fixup(A) ? k_fixup<FIX_ZERO> : k_fixup<FIX_ACTIVE>)<<<A.nel * A.nel, 256, 0, st>>>(A, S, K);
    }
    return cudaGetLastError();
  }
  {
    Mark m(prof, KC_K_NORMS, st);
    const cudaError_t e = launch_norms<NORM_PLAIN>(A, S, P, nullptr, symmetric, st);
    if (e != cudaSuccess) return e;
  }
  {
    Mark m(prof, KC_K_TILES, st);
    const size_t smem = sizeof(double) * (2 * n2 + 2 * A.NL * n2) + nang2;
    const int nunits = symmetric ? U.n_sym : U.n_all;
    const cudaError_t e = smem_limit(k_tiles, smem);
    if (e != cudaSuccess) return e;
    k_tiles<<<nunits, th, smem, st>>>(A, S, symmetric ? U.sym : U.all, U.diag_jk_src(symmetric), symmetric ? 1 : 0,
                                      P, K);
  }
  {
    Mark m(prof, KC_K_FIXUP, st);
    k_fixup<FIX_ALL><<<A.nel * A.nel, 256, 0, st>>>(A, S, K);
  }
  return cudaGetLastError();
}

cudaError_t launch_exchange_split(const DevAtom& A, const DevScratch& S, const KUnits& U, const double* P,
                                  double* K, bool symmetric, cudaStream_t st, Profiler* prof, const DevTC* tc,
                                  const SideStream* side) {
  const int n2 = A.nn * A.nn, th = threads_for(n2), nang2 = A.nang * A.nang;
  {
    Mark m(prof, KC_K_NORMS, st);
    const cudaError_t e = tc ? launch_norms<NORM_SPLIT>(A, S, P, S.p2, symmetric, st)
                             : launch_norms<NORM_COPY>(A, S, P, S.p2, symmetric, st);
    if (e != cudaSuccess) return e;
  }
  {
    Mark m(prof, KC_K_TILES, st);
    const size_t smem = sizeof(float2) * (2 * n2 + 2 * A.NL * n2) + sizeof(double) * n2 + nang2;
    const int4* units = symmetric ? U.sym : U.all;
    auto kern = (A.nn == 15) ? k_tiles_split<15> : k_tiles_split<0>;
    auto pairs = [&](int nunits) -> cudaError_t {
      const cudaError_t l = smem_limit(kern, smem);
      if (l != cudaSuccess) return l;
      if (nunits > 0)
        kern<<<nunits, th, smem, st>>>(A, S, units, U.diag_jk_src(symmetric), symmetric ? 1 : 0, K);
      return cudaGetLastError();
    };
    const cudaError_t e =
        tc ? launch_tiles_tc(A, S, *tc, symmetric, nullptr, K, st, side,
                             [&]() {
                               return tc->digits ? launch_k_tiles_tc(A, S, *tc, symmetric, nullptr, K, st)
                                                 : pairs(symmetric ? U.n_off_sym : U.n_off_all);
                             })
           : pairs(symmetric ? U.n_sym : U.n_all);
    if (e != cudaSuccess) return e;
  }
  {
    Mark m(prof, KC_K_FIXUP, st);
    (!tc ? k_fixup<FIX_ALL> : zero_in_fixup(A) ? k_fixup<FIX_ZERO> : k_fixup<FIX_ACTIVE>)
        <<<A.nel * A.nel, 256, 0, st>>>(A, S, K);
  }
  return cudaGetLastError();
}

// Upper part of a symmetric column-major n x n matrix from its lower
// column blocks: for blocks of bw columns, P(r, c) = P(c, r) wherever
// r / bw < c / bw (block c holds rows >= its first column, so the source
// is always present). 32 x 32 tiles through shared memory.
__global__ void k_mirror_blocks(double* __restrict__ P, int n, int bw) {
  __shared__ double t[32][33];
  const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  if (r0 / bw >= min(c0 + 31, n - 1) / bw) return;  // no element of the tile is mirrored
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int k = ty; k < 32; k += 8) {
    const int r = r0 + k, c = c0 + tx;
    if (r < n && c < n && r / bw < c / bw) t[k][tx] = P[c + (size_t)r * n];
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    const int c = c0 + k, r = r0 + tx;
    if (r < n && c < n && r / bw < c / bw) P[r + (size_t)c * n] = t[tx][k];
  }
}

cudaError_t launch_mirror_blocks(double* P, int n, int bw, cudaStream_t st) {
  if (n < 1 || bw < 1) return cudaErrorInvalidValue;
  const int nt = (n + 31) / 32;
  k_mirror_blocks<<<dim3(nt, nt), dim3(32, 8), 0, st>>>(P, n, bw);
  return cudaGetLastError();
}

}  // namespace hfg
