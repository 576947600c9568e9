// Recoupling of the diatomic exchange shared by the output blocks of one k
// (see dk_share.cu for the scheme): the arithmetic types, the lists of one
// chunk of density rows, and the recoupled tiles V0_i, V2_i.
#pragma once

#include "devdiatomic.cuh"
#include "ff.cuh"

namespace hfg {
namespace {

constexpr int IC = 4;  // density rows i at a time

__device__ __forceinline__ int sgf(const DevDiatomic& D, int e, int p) { return e * (D.nn - 1) + p; }
__device__ __forceinline__ int sal(const DevDiatomic& D, int a, int L, int M) {
  return (a * (D.Lmax + 1) + L) * D.nM + M + 2 * D.mmax;
}

struct ArD {  // FP64
  using V = double;
  using A = double;
  static __device__ __forceinline__ A zero() { return 0.0; }
  static __device__ __forceinline__ A acc(V v) { return v; }
  static __device__ __forceinline__ A fma(A a, V x, V y) { return a + x * y; }
  static __device__ __forceinline__ V val(A a) { return a; }
  static __device__ __forceinline__ V neg(V v) { return -v; }
  static __device__ __forceinline__ bool nz(V v) { return v != 0.0; }
  static __device__ __forceinline__ A sum(A a, A b) { return a + b; }
  static __device__ __forceinline__ A scale2(A a, int) { return a; }
  static __device__ __forceinline__ double out(V v) { return v; }
};
struct ArF {  // float pairs
  using V = float2;
  using A = ffv;
  static __device__ __forceinline__ A zero() { return {0.f, 0.f}; }
  static __device__ __forceinline__ A acc(V v) { return {v.x, v.y}; }
  static __device__ __forceinline__ A fma(A a, V x, V y) { return ff_fma(a, x, y); }
  static __device__ __forceinline__ V val(A a) { return ff2(a); }
  static __device__ __forceinline__ V neg(V v) { return make_float2(-v.x, -v.y); }
  static __device__ __forceinline__ bool nz(V v) { return v.x != 0.f; }
  static __device__ __forceinline__ A sum(A a, A b) { return ff_add(a, b); }
  static __device__ __forceinline__ A scale2(A a, int k) { return {ldexpf(a.hi, k), ldexpf(a.lo, k)}; }
  static __device__ __forceinline__ double out(V v) { return (double)v.x + (double)v.y; }
};

template <class AR>
struct Src {  // operand tables of one arithmetic type
  const typename AR::V *P, *c0, *c2, *fac, *p0, *p2, *q0, *q2;
};
template <class AR>
__device__ __forceinline__ Src<AR> src_of(const DevDiatomic& D, const DevDiatomicScratch& S, const double* Pd);
template <>
__device__ __forceinline__ Src<ArD> src_of<ArD>(const DevDiatomic& D, const DevDiatomicScratch&, const double* Pd) {
  return {Pd, D.al_c0, D.al_c2, D.lmfac, D.p0, D.p2, D.q0, D.q2};
}
template <>
__device__ __forceinline__ Src<ArF> src_of<ArF>(const DevDiatomic& D, const DevDiatomicScratch& S, const double*) {
  return {S.pd2, D.al_c0s, D.al_c2s, D.lmfacs, D.p0s, D.p2s, D.q0s, D.q2s};
}

__device__ __forceinline__ void share_store(const DevDiatomic& D, const DevDiatomicScratch& S, double* Kd, int a,
                                            int b, int jk, int p, int q, double y) {
  const int nn = D.nn;
  const int gp = sgf(D, a, p), gq = sgf(D, b, q);
  if (gp >= D.nrad || gq >= D.nrad) return;
  const int j = jk % D.nang, k = jk / D.nang;
  const size_t h = ((size_t)(a * D.nel + b) * (D.nang * D.nang) + jk) * (2 * nn - 1);
  if (p <= nn - 2 && q <= nn - 2)
    Kd[(size_t)(k * D.nrad + gq) * D.nd + (size_t)j * D.nrad + gp] = y;
  else if (p == nn - 1)
    S.khalo[h + q] = y;
  else
    S.khalo[h + nn + p] = y;
}

// One chunk of up to IC density rows i of (k; L, M): the l list and the
// couplings of the group's rows, in shared memory. Returns whether any
// density block of the chunk is active (uniform over the CTA). Buffers are
// double-buffered by par: the previous chunk's may still be read.
template <class AR, int JC>
struct Chunk {
  typename AR::V k0[256], k2[256];          // couplings of (k, l)
  typename AR::V j0[2][JC][IC], j2[2][JC][IC];  // couplings of (j, i)
  int l[256];
  unsigned char am[2][256];                 // active (i, l): bit ii of entry u
};

template <class AR, int JC>
__device__ __forceinline__ int chunk_fill(const DevDiatomic& D, const DevDiatomicScratch& S, const Src<AR>& T,
                                          Chunk<AR, JC>& C, const int* js, int nj, int k, int L, int M,
                                          const int* is, int ni, int par, bool first) {
  const int xk = sal(D, k, L, M), u0 = D.al_ptr[xk], nl = D.al_ptr[xk + 1] - u0;
  bool any = false;
  for (int u = threadIdx.x; u < nl; u += blockDim.x) {
    const int l = D.al_b[u0 + u];
    unsigned m = 0;
    for (int ii = 0; ii < ni; ++ii)
      if (S.act[is[ii] + l * D.nang]) m |= 1u << ii;
    C.am[par][u] = (unsigned char)m;
    any |= m != 0;
    if (first) {
      C.l[u] = l;
      C.k0[u] = T.c0[u0 + u];
      C.k2[u] = T.c2[u0 + u];
    }
  }
  for (int x = threadIdx.x; x < nj * IC; x += blockDim.x) {
    const int jj = x / IC, ii = x % IC;
    typename AR::V a = AR::val(AR::zero()), b = a;
    if (ii < ni) {
      const int xj = sal(D, js[jj], L, M);
      for (int u = D.al_ptr[xj]; u < D.al_ptr[xj + 1]; ++u)
        if (D.al_b[u] == is[ii]) {
          a = T.c0[u];
          b = T.c2[u];
        }
    }
    C.j0[par][jj][ii] = a;
    C.j2[par][jj][ii] = b;
  }
  return __syncthreads_or(any) ? nl : 0;
}

// V0_i, V2_i at this thread's tile entry for the chunk's rows; two l (eight
// density loads) in flight
template <class AR, int JC>
__device__ __forceinline__ void recouple_k(const DevDiatomic& D, const Chunk<AR, JC>& C, const typename AR::V* pb,
                                           bool live, const int* is, int ni, int nl, int par,
                                           typename AR::A (&v0)[IC], typename AR::A (&v2)[IC]) {
#pragma unroll
  for (int ii = 0; ii < IC; ++ii) v0[ii] = v2[ii] = AR::zero();
  size_t oi[IC];
#pragma unroll
  for (int ii = 0; ii < IC; ++ii) oi[ii] = (size_t)(ii < ni ? is[ii] : is[0]) * D.nrad;
  for (int u = 0; u < nl; u += 2) {
    typename AR::V x[2][IC];
    unsigned m[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      m[w] = (u + w < nl && live) ? C.am[par][u + w] : 0u;
      const typename AR::V* pl = pb + (size_t)(u + w < nl ? C.l[u + w] : 0) * D.nrad * D.nd;
#pragma unroll
      for (int ii = 0; ii < IC; ++ii)
        x[w][ii] = ((m[w] >> ii) & 1u) ? pl[oi[ii]] : AR::val(AR::zero());
    }
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      if (m[w] == 0) continue;
      const typename AR::V c0 = C.k0[u + w], c2 = C.k2[u + w];
#pragma unroll
      for (int ii = 0; ii < IC; ++ii) {
        if (ii >= ni) break;  // uniform
        v0[ii] = AR::fma(v0[ii], c0, x[w][ii]);
        v2[ii] = AR::fma(v2[ii], c2, x[w][ii]);
      }
    }
  }
}

constexpr int JC_OFF = 16;   // output rows per off-diagonal item
constexpr int JC_DIAG = 8;   // output rows per in-element item

}  // namespace
}  // namespace hfg
