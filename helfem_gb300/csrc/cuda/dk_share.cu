// Diatomic exchange (diatomic TwoDBasis::exchange, src/diatomic/basis.cpp:
// 1817-2061) with the recoupling and the outer-side products shared by the
// output blocks of one k.
//
// For one output column k and one multipole (L, M) the reference's sum over
// density blocks factorises: with the couplings c0 (cos^2-weighted) and c2 of
// (k; L, M; l) and of (j; L, M; i),
//   V0_i = sum_l c0(k, l) P_il,  V2_i = sum_l c2(k, l) P_il        (for every i)
//   U_i  = V0_i J0^T - V2_i J2^T
//   W0_j = sum_i c0(j, i) U_i,   W2_j = sum_i c2(j, i) U_i         (for every j)
//   K_jk -= fac (I0 W0_j - I2 W2_j)
// for an element pair (I: integrals of the row element, J: of the column
// element, P- or Q-type by element order). An item is one element pair, one k
// and one group of output rows j with a common m (they need the same i, m_i =
// m_j - M, so nothing is computed twice): per tile entry the recoupling costs
// O(n) per (i or j) instead of O(n^2) per output block, and the products 4 nn
// multiply-adds per (i or j) instead of 6 nn per block. The arithmetic type is a
// template parameter (FP64, or float pairs for the split form).
//
// Measured against one output block per item (GB300, whole K): N2, 12
// elements, l <= 10, split, element-pair tiles 45 -> 31 ms; in FP64 N2 on 6
// elements, l <= 5, m <= 1 5.10 -> 3.91 ms, H2 on 3 elements 0.85 -> 0.55 ms
// (with the in-element tiles below).
#include <algorithm>

#include "dk_recouple.cuh"
#include "smem_limit.hpp"

namespace hfg {
namespace {

// The next item of a persistent CTA. Its first one is its own index, so that
// few items spread over the SMs (consecutive CTAs start on different SMs);
// then the counter hands them out. A barrier on either side.
__device__ __forceinline__ int next_item(int* counter, int* slot) {
  __syncthreads();
  if (threadIdx.x == 0) *slot = gridDim.x + atomicAdd(counter, 1);
  __syncthreads();
  return *slot;
}

// s[x] += sum over columns lo..hi of table row entries times X[x], NJ rows x
template <int NJ>
__device__ __forceinline__ void row_products(const double* tx, int n2, const double* X, int lo, int hi,
                                             double (&s)[JC_DIAG]) {
#pragma unroll 4
  for (int v = lo; v < hi; ++v) {
    const double tv = tx[(size_t)v * n2];
#pragma unroll
    for (int x = 0; x < NJ; ++x) s[x] += tv * X[(size_t)x * 4 * n2 + v];
  }
}

}  // namespace

// Off-diagonal element pairs: persistent CTAs, items (element pair, active
// (k, group of output rows)) from a counter. In symmetric mode only a < b
// pairs are items and each also writes the transposed partner tiles.
template <class AR, int NN>
__global__ void __launch_bounds__(NN == 15 ? 256 : 320, 2) dk_share_off(DevDiatomic D, DevDiatomicScratch S,
                                                                        const double* __restrict__ Pd,
                                                                        double* __restrict__ Kd, int symmetric) {
  using V = typename AR::V;
  using A = typename AR::A;
  const int nn = NN > 0 ? NN : D.nn, n2 = nn * nn;
  extern __shared__ __align__(16) unsigned char smraw[];
  Chunk<AR, JC_OFF>& C = *reinterpret_cast<Chunk<AR, JC_OFF>*>(smraw);
  V* Vs = reinterpret_cast<V*>(smraw + sizeof(Chunk<AR, JC_OFF>));  // [IC][2][n2]
  V* I0 = Vs + 2 * IC * n2;
  V* I2 = I0 + n2;  // negated
  V* J0 = I2 + n2;
  V* J2 = J0 + n2;  // negated
  V* W = J2 + n2;   // [nj][2][n2]
  V* Kc = W + 2 * (size_t)D.gmax * n2;  // [nj][n2]
  __shared__ int s_item;
  const Src<AR> T = src_of<AR>(D, S, Pd);
  const int2* pairs = symmetric ? D.pairs_sym : D.pairs_all;
  const int nkg = S.counts[2];
  const int nparts = S.offparts, nitem = (symmetric ? D.npairs_sym : D.npairs_all) * nkg, total = nitem * nparts;
  const int t = threadIdx.x;
  const bool live = t < n2;
  const int p = live ? t % nn : 0, q = live ? t / nn : 0;
  for (int w = blockIdx.x; w < total; w = next_item(&S.counts[4], &s_item)) {
    // the items of one element pair follow one another: its tiles of P and
    // tables stay in L2
    const int it = w / nparts, lp = w % nparts;
    const int2 pr = pairs[it / nkg];
    const int a = pr.x, b = pr.y, kg = S.kg_list[it % nkg];
    const int k = kg / D.ngrp, g = kg % D.ngrp;
    const int* js = D.msh + D.grp_ptr[g];
    const int nj = D.grp_ptr[g + 1] - D.grp_ptr[g], mj = D.mval[js[0]];
    const int gp = sgf(D, a, p), gq = sgf(D, b, q);
    const bool vpq = live && gp < D.nrad && gq < D.nrad;
    const V* pb = T.P + (size_t)gq * D.nd + gp;
    if (live)
      for (int jj = 0; jj < nj; ++jj) Kc[jj * n2 + t] = AR::val(AR::zero());
    int par = 0;
    for (int ilm = lp; ilm < D.nlm; ilm += nparts) {
      const int L = D.lmL[ilm], Ma = D.lmM[ilm];
      bool wany = false;
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
          const int nl = chunk_fill<AR, JC_OFF>(D, S, T, C, js, nj, k, L, M, is + i0, ni, par, first);
          first = false;
          if (nl == 0) continue;
          if (!wany && live) {  // the pair's integrals for this multipole
            const size_t la = ((size_t)ilm * D.nel + a) * n2 + t, lb = ((size_t)ilm * D.nel + b) * n2 + t;
            I0[t] = (a < b) ? T.p0[la] : T.q0[la];
            I2[t] = AR::neg((a < b) ? T.p2[la] : T.q2[la]);
            J0[t] = (a < b) ? T.q0[lb] : T.p0[lb];
            J2[t] = AR::neg((a < b) ? T.q2[lb] : T.p2[lb]);
          }
          {
            A v0[IC], v2[IC];
            recouple_k<AR, JC_OFF>(D, C, pb, vpq, is + i0, ni, nl, par, v0, v2);
            if (live)
#pragma unroll
              for (int ii = 0; ii < IC; ++ii) {
                Vs[(2 * ii) * n2 + t] = AR::val(v0[ii]);
                Vs[(2 * ii + 1) * n2 + t] = AR::val(v2[ii]);
              }
          }
          __syncthreads();
          if (live) {
            A u[IC];
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) u[ii] = AR::zero();
#pragma unroll(NN > 0 ? 5 : 1)
            for (int c = 0; c < nn; ++c) {
              const V a0 = J0[q + c * nn], a2 = J2[q + c * nn];
#pragma unroll
              for (int ii = 0; ii < IC; ++ii) {
                if (ii >= ni) break;  // uniform
                u[ii] = AR::fma(u[ii], Vs[(2 * ii) * n2 + p + c * nn], a0);
                u[ii] = AR::fma(u[ii], Vs[(2 * ii + 1) * n2 + p + c * nn], a2);
              }
            }
            V uv[IC];
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) uv[ii] = AR::val(u[ii]);
            for (int jj = 0; jj < nj; ++jj) {
              A w0 = AR::zero(), w2 = AR::zero();
              if (wany) {
                w0 = AR::acc(W[(2 * jj) * n2 + t]);
                w2 = AR::acc(W[(2 * jj + 1) * n2 + t]);
              }
#pragma unroll
              for (int ii = 0; ii < IC; ++ii) {
                const V c0 = C.j0[par][jj][ii], c2 = C.j2[par][jj][ii];
                if (AR::nz(c0) || AR::nz(c2)) {
                  w0 = AR::fma(w0, c0, uv[ii]);
                  w2 = AR::fma(w2, c2, uv[ii]);
                }
              }
              W[(2 * jj) * n2 + t] = AR::val(w0);
              W[(2 * jj + 1) * n2 + t] = AR::val(w2);
            }
          }
          wany = true;
        }
      }
      if (!wany) continue;  // uniform over the CTA
      __syncthreads();
      if (live) {
        V fac = T.fac[ilm];
        if (Ma & 1) fac = AR::neg(fac);
        // the split tables carry powers of two per element: 2^(k_inner - k_outer)
        int dk = 0;
        if (D.kexp) {
          const int ka = D.kexp[(size_t)ilm * D.nel + a], kb = D.kexp[(size_t)ilm * D.nel + b];
          dk = (a < b) ? ka - kb : kb - ka;
        }
        constexpr int JU = 2;
        for (int jj = 0; jj < nj; jj += JU) {
          A s[JU];
#pragma unroll
          for (int x = 0; x < JU; ++x) s[x] = AR::zero();
          const V* Wj = W + (size_t)2 * jj * n2;
          const int two = jj + 1 < nj ? 2 * n2 : 0;  // the last odd row twice
#pragma unroll(NN > 0 ? 5 : 1)
          for (int c = 0; c < nn; ++c) {
            const V a0 = I0[p + c * nn], a2 = I2[p + c * nn];
#pragma unroll
            for (int x = 0; x < JU; ++x) {
              s[x] = AR::fma(s[x], a0, Wj[x * two + c + q * nn]);
              s[x] = AR::fma(s[x], a2, Wj[x * two + n2 + c + q * nn]);
            }
          }
#pragma unroll
          for (int x = 0; x < JU; ++x)
            if (jj + x < nj) {
              A r = AR::scale2(AR::fma(AR::zero(), fac, AR::val(s[x])), dk);
              Kc[(jj + x) * n2 + t] = AR::val(AR::sum(AR::acc(Kc[(jj + x) * n2 + t]), AR::acc(AR::val(r))));
            }
        }
      }
      __syncthreads();
    }
    if (nparts > 1) {  // summed by dk_share_sum
      if (live)
        for (int jj = 0; jj < nj; ++jj)
          S.offsum[(((size_t)lp * nitem + it) * D.gmax + jj) * n2 + t] = AR::out(Kc[jj * n2 + t]);
      continue;
    }
    if (live)
      for (int jj = 0; jj < nj; ++jj) share_store(D, S, Kd, a, b, js[jj] + k * D.nang, p, q, -AR::out(Kc[jj * n2 + t]));
    if (symmetric) {  // the transposed partner (each thread wrote its entry before the last barrier)
      if (live)
        for (int jj = 0; jj < nj; ++jj)
          share_store(D, S, Kd, b, a, k + js[jj] * D.nang, p, q, -AR::out(Kc[jj * n2 + q + p * nn]));
    }
  }
}

// The off-diagonal items' parts summed in order and stored; grid (items' upper
// bound, parts of their entries)
__global__ void dk_share_sum(DevDiatomic D, DevDiatomicScratch S, double* __restrict__ Kd, int symmetric) {
  const int2* pairs = symmetric ? D.pairs_sym : D.pairs_all;
  const int nkg = S.counts[2], nitem = (symmetric ? D.npairs_sym : D.npairs_all) * nkg, nn = D.nn, n2 = nn * nn;
  const int it = blockIdx.x;
  if (it >= nitem) return;
  const int2 pr = pairs[it / nkg];
  const int kg = S.kg_list[it % nkg], k = kg / D.ngrp, g = kg % D.ngrp;
  const int* js = D.msh + D.grp_ptr[g];
  const int nj = D.grp_ptr[g + 1] - D.grp_ptr[g];
  for (int x = blockIdx.y * blockDim.x + threadIdx.x; x < nj * n2; x += gridDim.y * blockDim.x) {
    const int jj = x / n2, t = x % n2, p = t % nn, q = t / nn;
    double s = 0.0;
#pragma unroll 8
    for (int lp = 0; lp < S.offparts; ++lp) s += S.offsum[(((size_t)lp * nitem + it) * D.gmax + jj) * n2 + t];
    share_store(D, S, Kd, pr.x, pr.y, js[jj] + k * D.nang, p, q, -s);
    if (symmetric) share_store(D, S, Kd, pr.y, pr.x, k + js[jj] * D.nang, q, p, -s);
  }
}

// In-element tiles, plain FP64: K_jk(e,e)[t] -= fac sum_ab sum_v tx_ab[t, v]
// X_ab[v], X_ab the four recoupled channel tiles of (j, k) and the multipole.
// dk_x64 forms X once per (element, output block, multipole) of the units
// [u0, u0 + cap) (a unit: 8 output blocks of one element), dk_prod64
// contracts it with the exchange-ordered kernel. The FP64 pipe of each SM is
// the bound (16 cycles per warp instruction), so the second pass is cut into
// parts of the rows and of the multipoles until every SM has several, and
// leaves out the output blocks that lack a multipole.
template <int NN>
__global__ void __launch_bounds__(NN == 15 ? 256 : 320, 2) dk_x64(DevDiatomic D, DevDiatomicScratch S, DevDia64 T,
                                                                  const double* __restrict__ Pd, int symmetric,
                                                                  int u0, int nchunk) {
  using AR = ArD;
  const int nn = NN > 0 ? NN : D.nn, n2 = nn * nn;
  __shared__ Chunk<AR, JC_DIAG> C;
  __shared__ int s_js[JC_DIAG], s_row[JC_DIAG], s_unit[JC_DIAG], s_nj, s_use;
  const int count = symmetric ? S.counts[1] : S.counts[0], nun = (count + 7) / 8;
  if (count == 0) return;
  const int e_lo = u0 / nun, e_hi = min(D.nel - 1, (u0 + T.cap - 1) / nun);
  if (e_lo > e_hi) return;
  const Src<AR> Sr = src_of<AR>(D, S, Pd);
  const int nitem = S.counts[3];
  const int* kgl = S.kg_list + (size_t)D.nang * D.ngrp;
  const long total = (long)(e_hi - e_lo + 1) * nitem * nchunk;
  const int t = threadIdx.x;
  const bool live = t < n2;
  const int p = live ? t % nn : 0, q = live ? t / nn : 0;
  for (long w = blockIdx.x; w < total; w += gridDim.x) {
    const int e = e_lo + (int)(w / ((long)nitem * nchunk)), c = (int)(w % nchunk),
              it = (int)((w / nchunk) % nitem);
    const int k = kgl[it] / D.ngrp8, g = kgl[it] % D.ngrp8;
    __syncthreads();
    if (t == 0) {
      int n = 0, use = 0;
      for (int x = D.grp8_ptr[g]; x < D.grp8_ptr[g + 1]; ++x) {
        const int pos = S.jk_pos[D.msh[x] + k * D.nang];
        if (pos < 0) continue;
        const int u = e * nun + pos / 8 - u0;
        s_js[n] = D.msh[x];
        s_row[n] = pos % 8;
        s_unit[n] = (u >= 0 && u < T.cap) ? u : -1;
        use |= s_unit[n] >= 0;
        ++n;
      }
      s_nj = n;
      s_use = use;
    }
    __syncthreads();
    if (!s_use) continue;  // uniform over the CTA
    const int nj = s_nj, mj = D.mval[s_js[0]];
    const int gp = sgf(D, e, p), gq = sgf(D, e, q);
    const bool vpq = live && gp < D.nrad && gq < D.nrad;
    const double* pb = Pd + (size_t)gq * D.nd + gp;
    int par = 0;
    for (int ilm = c; ilm < D.nlm; ilm += nchunk) {
      const int L = D.lmL[ilm], Ma = D.lmM[ilm];
      double x[JC_DIAG][4];
      unsigned has = 0;  // rows with a coupling (bits, uniform)
#pragma unroll
      for (int jj = 0; jj < JC_DIAG; ++jj)
#pragma unroll
        for (int ab = 0; ab < 4; ++ab) x[jj][ab] = 0.0;
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
          double v0[IC], v2[IC];
          recouple_k<AR, JC_DIAG>(D, C, pb, vpq, is + i0, ni, nl, par, v0, v2);
#pragma unroll
          for (int jj = 0; jj < JC_DIAG; ++jj) {
            if (jj >= nj) break;  // uniform
#pragma unroll
            for (int ii = 0; ii < IC; ++ii) {
              const double c0 = C.j0[par][jj][ii], c2 = C.j2[par][jj][ii];
              if (c0 != 0.0 || c2 != 0.0) {  // uniform
                has |= 1u << jj;
                x[jj][0] += c0 * v0[ii];
                x[jj][1] -= c0 * v2[ii];
                x[jj][2] -= c2 * v0[ii];
                x[jj][3] += c2 * v2[ii];
              }
            }
          }
          __syncthreads();  // the chunk's lists are read until here
        }
      }
      if (!has) continue;
#pragma unroll
      for (int jj = 0; jj < JC_DIAG; ++jj) {
        if (!((has >> jj) & 1u) || s_unit[jj] < 0) continue;
        const size_t ul = (size_t)s_unit[jj] * D.nlm + ilm;
        double* o = T.x + ul * 4 * n2 * 8 + s_row[jj];
        if (live)
#pragma unroll
          for (int ab = 0; ab < 4; ++ab) o[(size_t)(ab * n2 + t) * 8] = x[jj][ab];
        if (t == 0) atomicOr(&T.xact[ul], 1u << s_row[jj]);
      }
    }
  }
}

// CTA = (unit, part of the rows, part of the multipoles); vsplit threads share
// a row t and sum over the columns in turn
__global__ void __launch_bounds__(320) dk_prod64(DevDiatomic D, DevDiatomicScratch S, DevDia64 T, int symmetric,
                                                 int u0) {
  const int count = symmetric ? S.counts[1] : S.counts[0], nun = (count + 7) / 8;
  const int rp = blockIdx.x % T.rsplit, lp = (blockIdx.x / T.rsplit) % T.lparts,
            lu = blockIdx.x / (T.rsplit * T.lparts);
  const int u = u0 + lu;
  if (u >= D.nel * nun) return;
  const int e = u / nun, n2 = D.nn * D.nn, nv = 4 * n2;
  extern __shared__ __align__(16) double smp[];
  double* X = smp;                   // [8][nv]
  double* Y = X + (size_t)8 * nv;    // [8][blockDim]
  const int t = threadIdx.x, rows = (n2 + T.rsplit - 1) / T.rsplit, r0 = rp * rows, nr = min(rows, n2 - r0);
  const int row = t % rows, sub = t / rows;
  const bool work = sub < T.vsplit && row < nr;
  const int lo = nv * sub / T.vsplit, hi = nv * (sub + 1) / T.vsplit;
  for (int x = 0; x < 8; ++x) Y[x * blockDim.x + t] = 0.0;
  for (int ilm = lp; ilm < D.nlm; ilm += T.lparts) {
    const size_t ul = (size_t)lu * D.nlm + ilm;
    const unsigned m = T.xact[ul];
    if (m == 0) continue;  // uniform over the CTA
    const int nj = __popc(m);
    __syncthreads();
    for (int i = t; i < 8 * nv; i += blockDim.x) {  // rows with an entry, packed
      const int r = i % 8;
      if ((m >> r) & 1u) X[(size_t)__popc(m & ((1u << r) - 1)) * nv + i / 8] = T.x[ul * nv * 8 + i];
    }
    __syncthreads();
    if (work) {
      const double fac = (D.lmM[ilm] & 1) ? -D.lmfac[ilm] : D.lmfac[ilm];
      const double* tx = D.tx + ((size_t)ilm * D.nel + e) * nv * n2 + r0 + row;
      double s[JC_DIAG];
#pragma unroll
      for (int x = 0; x < JC_DIAG; ++x) s[x] = 0.0;
      switch (nj) {  // an idle slot would cost the FP64 pipe as much as a used one
        case 1: row_products<1>(tx, n2, X, lo, hi, s); break;
        case 2: row_products<2>(tx, n2, X, lo, hi, s); break;
        case 3: row_products<3>(tx, n2, X, lo, hi, s); break;
        case 4: row_products<4>(tx, n2, X, lo, hi, s); break;
        case 5: row_products<5>(tx, n2, X, lo, hi, s); break;
        case 6: row_products<6>(tx, n2, X, lo, hi, s); break;
        case 7: row_products<7>(tx, n2, X, lo, hi, s); break;
        default: row_products<8>(tx, n2, X, lo, hi, s); break;
      }
      int x = 0;
      for (unsigned b = m; b; b &= b - 1, ++x) {
        double v = s[0];
#pragma unroll
        for (int z = 1; z < JC_DIAG; ++z) v = x == z ? s[z] : v;
        Y[(__ffs(b) - 1) * blockDim.x + t] += fac * v;
      }
    }
  }
  __syncthreads();
  for (int i = t; i < 8 * nr; i += blockDim.x) {
    const int x = i / nr, r = i % nr;
    double s = 0.0;
    for (int z = 0; z < T.vsplit; ++z) s += Y[x * blockDim.x + z * rows + r];
    T.part[(((size_t)lp * T.cap + lu) * 8 + x) * n2 + r0 + r] = s;
  }
}

// the parts of every tile entry summed in order and written to K (and to the
// transposed partner of a symmetric density); one CTA per unit
__global__ void dk_store64(DevDiatomic D, DevDiatomicScratch S, DevDia64 T, int symmetric, int u0,
                           double* __restrict__ Kd) {
  const int count = symmetric ? S.counts[1] : S.counts[0], nun = (count + 7) / 8;
  const int* list = symmetric ? S.jk_list + (size_t)D.nang * D.nang : S.jk_list;
  const int lu = blockIdx.x, u = u0 + lu;
  if (u >= D.nel * nun) return;
  const int e = u / nun, n2 = D.nn * D.nn;
  for (int i = threadIdx.x; i < 8 * n2; i += blockDim.x) {
    const int x = i / n2, t = i % n2, pos = (u % nun) * 8 + x;
    if (pos >= count) break;
    double s = 0.0;
#pragma unroll 4
    for (int lp = 0; lp < T.lparts; ++lp) s += T.part[(((size_t)lp * T.cap + lu) * 8 + x) * n2 + t];
    const int jk = list[pos], j = jk % D.nang, k = jk / D.nang, p = t % D.nn, q = t / D.nn;
    share_store(D, S, Kd, e, e, jk, p, q, -s);
    if (symmetric && j != k) share_store(D, S, Kd, e, e, k + j * D.nang, q, p, -s);
  }
}

namespace {

int sm_count() {
  int dev = 0, n = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

size_t share_off_smem(const DevDiatomic& D);

template <class AR, int NN>
cudaError_t launch_off(const DevDiatomic& D, const DevDiatomicScratch& S, const double* Pd, double* Kd, bool symmetric,
                       cudaStream_t st) {
  const int n2 = D.nn * D.nn;
  const size_t smem = share_off_smem(D);
  auto kern = dk_share_off<AR, NN>;
  cudaError_t e = smem_limit(kern, smem);
  if (e != cudaSuccess) return e;
  int per = 1;
  const int th = ((n2 + 31) / 32) * 32;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, th, smem);
  if (e != cudaSuccess) return e;
  const long items = (long)(symmetric ? D.npairs_sym : D.npairs_all) * D.nang * D.ngrp;
  const int grid = (int)std::min<long>(items * S.offparts, (long)sm_count() * std::max(per, 1));
  kern<<<grid, th, smem, st>>>(D, S, Pd, Kd, symmetric ? 1 : 0);
  if (S.offparts > 1) dk_share_sum<<<dim3((int)items, (D.gmax * n2 + 255) / 256), 256, 0, st>>>(D, S, Kd, symmetric ? 1 : 0);
  return cudaGetLastError();
}

size_t share_off_smem(const DevDiatomic& D) {
  const size_t n2 = (size_t)D.nn * D.nn;
  return sizeof(Chunk<ArD, JC_OFF>) + 8 * n2 * (2 * IC + 4 + 3 * (size_t)D.gmax);
}

}  // namespace

cudaError_t launch_dk_share_off(const DevDiatomic& D, const DevDiatomicScratch& S, const double* Pd, double* Kd,
                                bool symmetric, bool split, cudaStream_t st) {
  if (split)
    return D.nn == 15 ? launch_off<ArF, 15>(D, S, Pd, Kd, symmetric, st)
                      : launch_off<ArF, 0>(D, S, Pd, Kd, symmetric, st);
  DevDiatomic D64 = D;
  D64.kexp = nullptr;  // the FP64 tables are not rescaled
  return D.nn == 15 ? launch_off<ArD, 15>(D64, S, Pd, Kd, symmetric, st)
                    : launch_off<ArD, 0>(D64, S, Pd, Kd, symmetric, st);
}

cudaError_t launch_dk_share_diag(const DevDiatomic& D, const DevDiatomicScratch& S, const DevDia64& T,
                                 const double* Pd, double* Kd, bool symmetric, cudaStream_t st) {
  const int n2 = D.nn * D.nn, th = ((n2 + 31) / 32) * 32;
  auto xk = D.nn == 15 ? dk_x64<15> : dk_x64<0>;
  int per = 1;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, xk, th, 0);
  if (e != cudaSuccess) return e;
  const int slots = sm_count() * std::max(per, 1);
  const int rows = (n2 + T.rsplit - 1) / T.rsplit, pth = (rows * T.vsplit + 31) / 32 * 32;
  const size_t smem = sizeof(double) * 8 * (4 * (size_t)n2 + pth);
  if ((e = smem_limit(dk_prod64, smem)) != cudaSuccess) return e;
  const long nblk = symmetric ? (long)D.nang * (D.nang + 1) / 2 : (long)D.nang * D.nang;
  const int units = (int)(D.nel * ((nblk + 7) / 8));
  // multipoles in parts where there are few (element, k) items (they share nothing)
  const int items = D.nel * D.nang, nchunk = std::max(1, std::min(D.nlm, (4 * slots + items - 1) / items));
  for (int u0 = 0; u0 < units; u0 += T.cap) {
    const int nu = std::min(T.cap, units - u0);
    if ((e = cudaMemsetAsync(T.xact, 0, sizeof(unsigned) * (size_t)T.cap * D.nlm, st)) != cudaSuccess) return e;
    xk<<<slots, th, 0, st>>>(D, S, T, Pd, symmetric ? 1 : 0, u0, nchunk);
    dk_prod64<<<nu * T.rsplit * T.lparts, pth, smem, st>>>(D, S, T, symmetric ? 1 : 0, u0);
    dk_store64<<<nu, 256, 0, st>>>(D, S, T, symmetric ? 1 : 0, u0, Kd);
  }
  return cudaGetLastError();
}

}  // namespace hfg
