// XC potential on the pure-m diatomic DFT grid, plain FP64.
//
// Restates PureMDFTGrid::eval_Fxc and its worker
// (src/diatomic/dftgrid_purem.cpp:83-199 basis values and weights, 213-291
// and 306-369 density and gradient, 480-530 and 575-650 Fock increments,
// 668-712 element loop) in separable form. On mu element e, at mu point q and
// nu point a, the dummy function (s, p) has the value Y_s(a) B_p(q); only
// same-m angular pairs couple. Everything is symmetric under s <-> t, so the
// sums run over unordered pairs k = (s <= t) with multiplicity c_k = 2 (s != t)
// or 1. With
//   D_k(q)  = c_k B(q)^T P_st B(q)
//   Dr_k(q) = c_k/2 [dB(q)^T P_st B(q) + B(q)^T P_st dB(q)]
// the density and its gradient components along mu and nu are
//   rho(q,a) = sum_k D_k(q) W_k(a),          W_k  = Y_s Y_t
//   g_mu     = 2/h sum_k Dr_k(q) W_k(a)
//   g_nu     = 1/h sum_k D_k(q) Wt_k(a),     Wt_k = Y_s' Y_t + Y_s Y_t'
// and the Fock tile of pair k on element e (the X + X^T of the reference
// summed over both orders of the pair) is the symmetric nn x nn matrix
//   V_ij = sum_q B_i B_j (U0_k + Unu_k) + (dB_i B_j + B_i dB_j) Umu_k,
//   U0_k = sum_a f_0 W_k,  Umu_k = sum_a f_mu W_k,  Unu_k = sum_a f_nu Wt_k
// with f_0 = w v_rho and f_c = w (2 v_ss g_c,s + v_ab g_c,s') / h
// (dftgrid_purem.cpp:509-528, 594-615). The same quadrature sums as the
// reference. Densities are read and potentials written in the pure basis
// directly (the mu = 0 function of an m != 0 shell is absent).
//
// The products of a pair and of its -m mirror are the same, so the mirror's
// density tile is added to the pair's before anything else, and only the
// symmetric part of a tile contributes (B^T P B and its derivative).
//
// Kernels: dxc_rad (D, Dr), dxc_point (density, functional, point weights,
// energy partials), dxc_ang (U), dxc_fock (tiles, shared-boundary corner),
// dxc_energy (fixed-order reduction). The FP64 pipe (16 cycles of an SM per
// warp instruction) bounds all of them: every lane works, and what several
// results share is computed once. NO on 14 elements, l <= 9, m <= 2, PBE,
// restricted, before and after (us): dxc_rad 199 and 64, dxc_point 130 and 77,
// dxc_ang 212 and 43, dxc_fock 185 and 90.
#include <algorithm>
#include <cmath>

#include "devatom.cuh"  // xc_func_is_gga
#include "devdiatomic.cuh"
#include "reduce.cuh"
#include "smem_limit.hpp"
#include "xc_func.cuh"

namespace hfg {
namespace {

__device__ __forceinline__ int dgfun(const DevDiatomic& D, int e, int p) { return e * (D.nn - 1) + p; }

// pure index of radial function g of shell s, or -1 where the function is
// not in the pure basis
__device__ __forceinline__ int dpure(const DevDiatomic& D, int s, int g) {
  const int st = D.pstart[s];
  return (g >= st && g < D.nrad) ? D.poff[s] + g - st : -1;
}

// D[s][e][k][q], Dr likewise; grid (nel, groups of np pairs, nsd), thread =
// (pair of the group, q): the group's size fills the warps (nq = 75: two pairs,
// 150 of 160 lanes). With the tile made symmetric, one product T = P B serves D
// and Dr: 17 multiply-adds per tile column instead of 33.
__global__ void dxc_rad(DevDiatomic D, DevDiatomicXC X, DiatomicXcScratch S, int np, const double* __restrict__ P0,
                        const double* __restrict__ P1) {
  const int e = blockIdx.x, k0 = blockIdx.y * np, s = blockIdx.z;
  const int nn = D.nn, nq = X.nq, n2 = nn * nn, nk = min(np, X.npair - k0);
  const double* P = s ? P1 : P0;
  extern __shared__ double sm[];
  double* Pt = sm;             // [np][nn*nn]
  double* R = Pt + np * n2;    // nq*nn
  double* dR = R + nq * nn;    // nq*nn
  for (int idx = threadIdx.x; idx < nk * n2; idx += blockDim.x) {
    const int kk = idx / n2, i = idx % nn, j = idx % n2 / nn;
    const int4 pr = X.pair[k0 + kk];
    const int gi = dgfun(D, e, i), gj = dgfun(D, e, j);
    double v = 0.0;
    auto add = [&](int sa, int ta) {
      const int pi = dpure(D, sa, gi), pj = dpure(D, ta, gj);
      if (pi >= 0 && pj >= 0) v += P[(size_t)pj * D.nbf + pi];
    };
    add(pr.x, pr.y);
    if (pr.z >= 0) add(pr.z, pr.w);
    Pt[idx] = v;
  }
  for (int idx = threadIdx.x; idx < nq * nn; idx += blockDim.x) {
    R[idx] = X.R[(size_t)e * nq * nn + idx];
    dR[idx] = X.dR[(size_t)e * nq * nn + idx];
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < nk * n2; idx += blockDim.x) {  // the symmetric part, in place
    const int kk = idx / n2, i = idx % nn, j = idx % n2 / nn;
    if (i >= j) continue;
    double* T = Pt + kk * n2;
    T[i + j * nn] = T[j + i * nn] = 0.5 * (T[i + j * nn] + T[j + i * nn]);
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < nk * nq; idx += blockDim.x) {
    const int kk = idx / nq, q = idx % nq;
    const double* Rq = R + q * nn;
    const double* dRq = dR + q * nn;
    const double* T = Pt + kk * n2;
    double d = 0.0, dr = 0.0;
    for (int j = 0; j < nn; ++j) {
      double t = 0.0;
      for (int i = 0; i < nn; ++i) t += T[i + j * nn] * Rq[i];
      d += t * Rq[j];
      dr += t * dRq[j];
    }
    const size_t o = (((size_t)s * D.nel + e) * X.npair + k0) * nq + idx;
    const double c = X.mult[k0 + kk];
    S.D[o] = c * d;
    S.Dr[o] = c * dr;
  }
}

// grid (blocks of DXC_POINTS points, nel); thread = point (q, a) of the element
template <bool POL>
__global__ void __launch_bounds__(DXC_POINTS, 16) dxc_point(DevDiatomic D, DevDiatomicXC X, DiatomicXcScratch S, int xid,
                                                           int cid, int gga, double thr) {
  constexpr int nsd = POL ? 2 : 1;
  const int e = blockIdx.y, nq = X.nq, na = X.na, np = X.npair;
  __shared__ double red[32];
  const int pt = blockIdx.x * DXC_POINTS + threadIdx.x, q = pt / na, a = pt % na;
  const bool live = q < nq;
  double rho[2] = {0.0, 0.0}, gm[2] = {0.0, 0.0}, gn[2] = {0.0, 0.0};
  if (live)
#pragma unroll
    for (int s = 0; s < nsd; ++s) {
      const double* Dq = S.D + ((size_t)s * D.nel + e) * np * nq + q;
      const double* Drq = S.Dr + ((size_t)s * D.nel + e) * np * nq + q;
      double rs = 0.0, mr = 0.0, nr = 0.0;
      if (gga) {
#pragma unroll 4
        for (int k = 0; k < np; ++k) {
          const double w = X.W[(size_t)k * na + a], d = Dq[(size_t)k * nq];
          rs += d * w;
          mr += Drq[(size_t)k * nq] * w;
          nr += d * X.Wt[(size_t)k * na + a];
        }
      } else {
#pragma unroll 8
        for (int k = 0; k < np; ++k) rs += Dq[(size_t)k * nq] * X.W[(size_t)k * na + a];
      }
      rho[s] = rs;
      gm[s] = mr;
      gn[s] = nr;
    }
  double esum = 0.0, nsum = 0.0;
  if (live) {
    const size_t pq = (size_t)e * nq * na + pt;
    const double w = X.w[pq], hinv = X.hinv[pq];
    double g[2][2];
    for (int s = 0; s < 2; ++s) {
      g[s][0] = 2.0 * gm[s] * hinv;
      g[s][1] = gn[s] * hinv;
    }
    if (!POL) {  // restricted: equal spin densities from the total P
      rho[0] *= 0.5;
      rho[1] = rho[0];
      for (int c = 0; c < 2; ++c) {
        g[0][c] *= 0.5;
        g[1][c] = g[0][c];
      }
    }
    double ra = rho[0], rb = rho[1];
    const double n = ra + rb;
    xcf::XcOut v = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (n >= thr) {  // density threshold: below it the point contributes nothing
      ra = fmax(ra, 0.5 * thr);
      rb = fmax(rb, 0.5 * thr);
      double saa = 0.0, sab = 0.0, sbb = 0.0;
      if (gga) {
        saa = g[0][0] * g[0][0] + g[0][1] * g[0][1];
        sab = g[0][0] * g[1][0] + g[0][1] * g[1][1];
        sbb = g[1][0] * g[1][0] + g[1][1] * g[1][1];
      }
      v = xc_eval<POL>(xid, cid, ra, rb, saa, sab, sbb);
    }
    esum = w * v.e;
    nsum = w * n;
#pragma unroll
    for (int s = 0; s < nsd; ++s) {
      const size_t cstride = (size_t)D.nel * nq * na;
      const size_t base = (size_t)s * 3 * cstride + pq;
      S.F[base] = w * (s ? v.vb : v.va);
      if (gga) {
        const double vss = s ? v.vbb : v.vaa, vab = v.vab;
        for (int c = 0; c < 2; ++c)
          S.F[base + (size_t)(c + 1) * cstride] = w * (2.0 * vss * g[s][c] + vab * g[1 - s][c]) * hinv;
      }
    }
  }
  esum = block_sum(esum, red);
  nsum = block_sum(nsum, red);
  if (threadIdx.x == 0) {
    S.epart[((size_t)e * gridDim.x + blockIdx.x) * 2 + 0] = esum;
    S.epart[((size_t)e * gridDim.x + blockIdx.x) * 2 + 1] = nsum;
  }
}

// U[o][c][e][k][q] = sum_a F[o][c][e][q][a] Wc[k][a]; grid (nel, groups of QB
// q, nout), thread = pair k with the sums of QB points q: a W value serves QB of
// them (8 leave one CTA per SM, 59 us against 43). (A warp per sum, its lanes over a, spent most of the pipe on adding the
// lanes up: 5 of 7 instructions.)
constexpr int QB = 4;
template <int NC>
__global__ void dxc_ang(DevDiatomic D, DevDiatomicXC X, DiatomicXcScratch S) {
  const int e = blockIdx.x, q0 = blockIdx.y * QB, o = blockIdx.z;
  const int nq = X.nq, na = X.na, np = X.npair, nqb = min(QB, nq - q0);
  extern __shared__ __align__(16) double Fq[];  // [na][NC][QB]
  const size_t cstride = (size_t)D.nel * nq * na;
  for (int idx = threadIdx.x; idx < NC * QB * na; idx += blockDim.x) {
    const int a = idx % na, q = idx / na % QB, c = idx / (na * QB);
    Fq[(a * NC + c) * QB + q] =
        q < nqb ? S.F[((size_t)o * 3 + c) * cstride + ((size_t)e * nq + q0 + q) * na + a] : 0.0;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < np; k += blockDim.x) {
    double acc[NC][QB];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
      for (int q = 0; q < QB; ++q) acc[c][q] = 0.0;
#pragma unroll 2
    for (int a = 0; a < na; ++a) {
      const double w = X.WT[(size_t)a * np + k], wt = NC == 3 ? X.WtT[(size_t)a * np + k] : 0.0;
      const double2* f = reinterpret_cast<const double2*>(Fq + a * NC * QB);
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int q = 0; q < QB; q += 2) {
          const double2 v = f[(c * QB + q) / 2];
          acc[c][q] += v.x * (c == 2 ? wt : w);
          acc[c][q + 1] += v.y * (c == 2 ? wt : w);
        }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      double* u = S.U + ((((size_t)o * 3 + c) * D.nel + e) * np + k) * nq + q0;
#pragma unroll
      for (int q = 0; q < QB; ++q)
        if (q < nqb) u[q] = acc[c][q];
    }
  }
}

// value v at row (a, gi), column (b, gj) of the pure H and at the transposed
// position, where both functions are in the pure basis
__device__ __forceinline__ void dxc_put(const DevDiatomic& D, double* H, int a, int gi, int b, int gj, double v) {
  const int pi = dpure(D, a, gi), pj = dpure(D, b, gj);
  if (pi < 0 || pj < 0) return;
  H[(size_t)pj * D.nbf + pi] = v;
  H[(size_t)pi * D.nbf + pj] = v;
}

// grid (groups of KB pairs, nel, nout). The tile of a pair is symmetric in (i,
// j): each thread builds one i <= j entry of KB pairs, sharing the basis
// products of a point (3 + 2 KB instead of 5 KB instructions per point; above: 4
// pairs 96 us, 6 pairs 90, 8, with few CTAs, 111; on 4 elements, l <= 4, one
// pair), and
// writes it to the (s, t) and (t, s) blocks at both (i, j) and (j, i), and to the
// mirror blocks of opposite m. The rest of H is zero.
template <bool GGA, int KB>
__global__ void dxc_fock(DevDiatomic D, DevDiatomicXC X, DiatomicXcScratch S, double* __restrict__ H0,
                         double* __restrict__ H1) {
  const int k0 = blockIdx.x * KB, e = blockIdx.y, o = blockIdx.z;
  const int nn = D.nn, nq = X.nq, np = X.npair, nk = min(KB, np - k0);
  double* H = o ? H1 : H0;
  extern __shared__ __align__(16) double sm[];
  double* Us = sm;            // [nq][KB]: U0 + Unu
  double* Um = Us + nq * KB;  // [nq][KB]: Umu
  double* R = Um + nq * KB;   // nq*nn
  double* dR = R + nq * nn;   // nq*nn
  __shared__ double corner[KB];
  auto U = [&](int c, int ee, int k) { return S.U + ((((size_t)o * 3 + c) * D.nel + ee) * np + k) * nq; };
  for (int idx = threadIdx.x; idx < nq * nn; idx += blockDim.x) {
    R[idx] = X.R[(size_t)e * nq * nn + idx];
    if (GGA) dR[idx] = X.dR[(size_t)e * nq * nn + idx];
  }
  for (int idx = threadIdx.x; idx < nq * KB; idx += blockDim.x) {
    const int q = idx % nq, kk = idx / nq;
    Us[q * KB + kk] = kk < nk ? U(0, e, k0 + kk)[q] + (GGA ? U(2, e, k0 + kk)[q] : 0.0) : 0.0;
    Um[q * KB + kk] = GGA && kk < nk ? U(1, e, k0 + kk)[q] : 0.0;
  }
  // the first function of element e is the last of element e-1: its diagonal
  // value there, V_{nn-1,nn-1}(e-1)
  for (int kk = threadIdx.x >> 5; kk < nk; kk += blockDim.x >> 5) {
    double c = 0.0;
    if (e > 0) {
      const double* Rp = X.R + (size_t)(e - 1) * nq * nn;
      const double* dRp = X.dR + (size_t)(e - 1) * nq * nn;
      for (int q = threadIdx.x & 31; q < nq; q += 32) {
        const double r = Rp[q * nn + nn - 1], dr = dRp[q * nn + nn - 1];
        c += r * r * (U(0, e - 1, k0 + kk)[q] + (GGA ? U(2, e - 1, k0 + kk)[q] : 0.0)) +
             (GGA ? 2.0 * dr * r * U(1, e - 1, k0 + kk)[q] : 0.0);
      }
    }
    c = warp_sum(c);
    if ((threadIdx.x & 31) == 0) corner[kk] = c;
  }
  __syncthreads();
  const int ntri = nn * (nn + 1) / 2;
  for (int idx = threadIdx.x; idx < ntri; idx += blockDim.x) {
    // idx -> (i <= j), j-major
    int j = (int)((sqrtf(8.0f * idx + 1.0f) - 1.0f) * 0.5f);
    while (j * (j + 1) / 2 > idx) --j;
    while ((j + 1) * (j + 2) / 2 <= idx) ++j;
    const int i = idx - j * (j + 1) / 2;
    if (i == nn - 1 && j == nn - 1) continue;  // owned by the next element (or dropped)
    const int gi = dgfun(D, e, i), gj = dgfun(D, e, j);
    if (gi >= D.nrad || gj >= D.nrad) continue;
    double v[KB];
#pragma unroll
    for (int kk = 0; kk < KB; ++kk) v[kk] = 0.0;
#pragma unroll 3
    for (int q = 0; q < nq; ++q) {
      const double Ri = R[q * nn + i], Rj = R[q * nn + j], G = Ri * Rj;
      const double Hd = GGA ? fma(dR[q * nn + i], Rj, Ri * dR[q * nn + j]) : 0.0;
#pragma unroll
      for (int kk = 0; kk < KB; ++kk) {
        v[kk] += G * Us[q * KB + kk];
        if (GGA) v[kk] += Hd * Um[q * KB + kk];
      }
    }
#pragma unroll
    for (int kk = 0; kk < KB; ++kk) {
      if (kk >= nk) break;
      const int4 pr = X.pair[k0 + kk];
      const double y = (i == 0 && j == 0) ? v[kk] + corner[kk] : v[kk];
      dxc_put(D, H, pr.x, gi, pr.y, gj, y);
      dxc_put(D, H, pr.x, gj, pr.y, gi, y);
      if (pr.z >= 0) {
        dxc_put(D, H, pr.z, gi, pr.w, gj, y);
        dxc_put(D, H, pr.z, gj, pr.w, gi, y);
      }
    }
  }
}

__global__ void dxc_energy(const double* __restrict__ part, int n, double* out) {
  __shared__ double red[32];
  double e = 0.0, nel = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    e += part[2 * i];
    nel += part[2 * i + 1];
  }
  e = block_sum(e, red);
  nel = block_sum(nel, red);
  if (threadIdx.x == 0) {
    out[0] = e;
    out[1] = nel;
  }
}

}  // namespace

cudaError_t launch_diatomic_xc(const DevDiatomic& D, const DevDiatomicXC& X, const DiatomicXcScratch& S, int xid,
                               int cid, const double* Pa, const double* Pb, double* Ha, double* Hb, double* energies,
                               double thr, cudaStream_t st) {
  const bool polarized = Pb != nullptr;
  const int nsd = polarized ? 2 : 1, nout = nsd;
  const bool gga = xc_func_is_gga(xid) || xc_func_is_gga(cid);
  if (X.na > 1024 || X.npair <= 0) return cudaErrorInvalidValue;
  const size_t bytes = sizeof(double) * (size_t)D.nbf * D.nbf;
  cudaError_t err = cudaMemsetAsync(Ha, 0, bytes, st);
  if (err == cudaSuccess && polarized) err = cudaMemsetAsync(Hb, 0, bytes, st);
  if (err != cudaSuccess) return err;
  // pairs per CTA of dxc_rad: the count with the least work per SM (partly
  // filled warps against CTAs for every SM)
  int np = 1;
  double best = 1e300;
  for (int n = 1; n <= 4; ++n) {
    const double warps = (n * X.nq + 31) / 32, ctas = (double)((X.npair + n - 1) / n) * D.nel * nsd / 152.0;
    const double cost = std::max(1.0, ctas) * std::max(ctas > 1.0 ? 0.0 : 1.0, warps / 4.0);
    if (32 * warps <= 512 && cost < best - 1e-9) {
      best = cost;
      np = n;
    }
  }
  const int tq = std::min(512, (np * X.nq + 31) / 32 * 32);
  const size_t rsm = sizeof(double) * ((size_t)np * D.nn * D.nn + 2 * (size_t)X.nq * D.nn);
  err = smem_limit(dxc_rad, rsm);
  if (err != cudaSuccess) return err;
  dxc_rad<<<dim3(D.nel, (X.npair + np - 1) / np, nsd), tq, rsm, st>>>(D, X, S, np, Pa, Pb);
  const int nblk = dxc_blocks(X.nq, X.na);
  auto point = polarized ? dxc_point<true> : dxc_point<false>;
  point<<<dim3(nblk, D.nel), DXC_POINTS, 0, st>>>(D, X, S, xid, cid, gga ? 1 : 0, thr);
  const int tk = std::min(256, (X.npair + 31) / 32 * 32);
  const size_t asm_ = sizeof(double) * (gga ? 3 : 1) * QB * X.na;
  auto ang = gga ? dxc_ang<3> : dxc_ang<1>;
  if ((err = smem_limit(ang, asm_)) != cudaSuccess) return err;
  ang<<<dim3(D.nel, (X.nq + QB - 1) / QB, nout), tk, asm_, st>>>(D, X, S);
  const int ntri = D.nn * (D.nn + 1) / 2;
  // pairs per CTA of dxc_fock: the fewest basis products while every SM has a CTA
  struct { int kb; void (*fn)(DevDiatomic, DevDiatomicXC, DiatomicXcScratch, double*, double*); } fock[4] = {
      {1, gga ? dxc_fock<true, 1> : dxc_fock<false, 1>},
      {2, gga ? dxc_fock<true, 2> : dxc_fock<false, 2>},
      {4, gga ? dxc_fock<true, 4> : dxc_fock<false, 4>},
      {6, gga ? dxc_fock<true, 6> : dxc_fock<false, 6>}};
  int fb = 0;
  double least = 1e300;
  for (int i = 0; i < 4; ++i) {
    const int kb = fock[i].kb;
    const double waves = std::ceil((double)((X.npair + kb - 1) / kb) * D.nel * nout / 152.0);
    const double cost = waves * (gga ? 3 + 2 * kb : 1 + kb);
    if (cost < least) {
      least = cost;
      fb = i;
    }
  }
  const int kb = fock[fb].kb;
  const size_t fsm = sizeof(double) * (2 * (size_t)X.nq * D.nn + 2 * (size_t)X.nq * kb);
  if ((err = smem_limit(fock[fb].fn, fsm)) != cudaSuccess) return err;
  fock[fb].fn<<<dim3((X.npair + kb - 1) / kb, D.nel, nout), ((ntri + 31) / 32) * 32, fsm, st>>>(D, X, S, Ha, Hb);
  if (energies) dxc_energy<<<1, 512, 0, st>>>(S.epart, D.nel * nblk, energies);
  return cudaGetLastError();
}

}  // namespace hfg
