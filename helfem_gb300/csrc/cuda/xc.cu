// XC potential on the atomic DFT grid, plain FP64.
//
// Restates DFTGrid::eval_Fxc and its worker (src/atomic/dftgrid.cpp:51-128,
// 304-359, 470-576, 591-712) and the split real/imaginary accumulations of
// src/general/dftgrid_common.h:128-217, in separable form. On element e with
// radial points q, polar points t and azimuthal points f (a product rule) the
// basis functions are phi_{alpha i} = R_i(r_q) T_alpha(t) e^{i m_alpha f}.
// Every quantity the reference forms from dense (functions x points) matrices
// factorises over unordered pairs p = (a <= b) with k = |m_a - m_b|:
//   rho     = sum_k cos(k f) sum_{p of k} Ds_p(q) W_p(t)
//   d_r rho = 2 sum_k cos(k f) sum_{p of k} Dr_p(q) W_p(t)
//   d_t rho = (2/r) sum_k cos(k f) sum_{p of k} (Ds_p Wt_p + Dd_p Wd_p)/2
//   d_f rho = (2/(r sin t)) sum_k sin(k f) sum_{p of k} -(k Ds_p + s_p Dd_p) W_p / 2
// with Ds = R^T (P_ab + P_ba^T) R, Dr = dR^T (P_ab + P_ba) R, Dd =
// R^T (P_ab - P_ba^T) R (zero for a symmetric density; a = b: Ds and Dr from
// P_aa alone), W = T_a T_b, Wt/Wd = T'_a T_b +- T_a T'_b, s = sign(m_a - m_b)
// (m_a + m_b). The Fock matrix is symmetric, and each of its tiles (a, b) is
// symmetric in (i, j) too:
//   V_{ai,bj} = sum_q R_i R_j S_p + (dR_i R_j + R_i dR_j) Ur_p,
//   S_p  = sum_t [(F0_k - k Fp_k) W_p + Ft_k Wt_p],  Ur_p = sum_t Fr_k W_p,
//   Fc_k(q,t) = sum_f f_c cos(k f)  (sin for the azimuthal component)
// with per-point weights f_0 = w v_rho, f_c = w (2 v_ss grad_c rho_s +
// v_ab grad_c rho_s') / scale_c (dftgrid.cpp:321-334). The same quadrature
// sums as the reference.
//
// The FP64 pipe bounds all of it (2 multiply-adds per cycle and SM), so the
// split is the one with the fewest FP64 operations: polar and azimuthal sums
// apart, half of the pairs, half of the azimuth (the density is even in f),
// one azimuthal point where no pair of k > 0 has a density (a density that
// does not mix m). On the Kr basis (40 elements, l <= 2, 75 x 20 x 20 points
// per element, PBE, two spins) the per-point sums over the 81 ordered pairs
// that this replaced took 9.69 ms a call; this takes 1.25 ms (density that
// does not mix m). 17 elements of 10 nodes, l <= 1, LDA: 0.397 -> 0.092 ms.
//
// Kernels: xc_rad (Ds, Dr, Dd), xc_point (density, functional, S and Ur,
// energy partials), xc_fock (V, shared-boundary corner as in J), xc_energy
// (fixed-order reduction).
#include <algorithm>
#include <cfloat>

#include "devatom.cuh"
#include "reduce.cuh"
#include "smem_limit.hpp"
#include "xc_func.cuh"

namespace hfg {
namespace {

__device__ __forceinline__ bool gvalid(const DevAtom& A, int g) { return g >= 0 && g < A.nrad; }

// Ds, Dr, Dd of pair p on element e; grid (nel, npair, nsd), one thread per
// radial point. With Q the symmetric part of (P_ab + P_ba^T) and Z the
// antisymmetric part of (P_ab + P_ba) (half of both for a = b), t = Q R gives
// Ds = t.R and Dr = t.dR + dR^T Z R: one matrix product for both where the
// density is symmetric (Z = 0 and P_ab = P_ba^T, tested per tile).
__global__ void xc_rad(DevAtom A, DevXC X, XcScratch S, const double* __restrict__ P0,
                       const double* __restrict__ P1) {
  const int e = blockIdx.x, p = blockIdx.y, s = blockIdx.z;
  const int nn = A.nn, nq = X.nquad;
  const int al = X.pair[3 * p], be = X.pair[3 * p + 1];
  const double* P = s ? P1 : P0;
  extern __shared__ double sm[];
  double* Pa = sm;                 // nn*nn: P_ab
  double* Pb = Pa + nn * nn;       // P_ba
  double* R = Pb + nn * nn;        // nq*nn
  double* dR = R + nq * nn;        // nq*nn
  for (int idx = threadIdx.x; idx < nn * nn; idx += blockDim.x) {
    const int i = idx % nn, j = idx / nn;
    const int gi = gfun(A, e, i), gj = gfun(A, e, j);
    const bool ok = gvalid(A, gi) && gvalid(A, gj);
    Pa[idx] = ok ? P[(size_t)(be * A.nrad + gj) * A.nbf + (size_t)al * A.nrad + gi] : 0.0;
    Pb[idx] = ok ? P[(size_t)(al * A.nrad + gj) * A.nbf + (size_t)be * A.nrad + gi] : 0.0;
  }
  for (int idx = threadIdx.x; idx < nq * nn; idx += blockDim.x) {
    R[idx] = X.R[(size_t)e * nq * nn + idx];
    dR[idx] = X.dR[(size_t)e * nq * nn + idx];
  }
  __syncthreads();
  bool odd = false;
  for (int idx = threadIdx.x; idx < nn * nn; idx += blockDim.x) {
    const int tr = idx / nn + (idx % nn) * nn;
    odd |= Pa[idx] != Pb[tr];
  }
  const bool general = __syncthreads_or(odd);
  const double half = al == be ? 0.25 : 0.5;
  const size_t np = X.npair, base = (((size_t)s * A.nel + e) * nq) * 3 * np + p;
  for (int q = threadIdx.x; q < nq; q += blockDim.x) {
    const double* Rq = R + q * nn;
    const double* dRq = dR + q * nn;
    double d = 0.0, dr = 0.0, dd = 0.0;
    if (!general) {  // P_ba = P_ab^T: Q = P_ab + P_ab^T
      for (int j = 0; j < nn; ++j) {
        double t = 0.0;
        for (int i = 0; i < nn; ++i) t += (Pa[i + j * nn] + Pb[i + j * nn]) * Rq[i];
        d += t * Rq[j];
        dr += t * dRq[j];
      }
      if (al == be) {
        d *= 0.5;
        dr *= 0.5;
      }
    } else {
      for (int j = 0; j < nn; ++j) {
        double t = 0.0, z = 0.0, u = 0.0;
        for (int i = 0; i < nn; ++i) {
          const double ij = Pa[i + j * nn], ji = Pa[j + i * nn], bij = Pb[i + j * nn], bji = Pb[j + i * nn];
          t += half * ((ij + bji) + (ji + bij)) * Rq[i];
          z += half * ((ij + bij) - (ji + bji)) * dRq[i];
          u += (ij - bji) * Rq[i];
        }
        d += t * Rq[j];
        dr += t * dRq[j] + z * Rq[j];
        dd += u * Rq[j];
      }
    }
    const size_t o = base + (size_t)q * 3 * np;
    S.D[o] = d;
    S.D[o + np] = dr;
    S.D[o + 2 * np] = al == be ? 0.0 : dd;
  }
}

// Shared memory of xc_point in doubles for qb radial points and tb polar
// points at a time
__host__ __device__ inline size_t xc_point_doubles(const DevXC& X, int nsd, int nc, int qb, int tb) {
  return (size_t)qb * nsd * X.npair * (3 + 2) + (size_t)qb * tb * nsd * nc * ((X.kmax + 1) + X.nphi);
}

// Density, functional and the angular sums of qb radial points of element e;
// grid (nel, ceil(nquad/qb)). Polar points in chunks of tb. One point per
// thread for the functional, which is the largest part where the density
// depends on the azimuth; several radial points per CTA keep its warps filled
// where it does not.
template <bool GGA, bool POL>
__global__ void __launch_bounds__(256) xc_point(DevAtom A, DevXC X, XcScratch S, int xid, int cid, int mdft, int qb,
                                                int tb, double thr) {
  constexpr int NS = POL ? 2 : 1, NC = GGA ? 4 : 1;
  const int e = blockIdx.x, q0 = blockIdx.y * qb;
  const int nq = X.nquad, np = X.npair, nth = X.nth, nph = X.nphi, K = X.kmax + 1;
  const int nqb = min(qb, nq - q0);
  extern __shared__ double sm[];
  double* D = sm;                                  // [qi][s][3][np]
  double* Ua = D + (size_t)qb * NS * 3 * np;       // [qi][s][np][2]
  double* C = Ua + (size_t)qb * NS * np * 2;       // [qi][s][c][tb][K]
  double* F = C + (size_t)qb * NS * NC * tb * K;   // [qi][s][c][tb][nph]
  __shared__ double red[32];
  const int tid = threadIdx.x, nt = blockDim.x;
  bool odd = false;
  for (int idx = tid; idx < nqb * NS * 3 * np; idx += nt) {
    const int p3 = idx % (3 * np), s = (idx / (3 * np)) % NS, qi = idx / (3 * np * NS);
    const double v = S.D[(((size_t)s * A.nel + e) * nq + q0 + qi) * 3 * np + p3];
    D[idx] = v;
    odd |= p3 >= 2 * np && v != 0.0;
  }
  for (int idx = tid; idx < nqb * NS * np * 2; idx += nt) Ua[idx] = 0.0;
  const bool general = __syncthreads_or(odd);  // a density that is not symmetric
  double esum = 0.0, nsum = 0.0;
  for (int t0 = 0; t0 < nth; t0 += tb) {
    const int nb = min(tb, nth - t0);
    // ---- sums over the pairs of each k ----
    bool mix = false;
    for (int idx = tid; idx < nqb * NS * nb * K; idx += nt) {
      const int k = idx % K, t = (idx / K) % nb, qs = idx / (K * nb);  // qs = qi*NS + s
      const double* Dq = D + (size_t)qs * 3 * np;
      double c0 = 0.0, c1 = 0.0, c2 = 0.0, c3 = 0.0;
      for (int p = X.kptr[k]; p < X.kptr[k + 1]; ++p) {
        const double w = X.W[(size_t)p * nth + t0 + t];
        c0 += Dq[p] * w;
        if (GGA) {
          c1 += Dq[np + p] * w;
          c2 += Dq[p] * X.Wt[(size_t)p * nth + t0 + t];
          if (general) {
            c2 += Dq[2 * np + p] * X.Wd[(size_t)p * nth + t0 + t];
            c3 += Dq[2 * np + p] * w * (double)X.pair[3 * p + 2];
          }
        }
      }
      double* Cq = C + ((size_t)qs * NC * tb + t) * K + k;
      Cq[0] = c0;
      mix |= k > 0 && c0 != 0.0;
      if (GGA) {
        c2 *= 0.5;
        c3 = -0.5 * (k * c0 + c3);
        Cq[(size_t)tb * K] = c1;
        Cq[(size_t)2 * tb * K] = c2;
        Cq[(size_t)3 * tb * K] = c3;
        mix |= k > 0 && (c1 != 0.0 || c2 != 0.0 || c3 != 0.0);
      }
    }
    const bool dep = __syncthreads_or(mix);  // the density depends on the azimuth
    const int nj = dep ? nph : 1, nk = dep ? K : 1;
    // ---- the functional at every point ----
    for (int idx = tid; idx < nqb * nb * nj; idx += nt) {
      const int j = idx % nj, t = (idx / nj) % nb, qi = idx / (nj * nb);
      const double r = X.r[(size_t)e * nq + q0 + qi], ir = 1.0 / r, isin = X.isin[t0 + t];
      double rho[2], g[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const double* Cq = C + ((size_t)(qi * NS + s) * NC * tb + t) * K;
        double a0 = Cq[0], a1 = 0.0, a2 = 0.0, a3 = 0.0;
        if (GGA) {
          a1 = Cq[(size_t)tb * K];
          a2 = Cq[(size_t)2 * tb * K];
        }
        for (int k = 1; k < nk; ++k) {
          const double co = X.cosk[(size_t)k * nph + j];
          a0 += co * Cq[k];
          if (GGA) {
            a1 += co * Cq[(size_t)tb * K + k];
            a2 += co * Cq[(size_t)2 * tb * K + k];
            a3 += X.sink[(size_t)k * nph + j] * Cq[(size_t)3 * tb * K + k];
          }
        }
        rho[s] = a0;
        if (GGA) {
          g[s][0] = 2.0 * a1;
          g[s][1] = 2.0 * a2 * ir;
          g[s][2] = 2.0 * a3 * ir * isin;
        }
      }
      if (!POL) {  // restricted: equal spin densities from the total P
        rho[0] *= 0.5;
        rho[1] = rho[0];
        for (int c = 0; c < 3; ++c) {
          g[0][c] *= 0.5;
          g[1][c] = g[0][c];
        }
      }
      const double w = X.wth[t0 + t] * X.wr[(size_t)e * nq + q0 + qi] * (dep ? X.phw[j] : (double)mdft);
      const double n = rho[0] + rho[1];
      xcf::XcOut v = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      if (n >= thr) {  // libxc density threshold: below it the point contributes nothing
        const double ra = fmax(rho[0], 0.5 * thr), rb = fmax(rho[1], 0.5 * thr);
        double saa = 0.0, sab = 0.0, sbb = 0.0;
        if (GGA) {
          saa = g[0][0] * g[0][0] + g[0][1] * g[0][1] + g[0][2] * g[0][2];
          sab = POL ? g[0][0] * g[1][0] + g[0][1] * g[1][1] + g[0][2] * g[1][2] : saa;
          sbb = POL ? g[1][0] * g[1][0] + g[1][1] * g[1][1] + g[1][2] * g[1][2] : saa;
        }
        v = xc_eval<POL>(xid, cid, ra, rb, saa, sab, sbb);
      }
      esum += w * v.e;
      nsum += w * n;
      const double scale[3] = {1.0, ir, isin * ir};
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        double* Fq = F + ((size_t)(qi * NS + s) * NC * tb + t) * nph + j;
        Fq[0] = w * (s ? v.vb : v.va);
        if (GGA) {
          const double vss = s ? v.vbb : v.vaa;
#pragma unroll
          for (int c = 0; c < 3; ++c)
            Fq[(size_t)(c + 1) * tb * nph] = w * (2.0 * vss * g[s][c] + v.vab * g[1 - s][c]) * scale[c];
        }
      }
    }
    __syncthreads();
    // ---- azimuthal sums, in place over the density coefficients ----
    for (int idx = tid; idx < nqb * NS * NC * nb * K; idx += nt) {
      const int k = idx % K, t = (idx / K) % nb, c = (idx / (K * nb)) % NC, qs = idx / (K * nb * NC);
      const double* Fq = F + (((size_t)qs * NC + c) * tb + t) * nph;
      double v = 0.0;
      if (!dep) {
        v = (c < 3 && k % mdft == 0) ? Fq[0] : 0.0;
      } else {
        const double* tr = (c == 3 ? X.sink : X.cosk) + (size_t)k * nph;
        for (int j = 0; j < nph; ++j) v += Fq[j] * tr[j];
      }
      C[(((size_t)qs * NC + c) * tb + t) * K + k] = v;
    }
    __syncthreads();
    // ---- polar sums per pair ----
    for (int idx = tid; idx < nqb * NS * np; idx += nt) {
      const int p = idx % np, qs = idx / np;
      int k = 0;
      while (p >= X.kptr[k + 1]) ++k;
      if (!dep && k % mdft != 0) continue;
      const double* Cq = C + (size_t)qs * NC * tb * K + k;
      double sp = 0.0, ur = 0.0;
      for (int t = 0; t < nb; ++t) {
        const double w = X.W[(size_t)p * nth + t0 + t];
        if (GGA) {
          const double f = Cq[(size_t)t * K] - (double)k * Cq[(size_t)(3 * tb + t) * K];
          sp += f * w + Cq[(size_t)(2 * tb + t) * K] * X.Wt[(size_t)p * nth + t0 + t];
          ur += Cq[(size_t)(tb + t) * K] * w;
        } else {
          sp += Cq[(size_t)t * K] * w;
        }
      }
      Ua[2 * idx] += sp;
      Ua[2 * idx + 1] += ur;
    }
    __syncthreads();
  }
  for (int idx = tid; idx < nqb * NS * np * 2; idx += nt) {
    const int qi = idx % nqb, c = (idx / nqb) % 2, p = (idx / (2 * nqb)) % np, s = idx / (2 * nqb * np);
    S.U[((((size_t)s * A.nel + e) * np + p) * 2 + c) * nq + q0 + qi] = Ua[((size_t)(qi * NS + s) * np + p) * 2 + c];
  }
  esum = block_sum(esum, red);
  nsum = block_sum(nsum, red);
  if (tid == 0) {
    S.epart[((size_t)e * gridDim.y + blockIdx.y) * 2 + 0] = esum;
    S.epart[((size_t)e * gridDim.y + blockIdx.y) * 2 + 1] = nsum;
  }
}

// Tile of pair p on element e, written to the (a, b) and (b, a) blocks: the
// upper triangle of V = R^T G + dR^T H (G = R S + dR Ur, H = R Ur), two
// multiply-adds per entry and radial point. grid (npair, nel, nout)
__global__ void xc_fock(DevAtom A, DevXC X, XcScratch S, int gga, double* __restrict__ H0, double* __restrict__ H1) {
  const int p = blockIdx.x, e = blockIdx.y, s = blockIdx.z;
  const int nn = A.nn, nq = X.nquad, al = X.pair[3 * p], be = X.pair[3 * p + 1];
  double* Hm = s ? H1 : H0;
  extern __shared__ double sm[];
  double* R = sm;             // nq*nn
  double* G = R + nq * nn;    // nq*nn
  double* V = G + nq * nn;    // nn*nn
  double* dR = V + nn * nn;   // nq*nn (gga)
  double* Hq = dR + nq * nn;  // nq*nn (gga)
  __shared__ double corner;
  const double* U = S.U + (((size_t)s * A.nel + e) * X.npair + p) * 2 * nq;
  for (int idx = threadIdx.x; idx < nq * nn; idx += blockDim.x) {
    const int q = idx / nn;
    const double r = X.R[(size_t)e * nq * nn + idx], u0 = U[q];
    R[idx] = r;
    if (gga) {
      const double dr = X.dR[(size_t)e * nq * nn + idx], u1 = U[nq + q];
      dR[idx] = dr;
      G[idx] = r * u0 + dr * u1;
      Hq[idx] = r * u1;
    } else {
      G[idx] = r * u0;
    }
  }
  // the first function of element e is the last of element e-1: its diagonal
  // value there
  if (threadIdx.x < 32) {
    double c = 0.0;
    if (e > 0) {
      const double* Up = S.U + (((size_t)s * A.nel + e - 1) * X.npair + p) * 2 * nq;
      for (int q = threadIdx.x; q < nq; q += 32) {
        const size_t o = ((size_t)(e - 1) * nq + q) * nn + nn - 1;
        const double r = X.R[o];
        c += r * r * Up[q] + (gga ? 2.0 * r * X.dR[o] * Up[nq + q] : 0.0);
      }
    }
    c = warp_sum(c);
    if (threadIdx.x == 0) corner = c;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < nn * (nn + 1) / 2; idx += blockDim.x) {
    // idx -> (i <= j), j-major
    int j = (int)((sqrtf(8.0f * idx + 1.0f) - 1.0f) * 0.5f);
    while (j * (j + 1) / 2 > idx) --j;
    while ((j + 1) * (j + 2) / 2 <= idx) ++j;
    const int i = idx - j * (j + 1) / 2;
    double v = 0.0, v2 = 0.0;
    if (gga)
      for (int q = 0; q < nq; ++q) {
        v += R[q * nn + i] * G[q * nn + j];
        v2 += dR[q * nn + i] * Hq[q * nn + j];
      }
    else
      for (int q = 0; q < nq; ++q) v += R[q * nn + i] * G[q * nn + j];
    v += v2;
    if (idx == 0) v += corner;
    V[i + j * nn] = v;
    V[j + i * nn] = v;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < nn * nn; idx += blockDim.x) {
    const int i = idx % nn, j = idx / nn;
    if (i == nn - 1 && j == nn - 1) continue;  // owned by the next element
    const int gi = gfun(A, e, i), gj = gfun(A, e, j);
    if (!gvalid(A, gi) || !gvalid(A, gj)) continue;
    const double v = V[idx];
    Hm[(size_t)(be * A.nrad + gj) * A.nbf + (size_t)al * A.nrad + gi] = v;
    if (al != be) Hm[(size_t)(al * A.nrad + gj) * A.nbf + (size_t)be * A.nrad + gi] = v;
  }
}

__global__ void xc_energy(const double* __restrict__ part, int n, double* out) {
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

// radial points and polar points per CTA step of xc_point: four radial points
// and every polar point where that stays within 100 KB (two CTAs per SM),
// else fewer polar points, then fewer radial points
void xc_point_shape(const DevXC& X, int nsd, int nc, int& qb, int& tb) {
  const size_t soft = 100 * 1024 / sizeof(double);
  for (qb = XC_QB; qb > 1; qb /= 2)
    if (xc_point_doubles(X, nsd, nc, qb, 1) <= soft) break;
  tb = X.nth;
  while (tb > 1 && xc_point_doubles(X, nsd, nc, qb, tb) > soft) tb = (tb + 1) / 2;
}

}  // namespace

bool xc_func_supported(int id) { return id == 0 || id == 1 || id == 7 || id == 12 || id == 101 || id == 130; }
bool xc_func_is_gga(int id) { return id == 101 || id == 130; }

cudaError_t launch_xc_fp64(const DevAtom& A, const DevXC& X, const XcScratch& S, int xid, int cid,
                           const double* Pa, const double* Pb, double* Ha, double* Hb, double* energies,
                           double thr, cudaStream_t st) {
  const bool polarized = Pb != nullptr;
  const int nsd = polarized ? 2 : 1, nout = nsd;
  const bool gga = xc_func_is_gga(xid) || xc_func_is_gga(cid);
  const int nc = gga ? 4 : 1;
  const size_t bytes = sizeof(double) * (size_t)A.nbf * A.nbf;
  cudaError_t err = cudaMemsetAsync(Ha, 0, bytes, st);
  if (err == cudaSuccess && polarized) err = cudaMemsetAsync(Hb, 0, bytes, st);
  if (err != cudaSuccess) return err;
  const size_t sm_rad = sizeof(double) * (2 * A.nn * A.nn + 2 * X.nquad * A.nn);
  if ((err = smem_limit(xc_rad, sm_rad)) != cudaSuccess) return err;
  const int tq = std::min(((X.nquad + 31) / 32) * 32, 1024);
  xc_rad<<<dim3(A.nel, X.npair, nsd), tq, sm_rad, st>>>(A, X, S, Pa, Pb);
  int qb = 1, tb = 1;
  xc_point_shape(X, nsd, nc, qb, tb);
  const size_t sm_pt = sizeof(double) * xc_point_doubles(X, nsd, nc, qb, tb);
  const int nqb = (X.nquad + qb - 1) / qb;
  auto point = polarized ? (gga ? xc_point<true, true> : xc_point<false, true>)
                         : (gga ? xc_point<true, false> : xc_point<false, false>);
  if ((err = smem_limit(point, sm_pt)) != cudaSuccess) return err;
  point<<<dim3(A.nel, nqb), 256, sm_pt, st>>>(A, X, S, xid, cid, X.mdft, qb, tb, thr);
  const size_t sm_fk = sizeof(double) * ((gga ? 4 : 2) * X.nquad * A.nn + A.nn * A.nn);
  if ((err = smem_limit(xc_fock, sm_fk)) != cudaSuccess) return err;
  xc_fock<<<dim3(X.npair, A.nel, nout), 128, sm_fk, st>>>(A, X, S, gga ? 1 : 0, Ha, Hb);
  if (energies) xc_energy<<<1, 512, 0, st>>>(S.epart, A.nel * nqb, energies);
  return cudaGetLastError();
}

}  // namespace hfg
