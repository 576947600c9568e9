// Exchange-correlation energy densities (per volume) in spin-resolved form
// with their analytic first derivatives, each functional in the fewest
// variables it depends on (one spin density and its gradient for exchange;
// n, zeta and the total gradient for correlation).
//
// Restated from the published papers (the reference evaluates them through
// libxc, src/general/dftgrid_common.cpp:98-255; libxc is not used here):
//   Slater/Dirac exchange                                   (libxc id 1)
//   VWN5 correlation, Vosko-Wilk-Nusair, CJP 58, 1200 (1980)      (id 7)
//   PW92 correlation, Perdew-Wang, PRB 45, 13244 (1992)            (id 12)
//   PBE exchange / correlation, Perdew-Burke-Ernzerhof, PRL 77, 3865
//   (1996); correlation built on PW92 with the more precise constants   (101, 130)
//
// Every operation here is on the FP64 pipe (1/64 of the FP32 rate), which is
// what bounds the XC point kernels: fractional powers are cube roots (a cbrt
// costs about a fifth of a pow), and a restricted point (POL = false, zeta =
// 0 exactly) skips the terms that zeta multiplies, which vanish there with
// their derivatives.
#pragma once

#include <cuda_runtime.h>

namespace hfg {
namespace xcf {

constexpr double PI = 3.14159265358979323846;

// energy density e and de/d(rho_a, rho_b, sigma_aa, sigma_ab, sigma_bb)
struct XcOut {
  double e, va, vb, vaa, vab, vbb;
};

// quantities of zeta, from opz = 1 + zeta = 2 rho_a / n and omz = 1 - zeta =
// 2 rho_b / n, formed from the spin densities rather than by subtracting
// zeta from one (which loses the relative precision of a minority spin)
struct Spin {
  double z, opz, omz, copz, comz;  // copz = cbrt(opz)
  double f, df;                    // f(zeta), f'(zeta)
};
template <bool POL>
__device__ __forceinline__ Spin spin_of(double ra, double rb, double in) {
  Spin s = {0.0, 1.0, 1.0, 1.0, 1.0, 0.0, 0.0};
  if (POL) {
    const double den = 1.0 / (2.5198420997897464 - 2.0);  // 2^{4/3} - 2
    s.z = (ra - rb) * in;
    s.opz = 2.0 * ra * in;
    s.omz = 2.0 * rb * in;
    s.copz = ::cbrt(s.opz);
    s.comz = ::cbrt(s.omz);
    s.f = (s.opz * s.copz + s.omz * s.comz - 2.0) * den;
    s.df = (4.0 / 3.0) * (s.copz - s.comz) * den;
  }
  return s;
}

// eps(rs, zeta) from its three branches (value, d/drs each):
// eP + ac f/f''(0) (1 - z^4) + (eF - eP) f z^4
__device__ __forceinline__ void interpolate(const Spin& s, double ifpp, const double (&P)[2], const double (&F)[2],
                                            const double (&A)[2], double& eps, double& drs, double& dz) {
  const double z3 = s.z * s.z * s.z, z4 = z3 * s.z;
  const double wa = s.f * (1.0 - z4) * ifpp, wf = s.f * z4;
  eps = P[0] + A[0] * wa + (F[0] - P[0]) * wf;
  drs = P[1] + A[1] * wa + (F[1] - P[1]) * wf;
  dz = A[0] * ifpp * (s.df * (1.0 - z4) - 4.0 * s.f * z3) + (F[0] - P[0]) * (s.df * z4 + 4.0 * s.f * z3);
}

// ---------------------------------------------------------------- Slater x
__device__ __forceinline__ void slater_x(double r, double& e, double& v) {
  const double c = -0.75 * 1.2407009817988531;  // (6/pi)^{1/3}
  const double cb = ::cbrt(r);
  e += c * r * cb;
  v += (4.0 / 3.0) * c * cb;
}

// ------------------------------------------------------------------- VWN5
// value and d/drs (x = sqrt(rs), dx/drs = 1/(2x))
__device__ __forceinline__ void vwn_eps(double x, double A, double b, double c, double x0, double (&o)[2]) {
  const double X = x * x + b * x + c, iX = 1.0 / X;
  const double X0 = x0 * x0 + b * x0 + c;
  const double Q = ::sqrt(4.0 * c - b * b);
  const double u = 2.0 * x + b, at = ::atan(Q / u), dat = -0.5 * Q * iX;  // u^2 + Q^2 = 4 X
  const double k = b * x0 / X0, k1 = 2.0 * b / Q, k2 = 2.0 * (b + 2.0 * x0) / Q;
  const double y = x - x0;
  o[0] = A * (::log(x * x * iX) + k1 * at - k * (::log(y * y * iX) + k2 * at));
  const double dx = 2.0 / x - u * iX + k1 * dat - k * (2.0 / y - u * iX + k2 * dat);
  o[1] = A * dx * 0.5 / x;
}
template <bool POL>
__device__ __forceinline__ void vwn5(double rs, const Spin& s, double& eps, double& drs, double& dz) {
  const double x = ::sqrt(rs);
  double P[2], F[2], A[2];
  vwn_eps(x, 0.0310907, 3.72744, 12.9352, -0.10498, P);
  if (!POL) {
    eps = P[0];
    drs = P[1];
    dz = 0.0;
    return;
  }
  vwn_eps(x, 0.01554535, 7.06042, 18.0578, -0.32500, F);
  vwn_eps(x, -1.0 / (6.0 * PI * PI), 1.13107, 13.0045, -0.0047584, A);
  interpolate(s, 9.0 * (1.2599210498948732 - 1.0) / 4.0, P, F, A, eps, drs, dz);
}

// ------------------------------------------------------------------- PW92
__device__ __forceinline__ void pw_G(double rs, double srs, double A, double a1, double b1, double b2, double b3,
                                     double b4, double (&o)[2]) {
  const double den = 2.0 * A * (b1 * srs + b2 * rs + b3 * rs * srs + b4 * rs * rs);
  const double dd = 2.0 * A * (0.5 * b1 / srs + b2 + 1.5 * b3 * srs + 2.0 * b4 * rs);
  const double L = ::log(1.0 + 1.0 / den), g = -2.0 * A * (1.0 + a1 * rs);
  o[0] = g * L;
  o[1] = -2.0 * A * a1 * L - g * dd / (den * (den + 1.0));
}
template <bool POL>
__device__ __forceinline__ void pw92(double rs, const Spin& s, bool mod, double& eps, double& drs, double& dz) {
  const double srs = ::sqrt(rs);
  double P[2], F[2], A[2];
  pw_G(rs, srs, mod ? 0.0310907 : 0.031091, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294, P);
  if (!POL) {
    eps = P[0];
    drs = P[1];
    dz = 0.0;
    return;
  }
  pw_G(rs, srs, mod ? 0.01554535 : 0.015545, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517, F);
  pw_G(rs, srs, mod ? 0.0168869 : 0.016887, 0.11125, 10.357, 3.6231, 0.88026, 0.49671, A);
  A[0] = -A[0];
  A[1] = -A[1];
  interpolate(s, 1.0 / (mod ? 1.709920934161365617563962776245 : 1.709921), P, F, A, eps, drs, dz);
}

// n eps(rs, zeta): e, de/dn at fixed zeta and de/dzeta -> spin potentials
__device__ __forceinline__ void add_lda_c(double n, double rs, const Spin& s, double eps, double drs, double dz,
                                          XcOut& o) {
  const double vn = eps - rs * drs * (1.0 / 3.0);
  o.e += n * eps;
  o.va += vn + s.omz * dz;
  o.vb += vn - s.opz * dz;
}

// -------------------------------------------------------------------- PBE
constexpr double PBE_KAPPA = 0.804;
constexpr double PBE_MU = 0.2195149727645171;
constexpr double PBE_BETA = 0.06672455060314922;
constexpr double PBE_GAMMA = 0.031090690869654895;  // (1 - ln 2) / pi^2

// one spin of E_x[a, b] = (E_x[2 a] + E_x[2 b]) / 2
__device__ __forceinline__ void pbe_x(double r, double sss, double& e, double& v, double& vs) {
  const double n = 2.0 * r;
  const double kf = ::cbrt(3.0 * PI * PI * n);
  const double d = 2.0 * kf * n, id2 = 1.0 / (d * d);
  const double exu = (-0.75 / PI) * kf * n;
  const double s2 = 4.0 * sss * id2;
  const double q = 1.0 / (1.0 + (PBE_MU / PBE_KAPPA) * s2);
  const double Fx = (1.0 + PBE_KAPPA) - PBE_KAPPA * q, dF = PBE_MU * q * q;
  e += 0.5 * exu * Fx;
  v += (exu / n) * ((4.0 / 3.0) * Fx - (8.0 / 3.0) * s2 * dF);
  vs += 2.0 * exu * dF * id2;
}

template <bool POL>
__device__ __forceinline__ void pbe_c(double n, double cn, double in, double rs, const Spin& s, double sig,
                                      XcOut& o) {
  constexpr double BG = PBE_BETA / PBE_GAMMA;
  double ec, drs, dz;
  pw92<POL>(rs, s, true, ec, drs, dz);
  const double ecn = -rs * drs * in * (1.0 / 3.0);  // d ec / dn
  const double kf = 3.0936677262801355 * cn;          // (3 pi^2)^{1/3} n^{1/3}
  double phi = 1.0, dphi = 0.0;
  if (POL) {
    phi = 0.5 * (s.copz * s.copz + s.comz * s.comz);
    dphi = (1.0 / 3.0) * (1.0 / s.copz - 1.0 / s.comz);
  }
  const double p2 = phi * phi, g3 = PBE_GAMMA * p2 * phi, ig3 = 1.0 / g3;
  // t^2 = sig / (2 phi ks n)^2, ks^2 = 4 kf / pi
  const double t2c = (PI / 16.0) / (p2 * kf * n * n), t2 = sig * t2c;
  const double E = ::exp(-ec * ig3), iE = 1.0 / (E - 1.0);
  const double A = BG * iE;
  const double Aec = A * E * iE * ig3;  // dA/dec; dA/dphi = -3 ec/phi of it
  const double y = A * t2;
  const double iD = 1.0 / (1.0 + y + y * y), g = (1.0 + y) * iD, dg = -y * (2.0 + y) * iD * iD;
  const double u = BG * t2 * g, L = ::log(1.0 + u), gu = g3 / (1.0 + u);
  const double H = g3 * L;
  const double Ht = gu * BG * (g + y * dg);      // dH/dt2 at fixed A
  const double HA = gu * BG * t2 * t2 * dg;      // dH/dA
  const double Hec = HA * Aec;
  const double Hn = Hec * ecn - (7.0 / 3.0) * Ht * t2 * in;
  double ez = 0.0;
  if (POL) {
    const double iphi = 1.0 / phi;
    const double Hphi = (3.0 * H - 2.0 * Ht * t2 - 3.0 * ec * Hec) * iphi;
    ez = dz * (1.0 + Hec) + Hphi * dphi;
  }
  const double vn = ec + H + n * (ecn + Hn);
  o.e += n * (ec + H);
  o.va += vn + s.omz * ez;
  o.vb += vn - s.opz * ez;
  const double vs = n * Ht * t2c;
  o.vaa += vs;
  o.vab += 2.0 * vs;
  o.vbb += vs;
}

}  // namespace xcf

// energy density and its partial derivatives of the exchange + correlation
// pair at one point; ids as in hfg_xc. POL = false: rb == ra and the three
// sigma are equal (the b results repeat the a ones). Not inlined: called from
// several branches of the point kernels.
template <bool POL>
__device__ __noinline__ xcf::XcOut xc_eval(int xid, int cid, double ra, double rb, double saa, double sab,
                                           double sbb) {
  using namespace xcf;
  XcOut o = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const double n = ra + rb, in = 1.0 / n, cn = ::cbrt(n);
  const double rs = 0.62035049089940002 / cn;  // (3 / (4 pi))^{1/3} n^{-1/3}
  const bool corr = xid == 7 || xid == 12 || xid == 130 || cid == 7 || cid == 12 || cid == 130;
  const Spin s = POL && corr ? spin_of<POL>(ra, rb, in) : Spin{0.0, 1.0, 1.0, 1.0, 1.0, 0.0, 0.0};
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    const int id = k ? cid : xid;
    double eps, drs, dz;
    switch (id) {
      case 1: {
        double e = 0.0;
        slater_x(ra, e, o.va);
        if (POL) slater_x(rb, e, o.vb); else { e *= 2.0; o.vb = o.va; }
        o.e += e;
        break;
      }
      case 7:
        vwn5<POL>(rs, s, eps, drs, dz);
        add_lda_c(n, rs, s, eps, drs, dz, o);
        break;
      case 12:
        pw92<POL>(rs, s, false, eps, drs, dz);
        add_lda_c(n, rs, s, eps, drs, dz, o);
        break;
      case 101: {
        double e = 0.0, v = 0.0, vs = 0.0;
        pbe_x(ra, saa, e, v, vs);
        o.va += v;
        o.vaa += vs;
        if (POL) {
          v = vs = 0.0;
          pbe_x(rb, sbb, e, v, vs);
        } else {
          e *= 2.0;
        }
        o.vb += v;
        o.vbb += vs;
        o.e += e;
        break;
      }
      case 130: pbe_c<POL>(n, cn, in, rs, s, saa + 2.0 * sab + sbb, o); break;
      default: break;
    }
  }
  return o;
}

}  // namespace hfg
