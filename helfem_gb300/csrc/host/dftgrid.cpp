// Host tables of the atomic DFT grid (src/atomic/dftgrid.cpp:470-576,
// src/general/angular.cpp:21-70): the element radial rule (modified
// Gauss-Chebyshev, nquad points), the angular product rule (ldft Chebyshev
// points in cos(theta) x mdft uniform phi points), the radial functions and
// their derivatives at the radial points, and the theta and phi factors that
// let the device evaluate the density and the Fock matrix in separable form.
#include <cmath>
#include <stdexcept>

#include "atom.hpp"

namespace hfg {
namespace {

// normalised associated Legendre Theta_l^m(x), m >= 0, Condon-Shortley phase
double theta_lm(int l, int m, double x) {
  if (m > l) return 0.0;
  const double s = std::sqrt(std::max((1.0 - x) * (1.0 + x), 0.0));
  double c = std::sqrt((2.0 * m + 1.0) / (4.0 * M_PI));
  for (int k = 1; k <= m; ++k) c *= std::sqrt((2.0 * k - 1.0) / (2.0 * k));
  double pmm = ((m & 1) ? -1.0 : 1.0) * c * std::pow(s, m);
  if (l == m) return pmm;
  double pm1 = x * std::sqrt(2.0 * m + 3.0) * pmm;
  if (l == m + 1) return pm1;
  double p2 = pmm, p1 = pm1;
  for (int ll = m + 2; ll <= l; ++ll) {
    const double a = std::sqrt((4.0 * ll * ll - 1.0) / ((double)ll * ll - (double)m * m));
    const double b = std::sqrt(((ll - 1.0) * (ll - 1.0) - (double)m * m) / (4.0 * (ll - 1.0) * (ll - 1.0) - 1.0));
    const double p = a * (x * p1 - b * p2);
    p2 = p1;
    p1 = p;
  }
  return p1;
}

}  // namespace

void ylm(int l, int m, double cth, double phi, double& re, double& im) {
  if (std::abs(m) > l) { re = im = 0.0; return; }
  const int am = std::abs(m);
  double t = theta_lm(l, am, cth);
  if (m < 0 && (am & 1)) t = -t;  // Y_l^{-m} = (-1)^m conj(Y_l^m)
  re = t * std::cos(m * phi);
  im = t * std::sin(m * phi);
}

void AtomHost::build_dft_grid(int ld, int md) {
  int mmx = 0;
  for (int m : mval) mmx = std::max(mmx, std::abs(m));
  ldft = ld > 0 ? ld : 4 * lmax + 12;
  mdft = md > 0 ? md : 4 * mmx + 12;
  std::vector<double> xc, wc;
  cheb_rule(ldft, xc, wc);
  nap = ldft * mdft;
  const double dphi = 2.0 * M_PI / mdft;
  xc_wth.assign(ldft, 0.0);
  xc_isin.assign(ldft, 0.0);
  for (int i = 0; i < ldft; ++i) {
    xc_wth[i] = wc[i] * dphi;
    xc_isin[i] = 1.0 / std::sqrt((1.0 - xc[i]) * (1.0 + xc[i]));
  }
  // Y_l^m = T(theta) e^{i m phi}: the theta factors and their derivatives
  // dY/dtheta = m cot(theta) Y_l^m + sqrt((l-m)(l+m+1)) e^{-i phi} Y_l^{m+1}
  std::vector<double> T((size_t)nang * ldft), dT((size_t)nang * ldft);
  for (int al = 0; al < nang; ++al) {
    const int l = lval[al], m = mval[al];
    for (int i = 0; i < ldft; ++i) {
      double y, im;
      ylm(l, m, xc[i], 0.0, y, im);
      double d = m * xc[i] * xc_isin[i] * y;
      if (m < l) {
        double u;
        ylm(l, m + 1, xc[i], 0.0, u, im);
        d += std::sqrt((double)(l - m) * (l + m + 1)) * u;
      }
      T[al * (size_t)ldft + i] = y;
      dT[al * (size_t)ldft + i] = d;
    }
  }
  // unordered pairs al <= be in ascending k = |m_al - m_be|
  xc_kmax = 0;
  for (int al = 0; al < nang; ++al)
    for (int be = al; be < nang; ++be) xc_kmax = std::max(xc_kmax, std::abs(mval[al] - mval[be]));
  xc_pair.clear();
  xc_kptr.assign(1, 0);
  for (int k = 0; k <= xc_kmax; ++k) {
    for (int be = 0; be < nang; ++be)
      for (int al = 0; al <= be; ++al) {
        const int dm = mval[al] - mval[be];
        if (std::abs(dm) != k) continue;
        xc_pair.push_back(al);
        xc_pair.push_back(be);
        xc_pair.push_back((dm > 0 ? 1 : -1) * (mval[al] + mval[be]));
      }
    xc_kptr.push_back((int)xc_pair.size() / 3);
  }
  const int np = (int)xc_pair.size() / 3;
  xc_npair = np;
  xc_W.assign((size_t)np * ldft, 0.0);
  xc_Wt.assign((size_t)np * ldft, 0.0);
  xc_Wd.assign((size_t)np * ldft, 0.0);
  for (int p = 0; p < np; ++p) {
    const double *ta = &T[(size_t)xc_pair[3 * p] * ldft], *tb = &T[(size_t)xc_pair[3 * p + 1] * ldft];
    const double *da = &dT[(size_t)xc_pair[3 * p] * ldft], *db = &dT[(size_t)xc_pair[3 * p + 1] * ldft];
    for (int i = 0; i < ldft; ++i) {
      xc_W[(size_t)p * ldft + i] = ta[i] * tb[i];
      xc_Wt[(size_t)p * ldft + i] = da[i] * tb[i] + ta[i] * db[i];
      xc_Wd[(size_t)p * ldft + i] = da[i] * tb[i] - ta[i] * db[i];
    }
  }
  // phi = 0 .. pi: the density is even in phi, so the points beyond pi repeat
  // those of the first half (weight 2)
  xc_nphi = mdft / 2 + 1;
  xc_phw.assign(xc_nphi, 2.0);
  xc_phw[0] = 1.0;
  if (mdft % 2 == 0) xc_phw[mdft / 2] = 1.0;
  xc_cos.assign((size_t)(xc_kmax + 1) * xc_nphi, 0.0);
  xc_sin.assign((size_t)(xc_kmax + 1) * xc_nphi, 0.0);
  for (int k = 0; k <= xc_kmax; ++k)
    for (int j = 0; j < xc_nphi; ++j) {
      xc_cos[(size_t)k * xc_nphi + j] = std::cos(k * (j * dphi));
      // exactly 0 at phi = 0 and pi
      xc_sin[(size_t)k * xc_nphi + j] = xc_phw[j] == 1.0 ? 0.0 : std::sin(k * (j * dphi));
    }
  // radial side
  const int nn = rad.nn, nel = rad.nel;
  std::vector<double> xq, wq;
  cheb_rule(nquad, xq, wq);
  xc_r.assign((size_t)nel * nquad, 0.0);
  xc_wr.assign((size_t)nel * nquad, 0.0);
  xc_R.assign((size_t)nel * nquad * nn, 0.0);
  xc_dR.assign((size_t)nel * nquad * nn, 0.0);
  for (int e = 0; e < nel; ++e) {
    std::vector<double> Rv, dRv;
    rad.R(e, xq, Rv);
    rad.dR(e, xq, dRv);
    for (int q = 0; q < nquad; ++q) {
      const double r = rad.mid(e) + rad.sf(e) * xq[q];
      xc_r[(size_t)e * nquad + q] = r;
      xc_wr[(size_t)e * nquad + q] = rad.sf(e) * wq[q] * r * r;
      for (int p = 0; p < nn; ++p) {
        xc_R[((size_t)e * nquad + q) * nn + p] = Rv[q + (size_t)p * nquad];
        xc_dR[((size_t)e * nquad + q) * nn + p] = dRv[q + (size_t)p * nquad];
      }
    }
  }
}

}  // namespace hfg
