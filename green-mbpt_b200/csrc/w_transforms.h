// The mirror-symmetric form of the bosonic transforms (host code without CUDA, tested on the CPU).
//
// W(tau) = sum_n B[t][n] f(sum_t' F[n][t'] P0(t')) with f the solve at one frequency and F [nw][nts / 2] the forward
// transform folded onto the first half of tau.  A transform of tau points that lie symmetric about beta / 2 has equal
// rows of F at +Omega and -Omega and, those merged, W(beta - tau) = W(tau).  The matrices that a caller gives are
// that up to the round-off of their construction, a least-squares solution for the synthetic grids, so which of its
// digits agree depends on the linear algebra library.  What is compared is therefore not the matrices but what the
// form changes in W.
#pragma once

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

namespace gb200 {

// Rows of F closer than this (relative to its largest element) are one frequency.  The synthetic grids' +-Omega rows
// agree to 1e-16 to 3.5e-14; distinct frequencies differ by many orders more, and a wrong merge would show in `change`.
constexpr double MIRROR_MERGE_TOL = 1.8e-12;
// The change of the composed transform B F, relative to its largest element, up to which the form is used: 2^-39, the
// unit in which five slices hold an operand.  (B is an inverse of the F that was given, so what merging takes from F and
// what averaging takes from B nearly cancel, whatever round-off the two carry.)  The synthetic Chebyshev grids change by
// 2e-15 (beta = 10, 14 times), 5e-14 (beta = 200, 120 times), 1.8e-13 (118 times), 3e-13 (beta = 500, 160 times); W
// itself by 2e-14 to 3e-13 of its largest element where rounding P0 to 2^-39 changes it by 5e-12.  The IR-type grid of
// 110 sampled times has no such symmetry (0.4).
constexpr double MIRROR_CHANGE_TOL = 1.0 / 549755813888.0;
// The same sums with magnitudes, which bound the change of W for any f that keeps |f(x)| <= |x|: this one sees an
// asymmetry of B that B F does not show.  Synthetic grids: 2e-14 to 7e-11; the IR-type grid 9.  Limit 2^-30.
constexpr double MIRROR_BOUND_TOL = 1.0 / 1073741824.0;

struct MirrorTransforms {
  bool ok = false;     // the form may be used: the tolerances hold and everything is finite
  int nu = 0;          // merged frequencies
  double change = 0.0, bound = 0.0;  // the two figures above
  std::vector<std::complex<double>> fwd;   // [nu][nts / 2]
  std::vector<std::complex<double>> full;  // [nts][nu]: columns of B summed over the merged frequencies
  std::vector<std::complex<double>> half;  // [nts / 2][nu]: the mean of its mirrored rows
};

inline MirrorTransforms mirror_transforms(const std::complex<double>* F, const std::complex<double>* B, int nts, int nw) {
  const int nth = nts / 2;
  MirrorTransforms m;
  auto magnitude = [](std::complex<double> z) { return std::max(std::fabs(z.real()), std::fabs(z.imag())); };
  double sum = 0.0, fmax = 0.0, bmax = 0.0;  // (a sum keeps a NaN or an infinity that a maximum may drop)
  for (size_t i = 0; i < (size_t)nw * nth; ++i) {
    fmax = std::max(fmax, magnitude(F[i]));
    sum += F[i].real() + F[i].imag();
  }
  for (size_t i = 0; i < (size_t)nts * nw; ++i) sum += B[i].real() + B[i].imag();
  if (!std::isfinite(sum) || nts % 2 != 0) return m;
  // frequencies with equal rows (each joins the first such one)
  std::vector<int> group(nw, -1), first;
  for (int n = 0; n < nw; ++n) {
    for (size_t u = 0; u < first.size() && group[n] < 0; ++u) {
      bool same = true;
      for (int t = 0; same && t < nth; ++t)
        same = magnitude(F[(size_t)n * nth + t] - F[(size_t)first[u] * nth + t]) <= MIRROR_MERGE_TOL * fmax;
      if (same) group[n] = (int)u;
    }
    if (group[n] < 0) {
      group[n] = (int)first.size();
      first.push_back(n);
    }
  }
  const int nu = m.nu = (int)first.size();
  m.fwd.assign((size_t)nu * nth, 0.0);
  m.full.assign((size_t)nts * nu, 0.0);
  m.half.assign((size_t)nth * nu, 0.0);
  std::vector<int> members(nu, 0);
  for (int n = 0; n < nw; ++n) {
    ++members[group[n]];
    for (int t = 0; t < nth; ++t) m.fwd[(size_t)group[n] * nth + t] += F[(size_t)n * nth + t];
    for (int t = 0; t < nts; ++t) m.full[(size_t)t * nu + group[n]] += B[(size_t)t * nw + n];
  }
  for (int u = 0; u < nu; ++u)
    for (int t = 0; t < nth; ++t) m.fwd[(size_t)u * nth + t] *= 1.0 / members[u];
  double asym = 0.0;
  for (int t = 0; t < nth; ++t)
    for (int u = 0; u < nu; ++u) {
      const std::complex<double> a = m.full[(size_t)t * nu + u], b = m.full[(size_t)(nts - 1 - t) * nu + u];
      bmax = std::max(bmax, std::max(magnitude(a), magnitude(b)));
      asym = std::max(asym, magnitude(a - b));
      m.half[(size_t)t * nu + u] = 0.5 * (a + b);
    }
  // no mirror symmetry to speak of (the synthetic grids have 2e-12 at most): the products below are not needed
  if (!(asym <= 1e-6 * bmax)) {
    m.change = m.bound = asym / bmax;
    return m;
  }
  // out += X Y for a row X [n] and Y [n][nth], and the sum of magnitudes
  struct Acc {
    std::vector<double> re, im, mag;
    explicit Acc(int n) : re(n), im(n), mag(n) {}
    void clear() {
      std::fill(re.begin(), re.end(), 0.0);
      std::fill(im.begin(), im.end(), 0.0);
      std::fill(mag.begin(), mag.end(), 0.0);
    }
    void add(std::complex<double> x, const double* yr, const double* yi, const double* ym, int n) {
      const double xr = x.real(), xi = x.imag(), xm = std::hypot(xr, xi);
      for (int t = 0; t < n; ++t) {
        re[t] += xr * yr[t] - xi * yi[t];
        im[t] += xr * yi[t] + xi * yr[t];
        mag[t] += xm * ym[t];
      }
    }
  };
  auto planes = [&](const std::vector<std::complex<double>>& y) {
    std::vector<double> p(3 * y.size());
    for (size_t i = 0; i < y.size(); ++i) {
      p[i] = y[i].real();
      p[y.size() + i] = y[i].imag();
      p[2 * y.size() + i] = std::abs(y[i]);
    }
    return p;
  };
  std::vector<std::complex<double>> dF;  // rows that a merge moves
  std::vector<int> moved;
  for (int n = 0; n < nw; ++n) {
    if (members[group[n]] == 1) continue;
    moved.push_back(n);
    for (int t = 0; t < nth; ++t) dF.push_back(F[(size_t)n * nth + t] - m.fwd[(size_t)group[n] * nth + t]);
  }
  const std::vector<double> pf = planes(m.fwd), pd = planes(dF);
  const size_t nf = m.fwd.size(), nd = dF.size();
  // the composed transform's size, and per time the change: (full - half) fwd + B dF
  Acc s(nth), skew(nth), d(nth);
  double scale = 0.0, change = 0.0, bound = 0.0;
  for (int t = 0; t < nth; ++t) {
    s.clear();
    skew.clear();
    for (int u = 0; u < nu; ++u) {
      const double *yr = &pf[(size_t)u * nth], *yi = yr + nf, *ym = yi + nf;
      const std::complex<double> h = m.half[(size_t)t * nu + u];
      s.add(h, yr, yi, ym, nth);
      skew.add(m.full[(size_t)t * nu + u] - h, yr, yi, ym, nth);
    }
    for (int mirror = 0; mirror < 2; ++mirror) {
      const int row = mirror ? nts - 1 - t : t;
      d.clear();
      for (size_t i = 0; i < moved.size(); ++i) {
        const double *yr = &pd[i * nth], *yi = yr + nd, *ym = yi + nd;
        d.add(B[(size_t)row * nw + moved[i]], yr, yi, ym, nth);
      }
      const double sign = mirror ? -1.0 : 1.0;  // the mirrored row of full - half is minus this one
      for (int k = 0; k < nth; ++k) {
        change = std::max(change, std::hypot(sign * skew.re[k] + d.re[k], sign * skew.im[k] + d.im[k]));
        bound = std::max(bound, skew.mag[k] + d.mag[k]);
      }
    }
    for (int k = 0; k < nth; ++k) scale = std::max(scale, std::hypot(s.re[k], s.im[k]));
  }
  m.change = scale > 0.0 ? change / scale : change;
  m.bound = scale > 0.0 ? bound / scale : bound;
  m.ok = m.change <= MIRROR_CHANGE_TOL && m.bound <= MIRROR_BOUND_TOL;
  return m;
}

}  // namespace gb200
