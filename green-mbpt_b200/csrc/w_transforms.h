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

// |z| without the scaling by which std::abs guards the ends of the double range
inline double modulus(std::complex<double> z) { return std::sqrt(std::norm(z)); }

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
  // a row of nth complex sums and the sum of magnitudes (separate arrays: the loop vectorizes)
  struct Row {
    std::vector<double> v;
    int n;
    explicit Row(int n_) : v(3 * (size_t)n_), n(n_) {}
    void clear() { std::fill(v.begin(), v.end(), 0.0); }
    void add(std::complex<double> x, const Row& y) {  // += x y
      const double xr = x.real(), xi = x.imag(), xm = modulus(x);
      double* __restrict re = v.data();
      double* __restrict im = re + n;
      double* __restrict mag = im + n;
      const double* __restrict yr = y.v.data();
      const double *yi = yr + n, *ym = yi + n;
      for (int t = 0; t < n; ++t) {
        re[t] += xr * yr[t] - xi * yi[t];
        im[t] += xr * yi[t] + xi * yr[t];
        mag[t] += xm * ym[t];
      }
    }
    void set(int t, std::complex<double> z) {
      v[t] = z.real();
      v[n + t] = z.imag();
      v[2 * (size_t)n + t] = modulus(z);
    }
    std::complex<double> at(int t) const { return {v[t], v[n + t]}; }
    double sum_of_magnitudes(int t) const { return v[2 * (size_t)n + t]; }
  };
  std::vector<Row> rows(nu, Row(nth)), moves;
  for (int u = 0; u < nu; ++u)
    for (int t = 0; t < nth; ++t) rows[u].set(t, m.fwd[(size_t)u * nth + t]);
  // what a merge takes from its members' rows sums to zero, so one of them (the group's first) goes without: B F changes
  // by the sum over the others of (B_member - B_first) dF_member
  std::vector<int> moved;
  for (int n = 0; n < nw; ++n) {
    if (n == first[group[n]]) continue;
    moved.push_back(n);
    moves.emplace_back(nth);
    for (int t = 0; t < nth; ++t) moves.back().set(t, F[(size_t)n * nth + t] - m.fwd[(size_t)group[n] * nth + t]);
  }
  // the composed transform's size, and per time the change: (full - half) fwd + B dF
  Row s(nth), skew(nth), d(nth);
  double scale = 0.0, change = 0.0, bound = 0.0;
  for (int t = 0; t < nth; ++t) {
    s.clear();
    skew.clear();
    for (int u = 0; u < nu; ++u) {
      const std::complex<double> h = m.half[(size_t)t * nu + u];
      s.add(h, rows[u]);
      skew.add(m.full[(size_t)t * nu + u] - h, rows[u]);
    }
    for (int k = 0; k < nth; ++k) scale = std::max(scale, modulus(s.at(k)));
    for (int mirror = 0; mirror < 2; ++mirror) {
      const std::complex<double>* b = B + (size_t)(mirror ? nts - 1 - t : t) * nw;
      d.clear();
      for (size_t i = 0; i < moved.size(); ++i) d.add(b[moved[i]] - b[first[group[moved[i]]]], moves[i]);
      const double sign = mirror ? -1.0 : 1.0;  // the mirrored row of full - half is minus this one
      for (int k = 0; k < nth; ++k) {
        change = std::max(change, modulus(sign * skew.at(k) + d.at(k)));
        bound = std::max(bound, skew.sum_of_magnitudes(k) + d.sum_of_magnitudes(k));
      }
    }
  }
  m.change = scale > 0.0 ? change / scale : change;
  m.bound = scale > 0.0 ? bound / scale : bound;
  m.ok = m.change <= MIRROR_CHANGE_TOL && m.bound <= MIRROR_BOUND_TOL;
  return m;
}

}  // namespace gb200
