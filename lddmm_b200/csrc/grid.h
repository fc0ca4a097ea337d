// Host tables of the gridded Gaussian sums (grid.cuh): the interpolation window's
// polynomials and the grid kernel.  Plain C++ (no device code).
#pragma once

#include <cmath>
#include <vector>

namespace lddmm {

constexpr int kWin = 10;        // nodes per axis under a point's window
constexpr int kWinDeg = 12;     // degree of the window's polynomial per node
constexpr int kWinCoef = kWinDeg + 1;
constexpr double kGridH = 0.25; // node spacing in scaled coordinates
constexpr int kGridTaps = 26;   // the grid kernel reaches this many nodes

struct GridTables {
  // win[k][i]: coefficient of z^i, z = 2 f - 1, of the window at node k for a point whose
  // cell fraction is f (distance f + kWin / 2 - 1 - k nodes); dwin: its derivative per
  // scaled unit
  double win[kWin][kWinCoef], dwin[kWin][kWinCoef];
  double ker[kGridTaps + 1];
};

// Window: Kaiser-Bessel psi(d) = I0(b sqrt(1 - (2 d / w)^2)) / I0(b), d in nodes, with
// shape b = 2.65 w.  Its Fourier transform is w h sinh(s) / (s I0(b)), s^2 = b^2 -
// (w h om / 2)^2.  The grid kernel T is the inverse transform of
//   h K^(om) psi^(om)^2 / (sum_k psi^(om + 2 pi k / h)^2)^2,
// the least-squares choice for K(x - y) ~ sum_mn psi(x - mh) T(m - n) psi(y - nh) with
// K(x) = 2^-x^2 (for the deconvolution 1 / psi^2 when the aliases vanish).
inline const GridTables &grid_tables() {
  static const GridTables t = [] {
    GridTables g{};
    const double pi = 3.14159265358979323846, ln2 = 0.69314718055994530942;
    const double b = 2.65 * kWin, i0b = std::cyl_bessel_i(0.0, b);
    auto psi = [&](double d) {
      const double u = 1.0 - (2.0 * d / kWin) * (2.0 * d / kWin);
      return u > 0.0 ? std::cyl_bessel_i(0.0, b * std::sqrt(u)) / i0b : (u == 0.0 ? 1.0 / i0b : 0.0);
    };
    // per node: Chebyshev interpolation on 32 points, truncated, as powers of z
    constexpr int nc = 32;
    for (int k = 0; k < kWin; ++k) {
      double val[nc], ch[kWinCoef];
      for (int j = 0; j < nc; ++j)
        val[j] = psi(0.5 * (std::cos(pi * (j + 0.5) / nc) + 1.0) + kWin / 2 - 1 - k);
      for (int i = 0; i < kWinCoef; ++i) {
        double s = 0.0;
        for (int j = 0; j < nc; ++j) s += val[j] * std::cos(pi * i * (j + 0.5) / nc);
        ch[i] = s * (i ? 2.0 : 1.0) / nc;
      }
      // sum ch_i T_i(z) in powers of z by the recurrence T_{i+1} = 2 z T_i - T_{i-1}
      std::vector<double> a(kWinCoef, 0.0), p(kWinCoef, 0.0), c(kWinCoef, 0.0);
      a[0] = 1.0;  // T_0
      p[1] = 1.0;  // T_1
      for (int i = 0; i < kWinCoef; ++i) {
        for (int q = 0; q < kWinCoef; ++q) c[q] += ch[i] * a[q];
        std::vector<double> nx(kWinCoef, 0.0);  // T_{i+2} from T_{i+1} = p and T_i = a
        for (int q = 0; q + 1 < kWinCoef; ++q) nx[q + 1] = 2.0 * p[q];
        for (int q = 0; q < kWinCoef; ++q) nx[q] -= a[q];
        a = p;
        p = nx;
      }
      for (int q = 0; q < kWinCoef; ++q) g.win[k][q] = c[q];
      for (int q = 0; q + 1 < kWinCoef; ++q) g.dwin[k][q] = (q + 1) * c[q + 1] * 2.0 / kGridH;
    }
    auto hat = [&](double om) {
      const double x = 0.5 * kWin * kGridH * om, s2 = b * b - x * x;
      const double s = std::sqrt(std::fabs(s2));
      const double r = s < 1e-8 ? 1.0 : (s2 > 0.0 ? std::sinh(s) / s : std::sin(s) / s);
      return kWin * kGridH * r / i0b;
    };
    constexpr int n = 1024;
    const double dom = 2.0 * pi / (kGridH * n);
    for (int k = 0; k < n; ++k) {
      const double om = (k + 0.5 - n / 2) * dom;
      double s = 0.0;
      for (int q = -4; q <= 4; ++q) {
        const double f = hat(om + 2.0 * pi * q / kGridH);
        s += f * f;
      }
      const double f0 = hat(om);
      const double tau = kGridH * std::sqrt(pi / ln2) * std::exp(-om * om / (4.0 * ln2)) * f0 *
                         f0 / (s * s);
      for (int m = 0; m <= kGridTaps; ++m)
        g.ker[m] += kGridH / (2.0 * pi) * tau * std::cos(om * m * kGridH) * dom;
    }
    return g;
  }();
  return t;
}

}  // namespace lddmm
