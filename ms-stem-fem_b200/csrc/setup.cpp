// Bit-exact host set-up (see setup.hpp).  Compile with -ffp-contract=off.
#include "setup.hpp"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace msf {

namespace {
const double kKirkland[103][12] = {
#include "kirkland_table.inc"
};
struct MassRule { double exact, lo, hi; int hi_inclusive; unsigned z; };
const MassRule kMassRules[] = {
#include "mass_table.inc"
};
}  // namespace

void wavelength(double VV, double* lambda, double* gamma) {
  const double m_e0 = 9.109e-31, cc = 299792458, ee = 1.60217662e-19;
  const double hh = 6.62607004e-34;
  *lambda = hh * cc * std::pow(10, 10) / std::sqrt(ee * VV * (2.0 * m_e0 * cc * cc + ee * VV));
  *gamma = (hh * std::pow(10, 10) / *lambda) * (hh * std::pow(10, 10) / *lambda) *
           (m_e0 * cc * cc + ee * VV) / ((2 * m_e0 * cc * cc + ee * VV) * ee * VV * m_e0);
}

Grid make_grid(int nx, int ny, double voltage, double xpd, double ypd, double zpd,
               double xmin, double ymin, double zmin, double xperiod, double yperiod,
               double zperiod) {
  Grid g;
  g.nx = nx; g.ny = ny; g.voltage = voltage;
  g.xpd = xpd; g.ypd = ypd; g.zpd = zpd;
  g.xperiod = xperiod; g.yperiod = yperiod; g.zperiod = zperiod;
  g.xmin = xmin; g.ymin = ymin; g.zmin = zmin;
  const long Nx = nx, Ny = ny;
  g.xx.resize(nx); g.yy.resize(ny); g.kx.resize(nx); g.ky.resize(ny);
  // tem.cpp:756-788, func.cpp:92-106 and 147-167
  const double dx = xpd / Nx, dy = ypd / Ny, dkx = 1.0 / xpd, dky = 1.0 / ypd;
  const double kxp = Nx / xpd, kyp = Ny / ypd;
  for (int i = 0; i < Nx; ++i) g.xx[i] = xmin + (i * dx);
  for (int i = 0; i < Ny; ++i) g.yy[i] = ymin + (i * dy);
  for (int i = 0; i < Nx / 2; ++i) g.kx[i] = i * dkx;
  for (int i = Nx / 2; i < Nx; ++i) g.kx[i] = i * dkx - kxp;
  for (int i = 0; i < Ny / 2; ++i) g.ky[i] = i * dky;
  for (int i = Ny / 2; i < Ny; ++i) g.ky[i] = i * dky - kyp;
  // tem.cpp:683-695
  if (Nx / (2 * xpd) < Ny / (2 * ypd)) g.bw_pap = Nx / (2 * xpd);
  else g.bw_pap = Ny / (2 * ypd);
  g.bw_t = (2.0 / 3.0) * g.bw_pap;
  wavelength(voltage, &g.lambda, &g.gamma);
  g.nxny = (double)(Nx * Ny);
  g.s = (Nx == Ny) ? (double)Nx : std::sqrt(g.nxny);
  return g;
}

Slicing slice_atoms(int64_t n, const double* q, double zmin, double zperiod,
                    double min_thickness) {
  Slicing sl;
  if (n == 0) {  // slice.cpp:632-639
    sl.start = {0, 0};
    sl.lower = {zmin};
    sl.thickness = {zperiod};
    return sl;
  }
  // scatterer_sorting_lt_z (scatterer.hpp:192); ties share a slice and a
  // mean, so their order is immaterial -- keep index order.  Sorting
  // contiguous (z, index) pairs lexicographically gives exactly that order
  // (a stable sort by z) without chasing q through an indirect comparator.
  // First into buckets of rising z (a few atoms each), then each bucket: the
  // same order in a third of the time of one sort over all.
  double z0 = q[2], z1 = q[2];
  for (int64_t k = 1; k < n; ++k) {
    z0 = std::min(z0, q[3 * k + 2]);
    z1 = std::max(z1, q[3 * k + 2]);
  }
  const int64_t buckets = std::max<int64_t>(1, n / 8);
  const bool spread = z1 > z0 && std::isfinite(z1 - z0);
  const double per = spread ? (double)buckets / (z1 - z0) : 0.0;
  auto bucket = [&](double z) {  // monotone in z
    return spread ? std::clamp<int64_t>((int64_t)((z - z0) * per), 0, buckets - 1) : 0;
  };
  std::vector<int64_t> begin((size_t)buckets + 1, 0);
  for (int64_t k = 0; k < n; ++k) ++begin[(size_t)bucket(q[3 * k + 2]) + 1];
  for (int64_t b = 0; b < buckets; ++b) begin[(size_t)b + 1] += begin[(size_t)b];
  std::vector<std::pair<double, int64_t>> keys((size_t)n);
  std::vector<int64_t> at(begin.begin(), begin.end() - 1);
  for (int64_t k = 0; k < n; ++k)
    keys[(size_t)at[(size_t)bucket(q[3 * k + 2])]++] = {q[3 * k + 2], k};
  for (int64_t b = 0; b < buckets; ++b)
    std::sort(keys.begin() + begin[(size_t)b], keys.begin() + begin[(size_t)b + 1]);
  sl.order.resize(n);
  for (int64_t k = 0; k < n; ++k) sl.order[(size_t)k] = keys[(size_t)k].second;
  sl.start.push_back(0);
  sl.lower.push_back(0.0);
  double first = q[3 * sl.order[0] + 2];
  for (int64_t k = 0; k < n; ++k) {
    const double z = q[3 * sl.order[k] + 2];
    if (z - first <= min_thickness) {
      sl.lower.back() += z;
    } else {
      sl.start.push_back(k);
      sl.lower.push_back(z);
      first = z;
    }
  }
  sl.start.push_back(n);
  const int64_t ns = (int64_t)sl.lower.size();
  for (int64_t s = 0; s < ns; ++s)
    sl.lower[s] = sl.lower[s] / (double)(size_t)(sl.start[s + 1] - sl.start[s]);
  sl.thickness.resize(ns);
  for (int64_t s = 0; s < ns; ++s) {
    if (s + 1 == ns)
      sl.thickness[s] = q[3 * sl.order[sl.start[s + 1] - 1] + 2] + min_thickness - sl.lower[s];
    else
      sl.thickness[s] = sl.lower[s + 1] - sl.lower[s];
  }
  return sl;
}

int64_t snap(const std::vector<double>& grid, double q, double half, int64_t fallback) {
  // The reference scans for the first i with grid[i] - q >= half.  grid is
  // increasing and rounded subtraction is monotone, so that predicate is
  // false then true along i: starting next to where uniform spacing puts the
  // change and stepping to it finds the same first index (a bisection over
  // the same predicate took 150 ns an atom axis, this takes 15).
  const int64_t n = (int64_t)grid.size();
  auto past = [&](int64_t i) { return grid[(size_t)i] - q >= half; };
  int64_t i = 0;
  if (n > 1) {
    const double guess = (q + half - grid[0]) / (grid[1] - grid[0]);
    i = guess > 0 ? (guess < (double)n ? (int64_t)guess : n) : 0;
  }
  while (i > 0 && past(i - 1)) --i;
  while (i < n && !past(i)) ++i;
  return i < n ? i - 1 : fallback;
}

bool probe_shifts(const Grid& g, const std::vector<double>& x_p,
                  const std::vector<double>& y_p, std::vector<int32_t>* shifts) {
  const double hx = 0.5 * (g.xx[1] - g.xx[0]);
  const double hy = 0.5 * (g.yy[1] - g.yy[0]);
  shifts->assign(2 * x_p.size() * y_p.size(), 0);
  int64_t sx = 0, sy = 0;  // adfstem.cpp:1525-1528, never reset per probe
  size_t k = 0;
  for (double xp : x_p) {
    for (double yp : y_p) {
      sx = snap(g.xx, xp, hx, sx);
      sy = snap(g.yy, yp, hy, sy);
      if (sx < 0 || sy < 0) return false;
      (*shifts)[2 * k] = (int32_t)sx;
      (*shifts)[2 * k + 1] = (int32_t)sy;
      ++k;
    }
  }
  return true;
}

void bandlimit_mask(const Grid& g, double cutoff, std::vector<int32_t>* lo,
                    std::vector<int32_t>* hi) {
  // kx*kx rises with i up to nx/2 and falls from there, so a column keeps a
  // run from 0 and a run up to nx; their ends are found by bisection (a
  // 1024^2 mask took 5 ms pixel by pixel).
  const double csq = std::pow(cutoff, 2);
  lo->assign(g.ny, 0);
  hi->assign(g.ny, g.nx);
  auto first = [](int a, int b, auto&& pred) {  // pred is false, then true
    while (a < b) {
      const int mid = a + (b - a) / 2;
      if (pred(mid)) b = mid;
      else a = mid + 1;
    }
    return a;
  };
  const int half = g.nx / 2;
  for (int j = 0; j < g.ny; ++j) {
    const double y2 = std::pow(g.ky[j], 2);
    auto keep = [&](int i) { return (std::pow(g.kx[i], 2) + y2) < csq; };
    const int a = first(0, half, [&](int i) { return !keep(i); });
    if (a == half && keep(half)) {
      (*lo)[j] = (*hi)[j] = g.nx;  // the whole column
      continue;
    }
    (*lo)[j] = a;
    (*hi)[j] = first(half, g.nx, keep);
  }
}

void propagator(const Grid& g, double thickness, std::vector<double>* px,
                std::vector<double>* py) {
  px->assign(2 * g.nx, 0.0);
  py->assign(2 * g.ny, 0.0);
  for (int i = 0; i < g.nx; ++i)
    if (g.kx[i] < g.bw_t && g.kx[i] > -1.0 * g.bw_t) {
      const double a = kPi * g.lambda * thickness * std::pow(g.kx[i], 2);
      (*px)[2 * i] = std::cos(a);
      (*px)[2 * i + 1] = -std::sin(a);
    }
  for (int j = 0; j < g.ny; ++j)
    if (g.ky[j] < g.bw_t && g.ky[j] > -1.0 * g.bw_t) {
      const double a = kPi * g.lambda * thickness * std::pow(g.ky[j], 2);
      (*py)[2 * j] = std::cos(a);
      (*py)[2 * j + 1] = -std::sin(a);
    }
}

Rings make_rings(const Grid& g, double dr) {
  Rings r;
  r.delta_k = dr * std::sqrt((g.kx[1] - g.kx[0]) * (g.kx[1] - g.kx[0]) +
                             (g.ky[1] - g.ky[0]) * (g.ky[1] - g.ky[0]));
  const unsigned nk = (unsigned)(g.bw_t / r.delta_k);
  r.n_k = (int32_t)nk;
  for (unsigned ii = 0; ii < nk + 1; ++ii) r.bounds.push_back(ii * r.delta_k);
  const int64_t np = (int64_t)g.nx * g.ny;
  r.bin.assign(np, -1);
  r.counts.assign(nk, 0);
  std::vector<double> ub2(nk);
  for (unsigned ii = 0; ii < nk; ++ii) ub2[ii] = r.bounds[ii + 1] * r.bounds[ii + 1];
  std::vector<std::pair<double, int32_t>> sorted;
  sorted.reserve(np);
  for (int i = 0; i < g.nx; ++i)
    for (int j = 0; j < g.ny; ++j) {
      const double ksq = g.kx[i] * g.kx[i] + g.ky[j] * g.ky[j];
      // smallest ii with ksq <= ub2[ii] (ub2 ascending)
      const auto it = std::lower_bound(ub2.begin(), ub2.end(), ksq);
      const int32_t b = (it == ub2.end()) ? -1 : (int32_t)(it - ub2.begin());
      r.bin[j + (int64_t)i * g.ny] = b;
      if (b >= 0) {
        r.counts[b] += 1;
        sorted.emplace_back(ksq, (int32_t)(j + (int64_t)i * g.ny));
      }
    }
  std::stable_sort(sorted.begin(), sorted.end(),
                   [](const std::pair<double, int32_t>& a, const std::pair<double, int32_t>& b) {
                     return a.first < b.first;
                   });
  r.start.assign(nk + 1, 0);
  for (unsigned ii = 0; ii < nk; ++ii) r.start[ii + 1] = r.start[ii] + r.counts[ii];
  r.pix.resize(sorted.size());
  for (size_t k = 0; k < sorted.size(); ++k) r.pix[k] = sorted[k].second;
  r.inside.assign(nk, 0);
  return r;
}

Cells make_cells(const Grid& g, const Rings& r) {
  Cells c;
  unsigned count = 0;
  for (double b : r.bounds)
    if (b >= 0.2 && b <= 1.0) ++count;
  c.n_phi = count > 0 ? (int32_t)(count - 1) : 0;
  const size_t n_cells = (size_t)r.n_k * c.n_phi;
  c.start.assign(n_cells + 1, 0);
  if (c.n_phi == 0) {
    c.phi_bounds.assign(1, 0.0);
    return c;
  }
  const double delta_phi = 2 * kPi / c.n_phi;
  for (int32_t ii = 0; ii < c.n_phi + 1; ++ii) c.phi_bounds.push_back(ii * delta_phi);
  // cell of every ring pixel, in ring order
  std::vector<int32_t> cell_of(r.pix.size(), -1);
  std::vector<int32_t> counts(n_cells, 0);
  for (int32_t ii = 0; ii < r.n_k; ++ii)
    for (int32_t q = r.start[ii]; q < r.start[ii + 1]; ++q) {
      const int32_t p = r.pix[q];
      const int i = p / g.ny, j = p % g.ny;
      const double phi = kPi + std::atan2(g.ky[j], g.kx[i]);
      double lower = c.phi_bounds[0];
      for (int32_t jj = 0; jj < c.n_phi; ++jj) {
        if (phi > lower && phi <= c.phi_bounds[jj + 1]) {
          cell_of[q] = ii * c.n_phi + jj;
          ++counts[(size_t)ii * c.n_phi + jj];
          break;
        }
        lower = c.phi_bounds[jj];  // lags one boundary behind, as there
      }
    }
  for (size_t k = 0; k < n_cells; ++k) c.start[k + 1] = c.start[k] + counts[k];
  c.pix.assign(c.start[n_cells], 0);
  std::vector<int32_t> fill(c.start.begin(), c.start.end() - 1);
  for (size_t q = 0; q < r.pix.size(); ++q)
    if (cell_of[q] >= 0) c.pix[fill[cell_of[q]]++] = r.pix[q];
  return c;
}

PixelRuns detector_runs(const Grid& g, double k1, double k2) {
  // Along a row ky*ky rises with j up to ny/2 and falls from there (rounded
  // products and sums are monotone), so each half of the row holds one run
  // and its ends are found by bisection on the annulus test itself.
  PixelRuns r;
  r.offset.push_back(0);
  auto first = [](int lo, int hi, auto&& pred) {  // pred is false, then true
    while (lo < hi) {
      const int mid = lo + (hi - lo) / 2;
      if (pred(mid)) hi = mid;
      else lo = mid + 1;
    }
    return lo;
  };
  const int half = g.ny / 2;
  for (int i = 0; i < g.nx; ++i) {
    auto ksq = [&](int j) { return g.kx[i] * g.kx[i] + g.ky[j] * g.ky[j]; };
    const int a0 = first(0, half, [&](int j) { return ksq(j) > k1; });
    const int a1 = first(a0, half, [&](int j) { return !(ksq(j) <= k2); });
    const int b0 = first(half, g.ny, [&](int j) { return ksq(j) <= k2; });
    const int b1 = first(b0, g.ny, [&](int j) { return !(ksq(j) > k1); });
    for (const auto& e : {std::pair<int, int>{a0, a1}, std::pair<int, int>{b0, b1}})
      if (e.second > e.first) {
        r.base.push_back((int32_t)(e.first + (int64_t)i * g.ny));
        r.offset.push_back(r.offset.back() + (e.second - e.first));
      }
  }
  return r;
}

std::vector<double> raster_points(double period, double origin, double spacing) {
  const size_t n = (size_t)std::floor(period / spacing);
  std::vector<double> out;
  const double d = period / (int)n;
  for (int i = 0; i < (int)n; ++i) out.push_back(origin + (i * d));
  return out;
}

double scherzer(int which, double lambda, double a) {
  switch (which) {
    case 0: return 0.87 * std::sqrt(a * lambda);
    case 1: return 1.34 * std::pow(lambda / a, 0.25);
    case 2: return -0.983 * std::pow(std::pow(lambda, 2) * a, 1.0 / 3.0);
    case 3: return 1.513 * std::pow(lambda / a, 1.0 / 6.0);
    case 4: return -2.289 * std::pow(lambda * std::pow(a, 2), 1.0 / 3.0);
  }
  return 0.0;
}

unsigned guess_z(double mass) {
  for (const MassRule& r : kMassRules) {
    if (r.exact >= 0.0 && mass == r.exact) return r.z;
    const bool below_hi = r.hi_inclusive ? (mass <= r.hi) : (mass < r.hi);
    if (mass >= r.lo && below_hi) return r.z;
  }
  return 0;
}

const double* kirkland_params(unsigned z) {
  if (z < 1 || z > 103) return nullptr;
  return kKirkland[z - 1];
}

}  // namespace msf

namespace msf {

std::vector<double> mtf_2d(const Grid& g, const double* mtf, const double* domain_sqr, int n,
                           double resolution) {
  std::vector<double> out(2 * (size_t)g.nx * g.ny, 0.0);
  const double nx = (double)g.nx, ny = (double)g.ny;
  for (int i = 0; i < g.nx; ++i)
    for (int j = 0; j < g.ny; ++j) {
      const double xxx = std::pow(g.xpd, 2) * g.kx[i] / nx;
      const double yyy = std::pow(g.ypd, 2) * g.ky[j] / ny;
      const double rsqr = std::pow(xxx, 2) + std::pow(yyy, 2);
      double v = 0.0;
      for (int k = 0; k + 1 < n; ++k) {
        if (rsqr >= domain_sqr[k] && rsqr < domain_sqr[k + 1]) {
          const double d1 = std::sqrt(domain_sqr[k]), d2 = std::sqrt(domain_sqr[k + 1]);
          v = mtf[k] + (mtf[k + 1] - mtf[k]) * (std::sqrt(rsqr) - d1) / (d2 - d1);
          double arg = xxx / resolution;
          const double sx = arg != 0 ? std::sin(arg) / arg : 1;
          arg = yyy / resolution;
          const double sy = arg != 0 ? std::sin(arg) / arg : 1;
          v = v * sx * sy;
        }
      }
      out[2 * ((size_t)i * g.ny + j)] = v;
    }
  return out;
}

}  // namespace msf
