"""Host searches that start from monotone or uniform structure (band-limit
mask, detector runs, pixel snap, slicing order) against the plain loops they
replace, over random cells, cut-offs, positions and their boundary values: the
same indices in every case.  The loops are restated here in C++ and compiled
with csrc/setup.cpp."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ms-stem-fem_b200" / "csrc"

HARNESS = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <random>
#include "setup.hpp"
using namespace msf;

static int64_t plain_snap(const std::vector<double>& x, double q, double half, int64_t last) {
  for (size_t i = 0; i < x.size(); ++i)
    if (x[i] - q >= half) return (int64_t)i - 1;
  return last;
}

int main() {
  std::mt19937_64 rng(3);
  std::uniform_real_distribution<double> u(0, 1);
  long bad = 0;
  for (int t = 0; t < 60; ++t) {
    const int nx = 64 << (rng() % 4), ny = 64 << (rng() % 4);
    const double x = nx * 0.1 * (0.3 + 2 * u(rng)), y = ny * 0.1 * (0.3 + 2 * u(rng));
    const Grid g = make_grid(nx, ny, 200000, x, y, 10, 0.1 * (t % 3), 0, 0, x, y, 10);
    for (double c : {g.bw_t, g.bw_pap, 0.0, 3 * g.bw_pap, g.kx[3], g.kx[nx / 2 - 1]}) {
      std::vector<int32_t> lo, hi;
      bandlimit_mask(g, c, &lo, &hi);
      for (int j = 0; j < ny; ++j)
        for (int i = 0; i < nx; ++i)
          bad += (std::pow(g.kx[i], 2) + std::pow(g.ky[j], 2) < std::pow(c, 2)) !=
                 (i < lo[j] || i >= hi[j]);
    }
    const double k = g.bw_pap * g.bw_pap;
    for (int q = 0; q < 4; ++q) {
      const double k1 = q == 3 ? g.ky[1] * g.ky[1] : k * (2 * u(rng) - 0.2);
      const double k2 = q == 3 ? g.kx[2] * g.kx[2] + g.ky[2] * g.ky[2] : k * 3 * u(rng);
      const PixelRuns r = detector_runs(g, k1, k2);
      std::vector<int32_t> got, want;
      for (size_t n = 0; n < r.base.size(); ++n)
        for (int32_t p = r.offset[n]; p < r.offset[n + 1]; ++p)
          got.push_back(r.base[n] + p - r.offset[n]);
      for (int i = 0; i < nx; ++i)
        for (int j = 0; j < ny; ++j) {
          const double ksq = g.kx[i] * g.kx[i] + g.ky[j] * g.ky[j];
          if (ksq > k1 && ksq <= k2) want.push_back(j + i * ny);
        }
      bad += got != want;
    }
    const double half = 0.5 * (g.xx[1] - g.xx[0]);
    std::vector<double> q{INFINITY, -INFINITY, NAN, 1e300, -1e300};
    for (double v : g.xx)
      for (double s : {-half, 0.0, half}) {
        q.push_back(v + s);
        q.push_back(std::nextafter(v + s, 1e9));
        q.push_back(std::nextafter(v + s, -1e9));
      }
    for (int n = 0; n < 200; ++n) q.push_back((u(rng) * 1.4 - 0.2) * x);
    for (double v : q) bad += snap(g.xx, v, half, 5) != plain_snap(g.xx, v, half, 5);
    const int64_t n = 1 + (int64_t)(rng() % 3000);
    std::vector<double> p(3 * n);
    for (double& v : p) v = t % 4 == 0 ? std::floor(u(rng) * 20) : u(rng) * 50;
    if (t % 5 == 1)
      for (int64_t a = 0; a < n; ++a) p[3 * a + 2] = 3.0;
    std::vector<int64_t> order(n);
    for (int64_t a = 0; a < n; ++a) order[a] = a;
    std::stable_sort(order.begin(), order.end(),
                     [&](int64_t a, int64_t b) { return p[3 * a + 2] < p[3 * b + 2]; });
    bad += slice_atoms(n, p.data(), 0, 50, 2.0).order != order;
  }
  std::printf("%ld\n", bad);
  return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_host_searches_equal_plain_loops(tmp_path):
    src = tmp_path / "harness.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "harness"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC),
                           str(src), str(CSRC / "setup.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
