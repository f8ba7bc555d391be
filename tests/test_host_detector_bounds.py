"""The detector annulus for bounds that are not ordinary numbers, or in no
order, against the plain test k1 < k^2 <= k2 of every pixel (compiled with
csrc/setup.cpp)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ms-stem-fem_b200" / "csrc"

HARNESS = r"""
#include <cmath>
#include <cstdio>
#include "setup.hpp"
using namespace msf;

int main() {
  long bad = 0;
  for (int nx : {64, 128})
    for (int ny : {64, 256}) {
      const Grid g = make_grid(nx, ny, 200000, nx * 0.1, ny * 0.13, 10, 0, 0, 0, 1, 1, 10);
      const double in = g.ky[3] * g.ky[3], out = g.ky[9] * g.ky[9];
      const double values[] = {NAN, INFINITY, -INFINITY, 0.0, -1.0, in, out, 1e300};
      for (double k1 : values)
        for (double k2 : values) {
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
    }
  std::printf("%ld\n", bad);
  return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_annulus_of_any_bounds(tmp_path):
    src = tmp_path / "harness.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "harness"
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(CSRC),
                           str(src), str(CSRC / "setup.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
