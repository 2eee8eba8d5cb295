"""rcp64 (renderx_gb300/csrc/rx_rcp.cuh), the reciprocal of the subpath records, against its
error bound over its whole range and against the division outside it. Compiled for the host:
the same IEEE operations as on the GPU (one single-precision division, four fused
multiply-adds)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include "rx_rcp.cuh"
int main() {
  // |1 - x y| of a result within 2^-53 (1 + 2^-38) of 1 / x; the fused residual is rounded once more
  const double bound = std::ldexp(1.0 + std::ldexp(1.0, -30), -53);
  double worst = 0.0;
  long n = 0, off = 0;
  auto near = [&](double x) {
    const double y = rx::rcp64(x), r = std::fabs(std::fma(-x, y, 1.0));
    if (!(r <= bound)) { printf("x %.17g y %.17g residual %g\n", x, y, r); return false; }
    worst = std::fmax(worst, r);
    n++;
    off += y != 1.0 / x;
    return true;
  };
  std::mt19937_64 rng(3);
  std::uniform_real_distribution<double> m(1.0, 2.0), e(-30.0, 30.0);
  for (int k = 0; k < 4000000; k++)
    if (!near(std::pow(10.0, e(rng))) || !near(m(rng))) return 1;
  for (int k = -99; k <= 99; k++)  // powers of two, their neighbours, and the points where the cast to single rounds
    for (double x : {1.0, 1.0 + 0x1p-24, 1.0 + 0x1p-23, 1.0 + 0x1p-52, 2.0 - 0x1p-52, 2.0 - 0x1p-24, 1.5 - 0x1p-24})
      for (double d : {0.0, 1e300, -1e300})
        if (!near(std::ldexp(d == 0.0 ? x : std::nextafter(x, d), k))) return 2;
  if (!near(std::nextafter(1e-30, 1.0)) || !near(std::nextafter(1e30, 0.0))) return 3;
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  for (double x : {1e-30, 1e30, std::nextafter(1e30, inf), 1e-45, 1e300, 5e-324, 0.0, -0.0, -1.0, -1e-40, -1e40, inf, -inf, nan}) {
    const double a = rx::rcp64(x), b = 1.0 / x;
    if (std::memcmp(&a, &b, 8) && !(std::isnan(a) && std::isnan(b))) { printf("x %g: %g %g\n", x, a, b); return 4; }
  }
  printf("ok %ld values, worst residual %.6f x 2^-53, %ld not the rounded quotient\n", n, worst * 0x1p53, off);
  return 0;
}
"""


@pytest.mark.skipif(not os.path.exists("/usr/local/cuda/include/cuda_runtime.h"), reason="no CUDA headers")
def test_rcp64_stays_within_its_bound(tmp_path):
    src, exe = tmp_path / "rcp.cpp", tmp_path / "rcp"
    src.write_text(SOURCE)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", "/usr/local/cuda/include",
                    "-I", os.path.join(ROOT, "renderx_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok "), r.stdout + r.stderr
