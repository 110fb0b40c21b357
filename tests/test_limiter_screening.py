"""The screening of a neighbour in the scaling limiters (csrc/fc_limiter.cuh)
against the limiter written out without it, bit for bit: ratios around the
values where a neighbour stops counting, projections around the literal 1.e-6,
fields far from zero and far apart, zeros, infinities and NaN."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "freecappuccino-dev_gb300", "csrc")

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <random>
#include "fc_limiter.cuh"
template <int KIND>
double plain(int m, const double* x, const double* y, const double* z, double pc, double gx, double gy, double gz,
             double lo, double hi) {
  double s = 1.0;
  for (int n = 1; n <= m; ++n) {
    const double d = gx * (x[n] - x[0]) + gy * (y[n] - y[0]) + gz * (z[n] - z[0]);
    const double r = (d < 0.0 ? -d : d) < fclim::kTinyDelta ? 1.0 : (d > 0.0 ? hi - pc : lo - pc) / d;
    s = fclim::dmin(s, fclim::limiter_fn<KIND>(r));
  }
  return s;
}
template <int KIND>
int run(int cases) {
  std::mt19937_64 rng(KIND);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  const double near[] = {0.0, 1e-16, -1e-16, 1e-12, -1e-12, 1e-9, -1e-8, 1e-7, -1e-6, 1e-5, 1e-3, -1e-3, 0.011, 0.05};
  int bad = 0, used = 0;
  for (int t = 0; t < cases; ++t) {
    const int m = 1 + (int)(rng() % 8), what = (int)(rng() % 8);
    double x[9], y[9], z[9];
    const double off = what == 1 ? 1e6 * u(rng) : 0.0, h = std::pow(10.0, 3.0 * u(rng));
    for (int n = 0; n <= m; ++n) { x[n] = off + h * u(rng); y[n] = off + h * u(rng); z[n] = h * u(rng); }
    double gs = std::pow(10.0, (what == 2 ? 60.0 : 4.0) * u(rng));
    if (what == 3) gs = 1e-6 / h;
    double g[3] = {gs * u(rng), gs * u(rng), gs * u(rng)};
    if (what == 4) g[rng() % 3] = rng() % 2 ? 0.0 : (rng() % 2 ? inf : nan);
    if (what == 5) { g[1] = g[2] = 0.0; g[0] = fclim::kTinyDelta * (1.0 + near[rng() % 14]) / (x[1] - x[0]); }
    const double pc = what == 1 ? 1e5 * u(rng) : u(rng);
    const double d1 = std::fabs(g[0] * (x[1] - x[0]) + g[1] * (y[1] - y[0]) + g[2] * (z[1] - z[0]));
    const double at[] = {0.5, 1.0, 1.01, 2.0, 2.02, 5.0, 1e3, 1e17};
    const double room = d1 * at[rng() % 8] * (1.0 + near[rng() % 14]);
    double hi = pc + room, lo = pc - room;
    if (what == 6) { hi = rng() % 2 ? inf : pc; lo = rng() % 2 ? -inf : nan; }
    const int ia[2] = {0, m + 1}, dg[1] = {0};
    int ja[9];
    for (int n = 0; n <= m; ++n) ja[n] = n;
    const double a = plain<KIND>(m, x, y, z, pc, g[0], g[1], g[2], lo, hi);
    const double b = fclim::limit_factor<KIND>(0, ia, ja, dg, x, y, z, &pc, g[0], g[1], g[2], lo, hi);
    bad += std::memcmp(&a, &b, 8) != 0;
    used += a < 1.0;
  }
  std::printf("kind %d bad %d limited %d\n", KIND, bad, used);
  return bad;
}
int main() { return run<1>(400000) + run<2>(400000) + run<3>(400000) ? 1 : 0; }
"""


def test_screened_neighbours_change_nothing(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "screen.cpp", str(tmp_path / "screen")
    src.write_text(SRC)
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert all(int(line.split()[-1]) > 1000 for line in out.stdout.splitlines()), out.stdout
