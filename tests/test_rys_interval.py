"""The look-up of the Rys tables stays inside them for every T (igpu_internal.hpp,
the functions that the kernels call, compiled here for the host): a NaN and T
from the crossover on take the closed form, everything else an interval of the
table, with the position inside it for T >= 0."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <limits>
#include "igpu_internal.hpp"
using namespace igpu;

template <typename R>
int check() {
  int bad = 0;
  const R inf = std::numeric_limits<R>::infinity(), nan = std::numeric_limits<R>::quiet_NaN();
  for (int n = 1; n <= MAX_ROOTS; ++n) {
    const R hi = R(rys_t_hi(n)), below = std::nextafter(hi, R(0));
    for (R T : {nan, -nan, inf, hi, std::nextafter(hi, inf)}) bad += rys_tabulated(n, T);
    for (R T : {R(-1e6), R(-100), R(-1), R(-1e-30), R(-0.0), R(0), std::numeric_limits<R>::denorm_min(), R(0.25),
                std::nextafter(R(1), R(0)), R(1), R(17.3), below}) {
      R xi = nan;
      const int s = rys_tabulated(n, T) ? rys_interval(n, T, xi) : -1;
      const bool in = s >= 0 && s < rys_nsub<R>(n) && (T < 0 || (xi >= R(-1) && xi <= R(1)));
      if (!in) {
        ++bad;
        std::printf("n %d T %g interval %d xi %g\n", n, (double)T, s, (double)xi);
      }
    }
  }
  return bad;
}
int main() { return check<double>() + check<float>() ? 1 : 0; }
"""


def test_every_T_has_an_interval_or_the_closed_form(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "integral_b200", "csrc"), src, "-o", exe],
                   check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
