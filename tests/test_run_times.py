"""How a run's device time is divided among launches that overlap
(run_times.hpp, compiled here for the host): records of launches one after
another are their own times, and the records of a run add up to its span."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "run_times.hpp"
using namespace igpu::host;

static int bad = 0;
static void expect(const std::vector<LaunchSpan>& l, const std::vector<double>& want, const char* what) {
  const std::vector<double> got = share_time(l);
  for (size_t k = 0; k < want.size(); ++k)
    if (!(std::fabs(got[k] - want[k]) <= 1e-12)) {
      ++bad;
      std::printf("%s: launch %zu %.17g, not %.17g\n", what, k, got[k], want[k]);
    }
}

int main() {
  expect({}, {}, "no launches");
  expect({{0, 2, 1}, {2, 5, 0.1}, {6, 7, 0.5}}, {2, 3, 1}, "one after another");
  expect({{0, 4, 1}, {0, 4, 1}}, {2, 2}, "two full ones side by side");
  expect({{0, 10, 1}, {0, 12, 0.25}}, {8, 4}, "a small one beside a full one, then alone");
  expect({{0, 9, 0.5}, {3, 6, 0.5}}, {7.5, 1.5}, "one inside another");
  expect({{1, 1, 1}, {0, 2, 1}}, {0, 2}, "one without a time");
  return bad != 0;
}
"""


def test_shares_of_overlapping_launches(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "integral_b200", "csrc"), src, "-o", exe],
                   check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
