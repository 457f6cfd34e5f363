"""How a run spreads its launches over streams when device memory is short
(run_streams.hpp, compiled here for the host): fewer streams, down to one with
the largest launch's scratch, before the call fails."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "run_streams.hpp"
using namespace igpu::host;

static int bad = 0;
static void expect(bool ok, const char* what) {
  if (!ok) {
    ++bad;
    std::printf("%s\n", what);
  }
}

// A buffer that only grows, on a device of `room` doubles; a refused growth
// loses the old buffer, as the plan's does.
struct Buffer {
  size_t room, held = 0;
  bool operator()(size_t total, bool) {
    if (total <= held) return true;
    held = 0;
    if (total > room) return false;
    held = total;
    return true;
  }
};

static size_t assign(std::vector<StreamItem>& run, size_t ns, Buffer& b, std::vector<size_t>& region) {
  std::vector<size_t> order(run.size());
  for (size_t k = 0; k < order.size(); ++k) order[k] = k;
  const size_t n = assign_streams(run, order, ns, [&](size_t t, bool s) { return b(t, s); }, region);
  if (n == 0) return 0;
  size_t sum = 0;
  for (size_t r : region) sum += r;
  expect(region.size() == n, "a region for every stream");
  expect(sum <= b.held, "the regions lie in the buffer");
  for (const StreamItem& r : run) {
    expect(r.stream < n && region[r.stream] >= r.doubles, "a launch fits its stream's region");
    expect(!r.full || r.stream == 0, "full launches on stream 0");
  }
  return n;
}

int main() {
  std::vector<StreamItem> run;
  for (size_t k = 0; k < 12; ++k) run.push_back({12.0 - k, k == 0, 1000 - 10 * k, 0});
  std::vector<size_t> region;
  const size_t room[] = {1u << 20, 7000, 3999, 1999, 1000, 999};
  const size_t want[] = {8, 4, 4, 2, 1, 0};
  for (int q = 0; q < 6; ++q) {
    Buffer b{room[q]};
    const size_t n = assign(run, 8, b, region);
    if (n != want[q]) std::printf("room %zu: %zu streams\n", room[q], n);
    expect(n == want[q], "streams for the room");
  }
  Buffer used{3999};
  used.held = 1500;  // what an earlier run left; the growth to eight regions loses it
  expect(assign(run, 8, used, region) == 4, "a lost buffer is had again");
  run[3].doubles = kScratchBudget;
  Buffer big{kScratchBudget + 999};
  expect(assign(run, 8, big, region) == 1, "the budget holds for several streams");
  run[3].doubles = 2 * kScratchBudget;
  Buffer huge{2 * kScratchBudget};
  expect(assign(run, 8, huge, region) == 1, "one stream takes what it needs");
  std::vector<StreamItem> none;
  Buffer empty{0};
  expect(assign(none, 1, empty, region) == 1, "no launches");
  return bad != 0;
}
"""


def test_streams_when_memory_is_short(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "integral_b200", "csrc"), src, "-o", exe],
                   check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
