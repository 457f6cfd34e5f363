// The device time of each launch of a run whose launches overlap; no CUDA here,
// so that it runs without a device.
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

namespace igpu {
namespace host {

// One launch: from its start event to its end event, which includes waiting for
// others, and the share of the device's resident blocks that its grid takes.
struct LaunchSpan {
  double begin, end, fill;
};

// Divides a run's device time among its launches: every moment goes to those
// between their events then, in proportion to the device that they take.  A
// launch alone gets its own time, a full one next to a few blocks of another
// nearly so, and together they get the run's span (less moments of none).
inline std::vector<double> share_time(const std::vector<LaunchSpan>& l) {
  std::vector<double> at, out(l.size(), 0.0);
  for (const LaunchSpan& x : l)
    if (x.end > x.begin) {
      at.push_back(x.begin);
      at.push_back(x.end);
    }
  std::sort(at.begin(), at.end());
  for (size_t k = 1; k < at.size(); ++k) {
    const double dt = at[k] - at[k - 1];
    double sum = 0.0;
    for (const LaunchSpan& x : l)
      if (x.begin <= at[k - 1] && at[k] <= x.end) sum += x.fill;
    for (size_t q = 0; q < l.size() && sum > 0.0; ++q)
      if (l[q].begin <= at[k - 1] && at[k] <= l[q].end) out[q] += dt * l[q].fill / sum;
  }
  return out;
}

}  // namespace host
}  // namespace igpu
