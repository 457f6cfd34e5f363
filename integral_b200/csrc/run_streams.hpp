// How a run's class launches are spread over streams, each with a scratch
// region of its own (run_tasks); no CUDA here, so that it runs without a device.
#pragma once
#include <algorithm>
#include <cstddef>
#include <numeric>
#include <vector>

namespace igpu {
namespace host {

// Scratch doubles (4 GiB) above which a run uses fewer streams, each of which
// needs a scratch region of its own.  256 MiB (or twice the largest launch's)
// left a 5-atom g molecule two streams and cost it 52 against 35 ms, an f
// gradient 39 against 28 ms; allocating the 4 GiB adds 3 ms to a first run.
constexpr size_t kScratchBudget = (size_t)1 << 29;
// Share of the device's free memory that the regions of more than one stream
// may take: a program with many plans, each of which keeps its scratch, runs on
// fewer streams before the device is full.
constexpr size_t kScratchShare = 8;

// One launch of a run.
struct StreamItem {
  double load;     // estimated time
  bool full;       // fills the device by itself: stream 0
  size_t doubles;  // scratch
  size_t stream;   // its stream (result)
};

// Spreads the launches, in `order`, over at most `ns` streams, each onto the one
// with the least load, and gives the scratch of every stream in `region`.
// Returns the number of streams: `ns`, halved while the regions exceed the
// budget or `have(doubles, several)` cannot provide them (several: they are of
// more than one stream).  0 when not even a single stream's region can be had.
template <class Have>
size_t assign_streams(std::vector<StreamItem>& run, const std::vector<size_t>& order, size_t ns, Have have,
                      std::vector<size_t>& region) {
  for (;; ns = (ns + 1) / 2) {
    std::vector<double> load(ns, 0.0);
    region.assign(ns, 0);
    for (size_t x : order) {
      StreamItem& r = run[x];
      r.stream = r.full ? 0 : (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
      load[r.stream] += r.load;
      region[r.stream] = std::max(region[r.stream], r.doubles);
    }
    const size_t total = std::accumulate(region.begin(), region.end(), (size_t)0);
    if ((ns == 1 || total <= kScratchBudget) && have(total, ns > 1)) return ns;
    if (ns == 1) return 0;
  }
}

}  // namespace host
}  // namespace igpu
