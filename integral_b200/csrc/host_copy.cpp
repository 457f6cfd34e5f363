// Large results to the caller's (pageable) buffers.
//
// One cudaMemcpy into freshly allocated pages runs at the rate of one host
// thread that takes the page faults (68 MB: 15 ms, thirty times the kernels of
// a 54-function dense tensor).  Several threads instead bring 1 MiB pieces over
// into pinned buffers and move them on, page faults included, while the others'
// transfers run.
#include "host_copy.hpp"

#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>

namespace igpu {
namespace host {

namespace {
constexpr size_t kPiece = (size_t)1 << 20;
constexpr size_t kStaged = (size_t)8 << 20;  // below this one copy is as fast

// The pinned buffers (kRunStreams pieces), made by the first large result and
// shared by the plans of the process: one copy at a time uses them, others fall
// back to a plain copy.  They stay until the process ends: pinning and freeing
// them with the last plan takes 4 to 10 ms, which a program with one plan at a
// time paid for every result (a 54-function dense tensor through a new plan:
// 16 to 21 ms then, 5.4 ms now; the 3-centre tensor of 8 atoms 25 and 14 ms).
std::mutex g_use;
char* g_buf = nullptr;
}  // namespace

int copy_to_host(igpu_plan* P, void* dst, const void* src, size_t bytes, cudaStream_t s) {
  std::unique_lock<std::mutex> use(g_use, std::defer_lock);
  const bool staged = bytes >= kStaged && use.try_lock();
  if (staged && !g_buf && cudaHostAlloc(&g_buf, kRunStreams * kPiece, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    g_buf = nullptr;
  }
  if (!staged || !g_buf) {
    CK(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    return IGPU_OK;
  }
  const size_t pieces = (bytes + kPiece - 1) / kPiece;
  const size_t nw = std::min<size_t>({kRunStreams, pieces, std::max(1u, std::thread::hardware_concurrency())});
  int rc = ensure_side_streams(P, nw - 1);
  if (rc) return rc;
  // the pieces' streams wait for what `s` has queued
  CK(cudaEventRecord(P->side_ev[nw - 1], s));
  for (size_t k = 1; k < nw; ++k) CK(cudaStreamWaitEvent(P->side[k - 1], P->side_ev[nw - 1], 0));
  std::atomic<size_t> next{0};
  std::atomic<int> err{(int)cudaSuccess};
  auto work = [&](size_t w) {
    cudaError_t e = cudaSetDevice(P->device);
    const cudaStream_t st = w == 0 ? s : P->side[w - 1];
    char* buf = g_buf + w * kPiece;
    for (size_t c; e == cudaSuccess && (c = next.fetch_add(1)) < pieces;) {
      const size_t at = c * kPiece, len = std::min(kPiece, bytes - at);
      e = cudaMemcpyAsync(buf, static_cast<const char*>(src) + at, len, cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      if (e == cudaSuccess) std::memcpy(static_cast<char*>(dst) + at, buf, len);
    }
    if (e != cudaSuccess) err = (int)e;
  };
  std::thread workers[kRunStreams];
  for (size_t w = 1; w < nw; ++w) {
    try {
      workers[w] = std::thread(work, w);
    } catch (const std::exception&) {
      break;  // the threads there are take every piece
    }
  }
  work(0);
  for (std::thread& t : workers)
    if (t.joinable()) t.join();
  CK((cudaError_t)err.load());
  return IGPU_OK;
}

}  // namespace host
}  // namespace igpu
