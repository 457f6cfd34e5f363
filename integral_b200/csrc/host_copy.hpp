// Device results to the caller's host buffers (host_copy.cpp).
#pragma once
#include "plan_internal.hpp"

namespace igpu {
namespace host {

// bytes from the device to `dst` once the work queued on `s` is done; returns
// when they are there.
int copy_to_host(igpu_plan* P, void* dst, const void* src, size_t bytes, cudaStream_t s);

}  // namespace host
}  // namespace igpu
