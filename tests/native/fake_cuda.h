// A stand-in for the CUDA runtime's host calls, for tests of host code without a device: "device"
// memory is host memory, and a stream runs late. A copy whose host side is page-locked waits in the
// stream until something synchronizes; a copy of pageable memory is complete on return, as the
// driver's is. Calls are told to fail through the counters below.
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <vector>

#include "sf_internal.h"

namespace fake {

inline std::deque<std::function<void()>> stream;
inline std::map<const char*, size_t> pinned;  // page-locked ranges
inline int pinned_left = 1 << 30;             // page-locked allocations that still succeed
inline cudaError_t last = cudaSuccess;        // what cudaGetLastError would return

inline void drain() {
  while (!stream.empty()) {
    auto f = std::move(stream.front());
    stream.pop_front();
    f();
  }
}
inline bool is_pinned(const void* p) {
  auto it = pinned.upper_bound((const char*)p);
  if (it == pinned.begin()) return false;
  --it;
  return (const char*)p < it->first + it->second;
}
inline cudaError_t failed(cudaError_t e) { return last = e; }

}  // namespace fake

extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (fake::pinned_left-- <= 0) return fake::failed(cudaErrorMemoryAllocation);
  *p = std::malloc(n);
  fake::pinned[(const char*)*p] = n;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  const bool late = fake::is_pinned(kind == cudaMemcpyHostToDevice ? src : dst);
  fake::stream.push_back([=] { std::memcpy(dst, src, n); });
  if (!late) fake::drain();
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  fake::drain();
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = (cudaEvent_t)std::malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) {
  fake::drain();
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = fake::last;
  fake::last = cudaSuccess;
  return e;
}
}

namespace sf {
sf_status fail(sf_status status, const char*) { return status; }
sf_status cuda_check(cudaError_t e, const char*) {
  if (e == cudaSuccess) return SF_OK;
  return e == cudaErrorMemoryAllocation ? SF_DEVICE_MEMORY_BUDGET : SF_CUDA_ERROR;
}
}  // namespace sf

#define CHECK(ok)                                                  \
  do {                                                             \
    if (!(ok)) {                                                   \
      std::printf("%s:%d: %s\n", __FILE__, __LINE__, #ok);         \
      std::exit(1);                                                \
    }                                                              \
  } while (0)
