// Arrays over the host link: the page-locked buffers and the chunked copies through them.
#pragma once

#include <algorithm>
#include <cstring>

#include "device.h"

namespace sf {

// An array of megabytes crosses in chunks through two pooled pinned buffers, so that the link moves
// one chunk at its own rate while `threads` host threads copy the other; a copy to or from pageable
// memory runs on one thread in the driver, page faults of a fresh result array included (the gate
// plate's 57 MB of fields, with the point records put together on the device instead of the host:
// 20.6 -> 3.8 ms a call; the 60^3 block's 42 MB of displacements 23 -> 4 ms). Where no page-locked
// memory is to be had, such a plain copy still serves.
constexpr size_t kCopyChunk = (size_t)4 << 20;
constexpr size_t kSmallCopy = (size_t)64 << 10;       // below this the driver's own staging is as quick

inline void host_copy(void* dst, const void* src, size_t bytes, int threads) {
  const int parts = bytes < ((size_t)1 << 20) ? 1 : threads;
#ifdef _OPENMP
#pragma omp parallel for schedule(static, 1) num_threads(parts) if (parts > 1)
#endif
  for (int p = 0; p < parts; ++p) {
    const size_t b = bytes * (size_t)p / parts / 64 * 64, e = p + 1 == parts ? bytes : bytes * (size_t)(p + 1) / parts / 64 * 64;
    std::memcpy((char*)dst + b, (const char*)src + b, e - b);
  }
}

// Two pinned chunks and their events (`ok`: all four were to be had); the buffers go back to the
// pool once nothing uses them.
struct Staging {
  void* buf[2] = {nullptr, nullptr};
  cudaEvent_t done[2] = {nullptr, nullptr};
  bool ok = true;
  explicit Staging(size_t chunk) {
    for (int i = 0; i < 2; ++i) {
      buf[i] = pinned_acquire(chunk);
      ok = buf[i] && cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming) == cudaSuccess && ok;
    }
    if (!ok) cudaGetLastError();  // the plain copy takes over: no later check may find this error
  }
  ~Staging() {
    for (int i = 0; i < 2; ++i) {
      if (buf[i]) pinned_return(buf[i]);
      if (done[i]) cudaEventDestroy(done[i]);
    }
  }
};

// Device bytes to host memory, complete on return. `from(at, len)` gives the device address of the
// bytes [at, at + len) of a chunk, enqueueing what makes them on d.stream first.
template <class F>
sf_status copy_out(const DeviceSolver& d, void* dst, size_t bytes, size_t chunk, int threads, F&& from) {
  if (bytes < kSmallCopy && bytes <= chunk) {
    if (bytes) copy_d2h(d, dst, from(0, bytes), bytes);
    return cuda_check(cudaStreamSynchronize(d.stream), "copy to the host");
  }
  Staging st(std::min(chunk, bytes));
  if (!st.ok) {
    for (size_t at = 0; at < bytes; at += chunk) {
      const size_t len = std::min(chunk, bytes - at);
      copy_d2h(d, (char*)dst + at, from(at, len), len);
    }
    return cuda_check(cudaStreamSynchronize(d.stream), "copy to the host");
  }
  const size_t count = (bytes + chunk - 1) / chunk;
  sf_status e = SF_OK;
  for (size_t i = 0; i <= count && !e; ++i) {
    if (i < count) {
      const size_t at = i * chunk, len = std::min(chunk, bytes - at);
      copy_d2h(d, st.buf[i & 1], from(at, len), len);
      cudaEventRecord(st.done[i & 1], d.stream);
    }
    if (i > 0) {
      const size_t at = (i - 1) * chunk, len = std::min(chunk, bytes - at);
      e = cuda_check(cudaEventSynchronize(st.done[(i - 1) & 1]), "copy to the host");
      if (!e) host_copy((char*)dst + at, st.buf[(i - 1) & 1], len, threads);
    }
  }
  const sf_status end = cuda_check(cudaStreamSynchronize(d.stream), "copy to the host");
  return e ? e : end;
}

// Host bytes to device memory and to `keep`, ordinary memory of the study's (null where `src` is that
// already); `src` may be reused on return.
inline sf_status copy_in(const DeviceSolver& d, void* dst, const void* src, void* keep, size_t bytes, int threads) {
  if (bytes < kSmallCopy) {
    if (keep) std::memcpy(keep, src, bytes);
    // not from a caller's src: a page-locked one is read when the stream gets there
    if (bytes) copy_h2d(d, dst, keep ? keep : src, bytes);
    return SF_OK;
  }
  Staging st(std::min(kCopyChunk, bytes));
  if (!st.ok) {
    if (keep) std::memcpy(keep, src, bytes);
    copy_h2d(d, dst, src, bytes);
    return cuda_check(cudaStreamSynchronize(d.stream), "copy to the device");
  }
  sf_status e = SF_OK;
  for (size_t i = 0, at = 0; at < bytes && !e; ++i, at += kCopyChunk) {
    const size_t len = std::min(kCopyChunk, bytes - at);
    if (i >= 2) e = cuda_check(cudaEventSynchronize(st.done[i & 1]), "copy to the device");
    host_copy(st.buf[i & 1], (const char*)src + at, len, threads);
    copy_h2d(d, (char*)dst + at, st.buf[i & 1], len);
    cudaEventRecord(st.done[i & 1], d.stream);
    if (keep) host_copy((char*)keep + at, (const char*)src + at, len, threads);
  }
  const sf_status end = cuda_check(cudaStreamSynchronize(d.stream), "copy to the device");
  return e ? e : end;
}

}  // namespace sf
