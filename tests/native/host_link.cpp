// The copies of host_link.h on a stand-in runtime: `host_link <case> <bytes>`.
#include "fake_cuda.h"

#include "host_link.h"

using namespace sf;

namespace {

std::vector<char> pattern(size_t n) {
  std::vector<char> v(n);
  for (size_t i = 0; i < n; ++i) v[i] = (char)(i * 2654435761u >> 13);
  return v;
}

// Both directions with `pinned` page-locked allocations to be had; chunks are made in two buffers
// in turn, as the result records are.
void round_trip(size_t n, int pinned) {
  fake::pinned_left = pinned;
  DeviceSolver d;
  std::vector<char> src = pattern(n), device(n), keep(n), out(n), half[2];
  CHECK(copy_in(d, device.data(), src.data(), keep.data(), n, 3) == SF_OK);
  fake::drain();
  CHECK(device == src && keep == src);
  const size_t chunk = kCopyChunk / 88 * 88;
  for (auto& h : half) h.resize(std::min(chunk, n) + 1);
  int turn = 0;
  CHECK(copy_out(d, out.data(), n, chunk, 3, [&](size_t at, size_t len) {
          char* to = half[turn ^= 1].data();
          fake::stream.push_back([=, &src] { std::memcpy(to, src.data() + at, len); });
          return to;
        }) == SF_OK);
  CHECK(out == src);
  CHECK(cudaGetLastError() == cudaSuccess);  // a refused allocation is nobody else's error
}

// A small array put together in less than its size at a time.
void small_chunks(size_t n) {
  DeviceSolver d;
  std::vector<char> src = pattern(n), half[2], out(n);
  for (auto& h : half) h.resize(176);
  int turn = 0;
  CHECK(copy_out(d, out.data(), n, 176, 3, [&](size_t at, size_t len) {
          CHECK(len <= 176);
          char* to = half[turn ^= 1].data();
          fake::stream.push_back([=, &src] { std::memcpy(to, src.data() + at, len); });
          return to;
        }) == SF_OK);
  CHECK(out == src);
}

// The caller's array may be reused once copy_in has returned, page-locked or not.
void reuse(size_t n) {
  DeviceSolver d;
  void* src = nullptr;
  CHECK(cudaMallocHost(&src, n) == cudaSuccess);
  const std::vector<char> first = pattern(n);
  std::memcpy(src, first.data(), n);
  std::vector<char> device(n), keep(n);
  CHECK(copy_in(d, device.data(), src, keep.data(), n, 3) == SF_OK);
  std::memset(src, 0xff, n);
  fake::drain();
  CHECK(device == first && keep == first);
}

}  // namespace

int main(int argc, char** argv) {
  const std::string what = argv[1];
  const size_t n = std::strtoull(argv[2], nullptr, 10);
  if (what == "pinned") round_trip(n, 1 << 30);
  if (what == "no-pinned") round_trip(n, 0);
  if (what == "one-pinned") round_trip(n, 1);
  if (what == "reuse") reuse(n);
  if (what == "small-chunks") small_chunks(n);
  return 0;
}
