// The FP64 numeric phases of the multigrid setup on the device: block-diagonal inversion, block
// norms for the join pass, the power iteration for lambda_max(D^-1 A), prolongator smoothing,
// A P and the Galerkin product P^T (A P) (crates/solidfem-solve/src/multigrid/setup.rs:269-321,
// 390-449, 527-647; transfer.rs:108-238; block.rs:186-245, 379-404).
//
// Built with -fmad=false and IEEE division and square root. Every output value is one thread's
// sequential sum over its contributions in the order the reference's serial loops visit them, so
// the device hierarchy equals the reference's to the bit. Parallelism comes from independent
// outputs: a thread owns one block row of the power iteration, one block of P, of A P or of the
// coarse matrix. The order-dependent graph work (strength, aggregation, tentative prolongator)
// and every sparsity pattern are built on the host (setup.cpp); only values live here.
//
// The one sequential reduction, the power iteration's norm (block.rs:398-404 sums the squares in
// index order), runs here too, in parallel and to the bit (norm_terms_kernel).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>

#include "device.h"

namespace sf {

namespace {

constexpr double kRankTolerance = 1e-10;  // transfer.rs:12
constexpr size_t kTentativeMaxSmem = 200 * 1024;  // an aggregate's rows x 6 modes, staged whole

const int kT = 256;

int grid_for(size_t n) { return (int)std::max<size_t>(1, std::min<size_t>((n + kT - 1) / kT, 148 * 32)); }

// C += A B for row-major dense blocks, the loop order of block.rs:229-245.
template <int AR, int MID, int BC>
__device__ __forceinline__ void add_product(double* out, const double* a, const double* b) {
#pragma unroll
  for (int r = 0; r < AR; ++r)
#pragma unroll
    for (int m = 0; m < MID; ++m) {
      double s = a[r * MID + m];
#pragma unroll
      for (int c = 0; c < BC; ++c) out[r * BC + c] += s * b[m * BC + c];
    }
}

__device__ __forceinline__ bool contains(const uint32_t* b, const uint32_t* e, uint32_t v) {
  while (b < e) {
    const uint32_t* mid = b + (e - b) / 2;
    if (*mid < v)
      b = mid + 1;
    else if (*mid > v)
      e = mid;
    else
      return true;
  }
  return false;
}

// Cholesky-based inverse of an SPD block (block.rs:186-224).
template <int N>
__device__ bool invert_spd(const double* in, double* out, double* pivot) {
  double lower[N * N];
  double inv[N * N];
#pragma unroll
  for (int i = 0; i < N * N; ++i) lower[i] = inv[i] = 0.0;
  for (int i = 0; i < N; ++i)
    for (int j = 0; j <= i; ++j) {
      double sum = in[i * N + j];
      for (int k = 0; k < j; ++k) sum -= lower[i * N + k] * lower[j * N + k];
      if (i == j) {
        if (!isfinite(sum) || sum <= 0.0) {
          *pivot = sum;
          return false;
        }
        lower[i * N + j] = sqrt(sum);
      } else {
        lower[i * N + j] = sum / lower[j * N + j];
      }
    }
  for (int c = 0; c < N; ++c)
    for (int i = c; i < N; ++i) {
      double sum = i == c ? 1.0 : 0.0;
      for (int k = c; k < i; ++k) sum -= lower[i * N + k] * inv[k * N + c];
      inv[i * N + c] = sum / lower[i * N + i];
    }
  for (int i = 0; i < N; ++i)
    for (int j = 0; j < N; ++j) {
      double sum = 0.0;
      for (int k = i > j ? i : j; k < N; ++k) sum += inv[k * N + i] * inv[k * N + j];
      out[i * N + j] = sum;
    }
  return true;
}

template <int N>
__global__ void inverse_diagonal_kernel(uint32_t rows, const uint32_t* __restrict__ starts,
                                        const uint32_t* __restrict__ cols, const double* __restrict__ vals,
                                        double* __restrict__ inv, unsigned long long* bad, double* __restrict__ pivots) {
  for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < rows; row += gridDim.x * blockDim.x) {
    const uint32_t* b = cols + starts[row];
    const uint32_t* e = cols + starts[row + 1];
    const uint32_t* lo = b;
    const uint32_t* hi = e;
    while (lo < hi) {
      const uint32_t* mid = lo + (hi - lo) / 2;
      if (*mid < row)
        lo = mid + 1;
      else
        hi = mid;
    }
    double pivot = 0.0;
    bool ok = lo != e && *lo == row &&
              invert_spd<N>(vals + (size_t)(lo - cols) * N * N, inv + (size_t)row * N * N, &pivot);
    if (!ok) {
      pivots[row] = pivot;
      atomicMin(bad, (unsigned long long)row);
    }
  }
}

template <int LEN>
__global__ void block_norms_kernel(size_t blocks, const double* __restrict__ vals, double* __restrict__ out) {
  for (size_t b = blockIdx.x * (size_t)blockDim.x + threadIdx.x; b < blocks; b += (size_t)gridDim.x * blockDim.x) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < LEN; ++i) {
      double v = vals[b * LEN + i];
      s += v * v;
    }
    out[b] = sqrt(s);
  }
}

// v = src / d, element by element, d on the device.
__global__ void scale_kernel(size_t n, const double* __restrict__ src, const double* __restrict__ d,
                             double* __restrict__ v) {
  const double by = *d;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    v[i] = src[i] / by;
}

// The power iteration's start vector (block.rs:379-382).
__global__ void start_vector_kernel(size_t n, double* __restrict__ v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const unsigned long long mixed = ((unsigned long long)i + 1) * 0x9E3779B97F4A7C15ull;
    v[i] = 0.5 + (double)(mixed >> 11) / (double)(1ull << 53);
  }
}

// ------------------------------------------------------------ the norm of a serial sum, in parallel
// s = 0; s = fl(s + fl(x_i x_i)) for i in order; sqrt(s): norm2 (block.rs:398-404) to the bit.
//
// While s stays in one binade [2^e, 2^(e+1)), s = m u with u = 2^(e-52) and an integer m, and adding
// y >= 0 adds an integer to m: floor(y / u), plus one when the fraction is above a half or is a half
// and m + floor(y / u) is odd (round to nearest, ties to even). So a run of terms is a function of
// m's parity alone, a pair of increments (for m even, for m odd), and pairs compose associatively:
// each chunk of 256 terms becomes one pair, computed by a warp, provided the chunk's binade is
// known. norm_sums_kernel predicts it from an ordinary parallel prefix of the chunk sums;
// norm_terms_kernel makes the pairs, and its last block walks the chunks in order, 32 at a time,
// and takes a pair only when s really lies in the predicted binade and stays in it; else it adds
// the chunk's terms one by one. The prediction therefore decides the time only, never a bit. The
// serial chunks are the first one and those where s crosses a power of two, about log2(chunks).
//
// The walk's dependent additions bound it (one chunk serially is 256 of them, about 1.3 us). On
// the host this sum took 0.8 ms for the gate plate's 603,000 unknowns, plus the iterate's copy and
// a synchronization each, 20 times a level.
constexpr int kNormChunk = 256;   // terms per chunk: eight consecutive ones per lane
constexpr int kNormThreads = 256;
constexpr int kNoBinade = INT_MIN;

__device__ __forceinline__ int binade(double s) {
  const int e = (int)((__double_as_longlong(s) >> 52) & 0x7ff) - 1023;
  return s > 0.0 && e >= -900 && e <= 900 ? e : kNoBinade;  // no subnormal, infinite or NaN sums
}

struct Increment {
  unsigned long long even, odd;
};
__device__ __forceinline__ Increment then(const Increment& l, const Increment& r) {
  Increment t;
  t.even = l.even + ((l.even & 1) ? r.odd : r.even);
  t.odd = l.odd + ((l.odd & 1) ? r.even : r.odd);
  return t;
}

// True in every thread of the grid's last block to arrive.
__device__ __forceinline__ bool last_block(unsigned* ticket) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last) *ticket = 0u;
  }
  __syncthreads();
  __threadfence();
  return last;
}

// A warp per chunk: its sum, in any order; then each chunk's binade by the prefix of the sums.
__global__ void __launch_bounds__(kNormThreads) norm_sums_kernel(size_t n, uint32_t chunks, const double* __restrict__ x,
                                                                 double* sums, int* __restrict__ binades,
                                                                 unsigned* ticket) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t c = blockIdx.x * (kNormThreads / 32) + warp;
  if (c < chunks) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kNormChunk / 32; ++k) {
      const size_t i = (size_t)c * kNormChunk + 32 * k + lane;
      const double v = i < n ? x[i] : 0.0;
      s += v * v;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) __stcg(sums + c, s);
  }
  if (!last_block(ticket)) return;
  // exclusive prefix: each thread a run of chunks, the threads' totals scanned in shared memory
  __shared__ double total[kNormThreads];
  const uint32_t per = (chunks + kNormThreads - 1) / kNormThreads;
  const uint32_t c0 = min(chunks, threadIdx.x * per), c1 = min(chunks, c0 + per);
  double mine = 0.0;
  for (uint32_t k = c0; k < c1; ++k) mine += __ldcg(sums + k);
  total[threadIdx.x] = mine;
  __syncthreads();
  for (int o = 1; o < kNormThreads; o <<= 1) {
    const double t = threadIdx.x >= o ? total[threadIdx.x - o] : 0.0;
    __syncthreads();
    total[threadIdx.x] += t;
    __syncthreads();
  }
  double before = total[threadIdx.x] - mine;
  if (threadIdx.x == 0) before = 0.0;
  for (uint32_t k = c0; k < c1; ++k) {
    const double after = before + __ldcg(sums + k);
    const int e = binade(before);
    binades[k] = e == binade(after) ? e : kNoBinade;
    before = after;
  }
}

// Chunk c's pair for the binade e, in lane 0 of the warp that makes it.
__device__ __forceinline__ Increment chunk_increment(size_t n, uint32_t c, const double* __restrict__ x, int e) {
  constexpr int kPer = kNormChunk / 32;
  const uint32_t lane = threadIdx.x & 31;
  const double scale = __longlong_as_double((long long)(52 - e + 1023) << 52);  // 1 / u
  Increment t = {0, 0};
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const size_t i = (size_t)c * kNormChunk + lane * kPer + k;
    const double v = i < n ? x[i] : 0.0;
    // y / u exactly (a result below one half may round, and stays below one half); a term past
    // the binade's end is held at 2^53, which no s in the binade survives.
    const double q = fmin(v * v * scale, 9007199254740992.0), whole = floor(q), part = q - whole;
    const unsigned long long m = (unsigned long long)whole;
    Increment one;
    one.even = m + (part > 0.5 || (part == 0.5 && (m & 1)) ? 1 : 0);
    one.odd = m + (part > 0.5 || (part == 0.5 && !(m & 1)) ? 1 : 0);
    t = then(t, one);
  }
  for (int o = 1; o < 32; o <<= 1) {
    Increment r;
    r.even = __shfl_down_sync(0xffffffffu, t.even, o);
    r.odd = __shfl_down_sync(0xffffffffu, t.odd, o);
    t = then(t, r);
  }
  t.even = min(t.even, 1ull << 53);
  t.odd = min(t.odd, 1ull << 53);
  return t;
}

// The walk over the chunks by one warp; y is its buffer of kNormChunk terms. Every lane returns s.
template <class Binade, class Pair>
__device__ __forceinline__ double norm_walk(size_t n, uint32_t chunks, const double* __restrict__ x, double* y,
                                            Binade&& binade_of, Pair&& pair_of) {
  constexpr int kPer = kNormChunk / 32;
  const uint32_t lane = threadIdx.x & 31;
  double s = 0.0;  // the same in every lane
  // s after the increment `t`, when it stays in its binade
  auto advance = [&](const Increment& t) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(s);
    const unsigned long long m = (bits & ((1ull << 52) - 1)) | (1ull << 52);
    const unsigned long long to = m + ((m & 1) ? t.odd : t.even);
    if (to >> 53) return false;
    s = __longlong_as_double((long long)((bits & ~((1ull << 52) - 1)) | (to & ((1ull << 52) - 1))));
    return true;
  };
  for (uint32_t b = 0; b < chunks; b += 32) {
    const uint32_t mine = b + lane;
    int e = kNoBinade;
    Increment p = {0, 0};
    if (mine < chunks) {
      e = binade_of(mine);
      if (e != kNoBinade) p = pair_of(mine);
    }
    const int now = binade(s);
    if (now != kNoBinade && __all_sync(0xffffffffu, mine >= chunks || e == now)) {
      Increment t = p;
      for (int o = 1; o < 32; o <<= 1) {
        Increment r;
        r.even = __shfl_down_sync(0xffffffffu, t.even, o);
        r.odd = __shfl_down_sync(0xffffffffu, t.odd, o);
        t = then(t, r);
      }
      t.even = __shfl_sync(0xffffffffu, t.even, 0);
      t.odd = __shfl_sync(0xffffffffu, t.odd, 0);
      if (advance(t)) continue;
    }
    for (int j = 0; j < 32 && b + j < chunks; ++j) {
      Increment t;
      t.even = __shfl_sync(0xffffffffu, p.even, j);
      t.odd = __shfl_sync(0xffffffffu, p.odd, j);
      const int ej = __shfl_sync(0xffffffffu, e, j);
      if (ej != kNoBinade && ej == binade(s) && advance(t)) continue;
      __syncwarp();
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const size_t i = (size_t)(b + j) * kNormChunk + 32 * k + lane;
        const double v = i < n ? x[i] : 0.0;
        y[32 * k + lane] = v * v;  // adding the zeros past the end changes nothing
      }
      __syncwarp();
#pragma unroll 16
      for (int i = 0; i < kNormChunk; ++i) s += y[i];
    }
  }
  return s;
}

__global__ void __launch_bounds__(kNormThreads) norm_terms_kernel(size_t n, uint32_t chunks, const double* __restrict__ x,
                                                                  const int* __restrict__ binades, Increment* pairs,
                                                                  unsigned* ticket, double* __restrict__ norm) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t c = blockIdx.x * (kNormThreads / 32) + warp;
  if (c < chunks && binades[c] != kNoBinade) {
    const Increment t = chunk_increment(n, c, x, binades[c]);
    if (lane == 0) {
      __stcg(&pairs[c].even, t.even);
      __stcg(&pairs[c].odd, t.odd);
    }
  }
  if (!last_block(ticket) || warp != 0) return;
  __shared__ double y[kNormChunk];
  const double s = norm_walk(
      n, chunks, x, y, [&](uint32_t k) { return __ldg(binades + k); },
      [&](uint32_t k) {
        Increment p;
        p.even = __ldcg(&pairs[k].even);
        p.odd = __ldcg(&pairs[k].odd);
        return p;
      });
  if (lane == 0) *norm = sqrt(s);
}

// The norm and v = x / norm of a small vector in one block, a chunk to a warp: the three launches of
// a large one cost more than their work (a level of 318 unknowns: its 20 power iterations
// 0.69 -> 0.55 ms).
constexpr uint32_t kSmallChunks = 32;
__global__ void __launch_bounds__(32 * kSmallChunks) small_normalize_kernel(size_t n, uint32_t chunks,
                                                                            const double* __restrict__ x,
                                                                            double* __restrict__ norm,
                                                                            double* __restrict__ v) {
  __shared__ double sums[kSmallChunks], y[kNormChunk], length;
  __shared__ int binades[kSmallChunks];
  __shared__ Increment pairs[kSmallChunks];
  const uint32_t lane = threadIdx.x & 31, c = threadIdx.x >> 5;
  double s = 0.0;
  if (c < chunks)
#pragma unroll
    for (int k = 0; k < kNormChunk / 32; ++k) {
      const size_t i = (size_t)c * kNormChunk + 32 * k + lane;
      const double w = i < n ? x[i] : 0.0;
      s += w * w;
    }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) sums[c] = s;
  __syncthreads();
  if (c < chunks) {
    double before = 0.0;
    for (uint32_t k = 0; k < c; ++k) before += sums[k];
    const int e = binade(before), use = e == binade(before + sums[c]) ? e : kNoBinade;
    Increment t = {0, 0};
    if (use != kNoBinade) t = chunk_increment(n, c, x, use);
    if (lane == 0) {
      binades[c] = use;
      pairs[c] = t;
    }
  }
  __syncthreads();
  if (c == 0) {
    const double total = norm_walk(
        n, chunks, x, y, [&](uint32_t k) { return binades[k]; }, [&](uint32_t k) { return pairs[k]; });
    if (lane == 0) *norm = length = sqrt(total);
  }
  __syncthreads();
  const double by = length;
  for (size_t i = threadIdx.x; i < n; i += blockDim.x) v[i] = x[i] / by;
}

// s2 = D^-1 (A v) for one block row per thread, in the order of setup.rs:404-432.
// One power step s2 = D^-1 (A v) (setup.rs:390-449). Lane p of a team of N lanes owns component
// p of a block row: its sum runs over the row's blocks in column order and, inside a block, over
// q in order, one running sum, as the reference's serial loop; the team's N sums then meet by
// shuffles for D^-1 y, again summed in q order. A warp holds 32 / N teams (10 rows of 3, 5 of
// 6), so a block's N value rows are read by N neighbouring lanes.
template <int N>
__global__ void power_step_kernel(uint32_t rows, const uint32_t* __restrict__ starts, const uint32_t* __restrict__ cols,
                                  const double* __restrict__ vals, const double* __restrict__ inv,
                                  const double* __restrict__ v, double* __restrict__ s2) {
  constexpr uint32_t kTeams = 32 / N;
  const uint32_t lane = threadIdx.x & 31, team = lane / N, p = lane - team * N;
  const bool on = team < kTeams;
  const uint32_t warps = blockDim.x >> 5;
  const uint32_t warp0 = blockIdx.x * warps + (threadIdx.x >> 5);
  for (uint32_t base = warp0 * kTeams; base < rows; base += gridDim.x * warps * kTeams) {
    const uint32_t row = base + team;
    const bool live = on && row < rows;
    double y = 0.0;
    if (live) {
      for (uint32_t at = starts[row]; at < starts[row + 1]; ++at) {
        const double* b = vals + (size_t)at * N * N + (size_t)p * N;
        const double* x = v + (size_t)cols[at] * N;
        double sum = y;
#pragma unroll
        for (int q = 0; q < N; ++q) sum += b[q] * x[q];
        y = sum;
      }
    }
    const uint32_t first = team * N;
    double yq[N];
#pragma unroll
    for (int q = 0; q < N; ++q) yq[q] = __shfl_sync(0xffffffffu, y, (first + q) & 31);
    if (live) {
      const double* d = inv + (size_t)row * N * N + (size_t)p * N;
      double sum = 0.0;
#pragma unroll
      for (int q = 0; q < N; ++q) sum += d[q] * yq[q];
      s2[(size_t)row * N + p] = sum;
    }
  }
}

// Row r of a union pattern: the sorted distinct columns inner_cols[k] over the inner rows j of r's
// outer list (j = r itself first when `self`); with inner_starts null each j has the one column
// inner_cols[j]. A warp per row sets the columns' bits in its own bitmap of `words` words in shared
// memory, then walks the bitmap in order: 32 words at a time, a warp prefix sum of their popcounts
// places each word's set bits. The count pass (out_starts null) writes the row's column count to
// out[r]; the fill pass writes the columns at out[out_starts[r] ..]. Every bit is cleared after use.
__global__ void union_rows_kernel(uint32_t rows, uint32_t words, const uint32_t* __restrict__ outer_starts,
                                  const uint32_t* __restrict__ outer_idx, int self,
                                  const uint32_t* __restrict__ inner_starts, const uint32_t* __restrict__ inner_cols,
                                  const uint32_t* __restrict__ out_starts, uint32_t* __restrict__ out) {
  extern __shared__ uint32_t union_bits[];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  uint32_t* bm = union_bits + (size_t)warp * words;
  for (uint32_t i = lane; i < words; i += 32) bm[i] = 0;
  __syncwarp();
  for (uint32_t r = blockIdx.x * warps + warp; r < rows; r += gridDim.x * warps) {
    const uint32_t o0 = outer_starts[r], n = outer_starts[r + 1] - o0 + (self ? 1u : 0u);
    for (uint32_t t = lane; t < n; t += 32) {
      const uint32_t j = self ? (t == 0 ? r : outer_idx[o0 + t - 1]) : outer_idx[o0 + t];
      if (inner_starts) {
        for (uint32_t k = inner_starts[j]; k < inner_starts[j + 1]; ++k) {
          const uint32_t c = inner_cols[k];
          atomicOr(&bm[c >> 5], 1u << (c & 31));
        }
      } else {
        const uint32_t c = inner_cols[j];
        atomicOr(&bm[c >> 5], 1u << (c & 31));
      }
    }
    __syncwarp();
    const uint32_t base = out_starts ? out_starts[r] : 0u;
    uint32_t total = 0;
    for (uint32_t w0 = 0; w0 < words; w0 += 32) {
      const uint32_t w = w0 + lane;
      uint32_t bits = w < words ? bm[w] : 0u;
      const uint32_t cnt = (uint32_t)__popc(bits);
      uint32_t inc = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(full, inc, o);
        if (lane >= o) inc += v;
      }
      if (out_starts) {
        uint32_t at = base + total + (inc - cnt);
        while (bits) {
          out[at++] = w * 32u + (uint32_t)(__ffs(bits) - 1);
          bits &= bits - 1;
        }
      }
      if (w < words) bm[w] = 0u;
      total += __shfl_sync(full, inc, 31);
    }
    if (!out_starts && lane == 0) out[r] = total;
    __syncwarp();
  }
}

// The block row of each entry of a block pattern.
__global__ void entry_rows_kernel(uint32_t rows, const uint32_t* __restrict__ starts, uint32_t* __restrict__ out) {
  for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < rows; row += gridDim.x * blockDim.x)
    for (uint32_t j = starts[row]; j < starts[row + 1]; ++j) out[j] = row;
}

// The transpose's parts: column counts; each entry into its column's list in any order; then a block
// per column puts its list in ascending order (an entry's place is the number of smaller ones, read
// from shared memory: lists hold tens to hundreds of entries) and adds the entries' rows.
__global__ void column_counts_kernel(size_t entries, const uint32_t* __restrict__ cols, uint32_t* counts) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < entries; i += (size_t)gridDim.x * blockDim.x)
    atomicAdd(counts + cols[i], 1u);
}
__global__ void transpose_fill_kernel(size_t entries, const uint32_t* __restrict__ cols, uint32_t* cursors,
                                      uint32_t* __restrict__ at) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < entries; i += (size_t)gridDim.x * blockDim.x)
    at[atomicAdd(cursors + cols[i], 1u)] = (uint32_t)i;
}
__global__ void transpose_sort_kernel(uint32_t width, const uint32_t* __restrict__ starts,
                                      const uint32_t* __restrict__ entry_row, uint32_t* __restrict__ at,
                                      uint32_t* __restrict__ rows) {
  extern __shared__ uint32_t list[];
  for (uint32_t c = blockIdx.x; c < width; c += gridDim.x) {
    const uint32_t b = starts[c], n = starts[c + 1] - b;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) list[i] = at[b + i];
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
      const uint32_t mine = list[i];
      uint32_t place = 0;
      for (uint32_t k = 0; k < n; ++k) place += list[k] < mine;
      at[b + place] = mine;
      rows[b + place] = entry_row[mine];
    }
    __syncthreads();
  }
}

// One block of P = T - omega D^-1 A_f T (transfer.rs:108-152): A's blocks whose column is the row
// or a smoothing neighbour act on that column's tentative block; the others are lumped onto the
// row's own (src = row). Contributions to this block's coarse column add in A's column order.
template <int N>
__global__ void smooth_kernel(size_t entries, const uint32_t* __restrict__ entry_row, const uint32_t* __restrict__ p_cols,
                              const uint32_t* __restrict__ a_starts, const uint32_t* __restrict__ a_cols,
                              const double* __restrict__ a_vals, const uint32_t* __restrict__ n_starts,
                              const uint32_t* __restrict__ n_cols, const uint32_t* __restrict__ aggregate,
                              const double* __restrict__ t_vals, const double* __restrict__ inv, double omega,
                              double* __restrict__ p_vals) {
  constexpr int L = N * 6;
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < entries; j += (size_t)gridDim.x * blockDim.x) {
    const uint32_t row = entry_row[j], c = p_cols[j];
    const uint32_t* nb = n_cols + n_starts[row];
    const uint32_t* ne = n_cols + n_starts[row + 1];
    double acc[L];
#pragma unroll
    for (int i = 0; i < L; ++i) acc[i] = 0.0;
    for (uint32_t at = a_starts[row]; at < a_starts[row + 1]; ++at) {
      const uint32_t col = a_cols[at];
      const uint32_t src = (col == row || contains(nb, ne, col)) ? col : row;
      if (aggregate[src] != c) continue;
      add_product<N, N, 6>(acc, a_vals + (size_t)at * N * N, t_vals + (size_t)src * L);
    }
    const double* d = inv + (size_t)row * N * N;
    const double* t = t_vals + (size_t)row * L;
    const bool own = c == aggregate[row];
    double* out = p_vals + j * L;
#pragma unroll
    for (int r = 0; r < N; ++r)
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        double s = 0.0;
#pragma unroll
        for (int m = 0; m < N; ++m) s += d[r * N + m] * acc[m * 6 + q];
        double tv = own ? t[r * 6 + q] : 0.0;
        out[r * 6 + q] = tv - omega * s;
      }
  }
}

// One block of A P (transfer.rs:155-169): A's blocks in column order, each times the blocks of
// P's row at that column whose coarse column is this block's.
template <int N>
__global__ void product_kernel(size_t entries, const uint32_t* __restrict__ entry_row, const uint32_t* __restrict__ ap_cols,
                               const uint32_t* __restrict__ a_starts, const uint32_t* __restrict__ a_cols,
                               const double* __restrict__ a_vals, const uint32_t* __restrict__ p_starts,
                               const uint32_t* __restrict__ p_cols, const double* __restrict__ p_vals,
                               double* __restrict__ ap_vals) {
  constexpr int L = N * 6;
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < entries; j += (size_t)gridDim.x * blockDim.x) {
    const uint32_t row = entry_row[j], c = ap_cols[j];
    double acc[L];
#pragma unroll
    for (int i = 0; i < L; ++i) acc[i] = 0.0;
    for (uint32_t at = a_starts[row]; at < a_starts[row + 1]; ++at) {
      const uint32_t col = a_cols[at];
      for (uint32_t in = p_starts[col]; in < p_starts[col + 1]; ++in) {
        const uint32_t pc = p_cols[in];
        if (pc < c) continue;
        if (pc == c) add_product<N, N, 6>(acc, a_vals + (size_t)at * N * N, p_vals + (size_t)in * L);
        break;
      }
    }
    double* out = ap_vals + j * L;
#pragma unroll
    for (int i = 0; i < L; ++i) out[i] = acc[i];
  }
}

// ROWS rows of a block of P^T (A P) per thread (transfer.rs:173-238): the fine rows of P's column in
// ascending order, those rows of each P block transposed times the A P block of that fine row at this
// block's column; a zero on the diagonal of a diagonal block becomes one (finish_level,
// setup.rs:650-695). A coarse row sums tens to hundreds of fine rows, and where a level has few blocks
// the chain of one thread bounds it: six threads a block then, each of the same terms in the same
// order. Where the blocks fill the device, a whole block to a thread reads each A P block and searches
// for it once instead of six times (kSplit below).
template <int N, int ROWS>
__global__ void galerkin_kernel(size_t entries, const uint32_t* __restrict__ entry_row, const uint32_t* __restrict__ c_cols,
                                const uint32_t* __restrict__ pt_starts, const uint32_t* __restrict__ pt_rows,
                                const uint32_t* __restrict__ pt_at, const double* __restrict__ p_vals,
                                const uint32_t* __restrict__ ap_starts, const uint32_t* __restrict__ ap_cols,
                                const double* __restrict__ ap_vals, double* __restrict__ c_vals) {
  constexpr int L = N * 6;
  constexpr int SHARES = 6 / ROWS;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < SHARES * entries; i += (size_t)gridDim.x * blockDim.x) {
    const size_t j = i / SHARES;
    const int r = (int)(i % SHARES) * ROWS;
    const uint32_t crow = entry_row[j], c = c_cols[j];
    double acc[ROWS][6];
#pragma unroll
    for (int o = 0; o < ROWS; ++o)
#pragma unroll
      for (int q = 0; q < 6; ++q) acc[o][q] = 0.0;
    for (uint32_t k = pt_starts[crow]; k < pt_starts[crow + 1]; ++k) {
      const uint32_t fine_row = pt_rows[k];
      const uint32_t* b = ap_cols + ap_starts[fine_row];
      const uint32_t* e = ap_cols + ap_starts[fine_row + 1];
      const uint32_t* lo = b;
      const uint32_t* hi = e;
      while (lo < hi) {
        const uint32_t* mid = lo + (hi - lo) / 2;
        if (*mid < c)
          lo = mid + 1;
        else
          hi = mid;
      }
      if (lo == e || *lo != c) continue;
      const double* pb = p_vals + (size_t)pt_at[k] * L + r;
      const double* ab = ap_vals + (size_t)(lo - ap_cols) * L;
#pragma unroll
      for (int o = 0; o < ROWS; ++o)
#pragma unroll
        for (int m = 0; m < N; ++m) {
          double s = pb[m * 6 + o];
#pragma unroll
          for (int q = 0; q < 6; ++q) acc[o][q] += s * ab[m * 6 + q];
        }
    }
    if (crow == c)
#pragma unroll
      for (int o = 0; o < ROWS; ++o)
#pragma unroll
        for (int q = 0; q < 6; ++q)
          if (q == r + o && acc[o][q] == 0.0) acc[o][q] = 1.0;
    double* out = c_vals + j * 36 + r * 6;
#pragma unroll
    for (int o = 0; o < ROWS; ++o)
#pragma unroll
      for (int q = 0; q < 6; ++q) out[o * 6 + q] = acc[o][q];
  }
}

// The tentative prolongator (setup.rs:327-386, orthonormalize_aggregate, transfer.rs:19-68): per
// aggregate, its members' rows of the near-null modes, orthonormalised column by column with two
// Gram-Schmidt passes against the earlier columns; a column whose remainder falls to
// RANK_TOLERANCE of its original norm is zeroed. One warp per aggregate stages the aggregate's
// rows (members in order, rb rows each, 6 modes) in shared memory; lane 0 runs every sum of the
// reference's loops in their order (sequential over the aggregate's rows), and the lanes share the
// element-wise updates, each of which depends only on its own entry. So T (written back at the
// members' own rows) and the coarse near-null space (the projections and remainders, 6 x 6 per
// aggregate) carry the host loops' bits.
__global__ void __launch_bounds__(32) tentative_kernel(uint32_t aggregates, int rb,
                                                       const uint32_t* __restrict__ member_starts,
                                                       const uint32_t* __restrict__ members,
                                                       const double* __restrict__ near_null, double* __restrict__ t,
                                                       double* __restrict__ coarse) {
  extern __shared__ double local[];  // lrows x 6
  const uint32_t a = blockIdx.x;
  const unsigned lane = threadIdx.x;
  if (a >= aggregates) return;
  const uint32_t m0 = member_starts[a];
  const uint32_t lrows = (member_starts[a + 1] - m0) * (uint32_t)rb;
  auto slot = [&](uint32_t r) { return ((size_t)members[m0 + r / rb] * rb + r % rb) * 6; };
  for (uint32_t r = lane; r < lrows; r += 32) {
    const size_t at = slot(r);
    for (int k = 0; k < 6; ++k) local[r * 6 + k] = near_null[at + k];
  }
  __syncwarp();
  double* c = coarse + (size_t)a * 36;
  if (lane == 0)
    for (int i = 0; i < 36; ++i) c[i] = 0.0;
  auto column_norm = [&](int col) {  // lane 0's sequential sum, broadcast
    double s = 0.0;
    if (lane == 0)
      for (uint32_t r = 0; r < lrows; ++r) s += local[r * 6 + col] * local[r * 6 + col];
    return __shfl_sync(0xffffffffu, sqrt(s), 0);
  };
  for (int col = 0; col < 6; ++col) {
    const double original = column_norm(col);
    for (int pass = 0; pass < 2; ++pass)
      for (int prev = 0; prev < col; ++prev) {
        double proj = 0.0;
        if (lane == 0) {
          for (uint32_t r = 0; r < lrows; ++r) proj += local[r * 6 + prev] * local[r * 6 + col];
          c[prev * 6 + col] += proj;
        }
        proj = __shfl_sync(0xffffffffu, proj, 0);
        for (uint32_t r = lane; r < lrows; r += 32) local[r * 6 + col] -= proj * local[r * 6 + prev];
        __syncwarp();
      }
    const double rem = column_norm(col);
    const bool drop = original == 0.0 || rem <= kRankTolerance * original;
    for (uint32_t r = lane; r < lrows; r += 32) local[r * 6 + col] = drop ? 0.0 : local[r * 6 + col] / rem;
    if (lane == 0) c[col * 6 + col] = drop ? 0.0 : rem;
    __syncwarp();
  }
  for (uint32_t r = lane; r < lrows; r += 32) {
    const size_t at = slot(r);
    for (int k = 0; k < 6; ++k) t[at + k] = local[r * 6 + k];
  }
}

// The free nodes' rigid-body modes (free_rigid_body_modes, rigid_modes.rs:36-83) about the centre
// and scale the host summed: for free block row r (node row_node[r]) the three rows
// [1 0 0 0 z -y], [0 1 0 -z 0 x], [0 0 1 y -x 0] of the scaled offsets, (row, mode) at 6 row + mode.
__global__ void rigid_modes_kernel(uint32_t rows, const uint32_t* __restrict__ row_node, const double* __restrict__ nodes,
                                   double cx, double cy, double cz, double scale, double* __restrict__ modes) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const double* p = nodes + (size_t)row_node[r] * 3;
  const double x = (p[0] - cx) * scale, y = (p[1] - cy) * scale, z = (p[2] - cz) * scale;
  const double v[18] = {1, 0, 0, 0, z, -y, 0, 1, 0, -z, 0, x, 0, 0, 1, y, -x, 0};
  double* m = modes + (size_t)r * 18;
  for (int i = 0; i < 18; ++i) m[i] = v[i];
}

// ------------------------------------------------------------ the coarsest level's dense factor
// DenseCholesky (block.rs:307-374) and the explicit inverse L^-T L^-1 the cycle applies, n up to
// DENSE_LIMIT, row-major n x n in device memory. Both run right-looking in panels of kPanel columns:
// a panel launch finishes the panel's rows of the factor and its rows of L^-1 (right-hand side the
// identity), an update launch subtracts the panel's terms from every later entry of both. An entry
// of L thus subtracts L[i][k] L[j][k], and an entry of L^-1 subtracts L[i][k] X[k][c], for k = 0, 1,
// ... in order from its original value, exactly the host's left-looking loops, so both have the
// host loops' bits (entries of X above the diagonal are exact zeros, which subtract nothing).
//
// The launches bound it, not the arithmetic: 2 n / 32 of them in a row, each a few microseconds
// (the panel's 32 dependent square roots and divisions, then the update's 32 terms per entry from
// shared memory). The panel's diagonal block is factored by one warp of every block, which is
// cheaper than a launch of its own. Before, one thread per column of L^-1 walked n^2 / 2 dependent
// global loads: a study's whole creation went from 11.2 to 6.3 ms at n = 318, from 35 to 7.4 ms at
// 714 and from 85 to 9.2 ms at 1,152.
constexpr int kPanel = 32;
constexpr int kDenseThreads = 128;

__global__ void dense_from_blocks_kernel(uint32_t rows, int rb, int cb, const uint32_t* __restrict__ starts,
                                         const uint32_t* __restrict__ cols, const double* __restrict__ vals, size_t n,
                                         double* __restrict__ f, double* __restrict__ li) {
  const uint32_t row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  for (uint32_t at = starts[row]; at < starts[row + 1]; ++at) {
    const size_t col = cols[at];
    for (int p = 0; p < rb; ++p)
      for (int q = 0; q < cb; ++q) f[((size_t)row * rb + p) * n + col * cb + q] = vals[(size_t)at * rb * cb + p * cb + q];
  }
  for (int p = 0; p < rb; ++p) li[((size_t)row * rb + p) * (n + 1)] = 1.0;
}

// Columns [j0, j0 + w) of the factor below their diagonal block (blocks below `row_blocks`, a
// thread per row) and rows [j0, j0 + w) of L^-1 (the other blocks, a thread per column). Every
// block factors the diagonal block for itself; the first non-positive pivot is recorded (its
// column and value) and everything stops there.
__global__ void __launch_bounds__(kDenseThreads) dense_panel_kernel(size_t n, size_t j0, unsigned row_blocks,
                                                                    double* __restrict__ f, double* __restrict__ li,
                                                                    unsigned long long* bad, double* pivot) {
  __shared__ double col[kPanel][kPanel + 1];  // col[j][i] = L[j0 + i][j0 + j]
  __shared__ int failed;
  if (threadIdx.x == 0) failed = *bad != ~0ull;
  __syncthreads();
  if (failed) return;
  const int w = (int)(n - j0 < (size_t)kPanel ? n - j0 : (size_t)kPanel);
  if (threadIdx.x < 32) {
    const int i = threadIdx.x;  // this lane's row of the diagonal block
    double a[kPanel];
#pragma unroll
    for (int j = 0; j < kPanel; ++j) a[j] = i < w && j <= i ? f[(j0 + i) * n + j0 + j] : 0.0;
#pragma unroll
    for (int j = 0; j < kPanel; ++j) {
      if (j >= w) break;
      const double sum = __shfl_sync(0xffffffffu, a[j], j);
      if (!isfinite(sum) || sum <= 0.0) {
        if (i == 0) {
          failed = 1;
          if (blockIdx.x == 0) {
            *pivot = sum;
            *bad = j0 + j;
          }
        }
        break;
      }
      const double d = sqrt(sum);
      const double l = i == j ? d : a[j] / d;
      a[j] = l;
      col[j][i] = l;
      __syncwarp();
#pragma unroll
      for (int m = j + 1; m < kPanel; ++m) a[m] -= l * col[j][m];  // entries m > i are never used
    }
  }
  __syncthreads();
  if (failed) return;
  if (blockIdx.x < row_blocks) {
    const size_t i = j0 + kPanel + (size_t)blockIdx.x * kDenseThreads + threadIdx.x;
    if (i >= n) return;
    double* row = f + i * n + j0;
    double a[kPanel];
#pragma unroll
    for (int j = 0; j < kPanel; ++j) a[j] = row[j];
#pragma unroll
    for (int j = 0; j < kPanel; ++j) {
      a[j] = a[j] / col[j][j];
#pragma unroll
      for (int m = j + 1; m < kPanel; ++m) a[m] -= a[j] * col[j][m];
    }
#pragma unroll
    for (int j = 0; j < kPanel; ++j) row[j] = a[j];
  } else {
    const size_t c = (size_t)(blockIdx.x - row_blocks) * kDenseThreads + threadIdx.x;
    if (c >= j0 + w) return;
    double x[kPanel];
#pragma unroll
    for (int r = 0; r < kPanel; ++r) x[r] = r < w ? li[(j0 + r) * n + c] : 0.0;
#pragma unroll
    for (int r = 0; r < kPanel; ++r) {
      if (r >= w) break;
      x[r] = x[r] / col[r][r];
      li[(j0 + r) * n + c] = x[r];
#pragma unroll
      for (int m = r + 1; m < kPanel; ++m) x[m] -= col[r][m] * x[r];  // rows m >= w are never used
    }
  }
}

// The panel's terms off every later row i: the factor's entries (i, j), j1 <= j <= i, lose
// L[i][k] L[j][k], the inverse's entries (i, c), c < j1, lose L[i][k] X[k][c], k ascending. A block
// of 256 threads per 32 x 32 tile, four entries a thread; columns below j1 are the inverse's.
__global__ void __launch_bounds__(256) dense_update_kernel(size_t n, size_t j0, double* __restrict__ f,
                                                           double* __restrict__ li, const unsigned long long* bad) {
  __shared__ double a[32][kPanel + 1];  // a[i][k] = L[i0 + i][j0 + k]
  __shared__ double b[kPanel][33];      // b[k][j]
  if (*bad != ~0ull) return;
  const size_t j1 = j0 + kPanel, i0 = j1 + (size_t)blockIdx.y * 32, c0 = (size_t)blockIdx.x * 32;
  const bool factor = c0 >= j1;
  if (factor && c0 > i0) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int r = ty; r < 32; r += 8) {
    a[r][tx] = i0 + r < n ? f[(i0 + r) * n + j0 + tx] : 0.0;
    if (factor)
      b[tx][r] = c0 + r < n ? f[(c0 + r) * n + j0 + tx] : 0.0;
    else
      b[r][tx] = li[(j0 + r) * n + c0 + tx];
  }
  __syncthreads();
  const size_t c = c0 + tx;
  if (c >= n) return;
  double* out = factor ? f : li;
  double s[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) s[q] = i0 + ty + 8 * q < n ? out[(i0 + ty + 8 * q) * n + c] : 0.0;
#pragma unroll 8
  for (int k = 0; k < kPanel; ++k) {
    const double v = b[k][tx];
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] -= a[ty + 8 * q][k] * v;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const size_t i = i0 + ty + 8 * q;
    if (i < n && !(factor && c > i)) out[i * n + c] = s[q];
  }
}

// A^-1 = L^-T L^-1, entry (i, j) summing k from max(i, j) up: 32 x 32 tiles, four entries a
// thread, 32 rows of L^-1 at a time in shared memory from the tile's first nonzero row on (the
// zeros above the diagonal add nothing).
__global__ void __launch_bounds__(256) gram_inverse_kernel(size_t n, const double* __restrict__ li,
                                                           double* __restrict__ out) {
  __shared__ double a[32][33], b[32][33];
  const size_t i0 = (size_t)blockIdx.y * 32, c0 = (size_t)blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (size_t k0 = i0 > c0 ? i0 : c0; k0 < n; k0 += 32) {
    for (int r = ty; r < 32; r += 8) {
      const bool in = k0 + r < n;
      a[r][tx] = in && i0 + tx < n ? li[(k0 + r) * n + i0 + tx] : 0.0;
      b[r][tx] = in && c0 + tx < n ? li[(k0 + r) * n + c0 + tx] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
      const double v = b[k][tx];
#pragma unroll
      for (int q = 0; q < 4; ++q) s[q] += a[k][ty + 8 * q] * v;
    }
    __syncthreads();
  }
  const size_t c = c0 + tx;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const size_t i = i0 + ty + 8 * q;
    if (i < n && c < n) out[i * n + c] = s[q];
  }
}

template <typename S>
__global__ void convert_kernel(size_t n, const double* __restrict__ in, S* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = (S)in[i];
}

// R = P^T block by block: R block o is P block src[o] transposed (rb x cb into cb x rb).
template <typename S>
__global__ void transpose_blocks_kernel(size_t blocks, int rb, int cb, const uint32_t* __restrict__ src,
                                        const double* __restrict__ in, S* __restrict__ out) {
  const int len = rb * cb;
  for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < blocks; o += (size_t)gridDim.x * blockDim.x) {
    const double* p = in + (size_t)src[o] * len;
    S* t = out + o * len;
    for (int a = 0; a < rb; ++a)
      for (int b = 0; b < cb; ++b) t[b * rb + a] = (S)p[a * cb + b];
  }
}

// Fills a SELL-32 copy from a block CSR matrix (f64 values, converted to S): one thread per slice
// lane places its row's columns and values at their chunked positions; padding stays zero.
template <typename S, int LEN>
__global__ void sell_fill_kernel(size_t slots, const uint32_t* __restrict__ sell_rows, const uint32_t* __restrict__ sell_len,
                                 const uint32_t* __restrict__ sell_start, uint32_t nrows,
                                 const uint32_t* __restrict__ starts, const uint32_t* __restrict__ cols,
                                 const double* __restrict__ in, uint32_t* __restrict__ out_cols, S* __restrict__ out) {
  constexpr int U = sell_chunk_blocks(LEN, (int)sizeof(S));
  constexpr int VEC = 16 / (int)sizeof(S);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < slots; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t row = sell_rows[i];
    if (row >= nrows) continue;
    const uint32_t s = (uint32_t)(i / 32), t = (uint32_t)(i % 32), n = sell_len[i], b0 = starts[row];
    for (uint32_t k = 0; k < n; ++k) {
      const size_t q = sell_start[s] + 32 * (k - k % U) + t * U + k % U;
      out_cols[q] = cols[b0 + k];
#pragma unroll
      for (int e = 0; e < LEN; ++e) out[sell_value_offset(q, LEN, U, VEC, e)] = (S)in[(size_t)(b0 + k) * LEN + e];
    }
  }
}

// Fills a split-row copy of a 6 x CB block CSR matrix: lane t = 6 m + p of a slice places row p
// of each block of its block row as a 1 x CB block at its chunked SELL position; the lane with
// p = 0 also places the block's column in the block row's shared column chunk.
template <typename S, int CB>
__global__ void split_fill_kernel(size_t slots, const uint32_t* __restrict__ sell_rows, const uint32_t* __restrict__ sell_len,
                                  const uint32_t* __restrict__ sell_start, uint32_t nrows,
                                  const uint32_t* __restrict__ starts, const uint32_t* __restrict__ cols,
                                  const double* __restrict__ in, uint32_t* __restrict__ out_cols, S* __restrict__ out) {
  constexpr int U = sell_chunk_blocks(CB, (int)sizeof(S));
  constexpr int VEC = 16 / (int)sizeof(S);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < slots; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t row = sell_rows[i];
    if (row >= nrows) continue;
    const uint32_t s = (uint32_t)(i / 32), t = (uint32_t)(i % 32), m = t / 6, p = t % 6;
    const uint32_t n = sell_len[i], b0 = starts[row];
    const size_t cbase = (size_t)(sell_start[s] / 32) * kSplitRowsPerSlice + (size_t)m * U;
    for (uint32_t k = 0; k < n; ++k) {
      const uint32_t c = k / U, u = k % U;
      const size_t q = sell_start[s] + 32 * (size_t)(c * U) + t * U + u;
      if (p == 0) out_cols[cbase + (size_t)kSplitRowsPerSlice * U * c + u] = cols[b0 + k];
#pragma unroll
      for (int e = 0; e < CB; ++e)
        out[sell_value_offset(q, CB, U, VEC, e)] = (S)in[(size_t)(b0 + k) * 6 * CB + p * CB + e];
    }
  }
}

// How many of the lanes' `block`s (ascending, a lane each) are below `key`.
__device__ __forceinline__ uint32_t lanes_below(uint32_t block, uint32_t key) {
  uint32_t at = 0;
#pragma unroll
  for (uint32_t step = 16; step > 0; step >>= 1)
    if (__shfl_sync(0xffffffffu, block, at + step - 1) < key) at += step;
  return at + (__shfl_sync(0xffffffffu, block, at) < key);
}

// A warp per block row merges its three scalar rows (and, for the padded last block row, its own
// diagonal block), 32 entries of each at a time: what lies below the first block column that may go
// on past a row's 32 is taken. A block's place is the number of first entries of smaller blocks, a
// first entry being a block's first in its row where no row before it has the block. Columns are
// strictly ascending, so a block has three entries of a row at most and every step takes 29 or more
// of some row. A thread per block row read a dense row as one chain of loads: 91,125 unknowns with
// one full row and column were created in 48 ms.
// Block rows [first_row, end_row); cols and scalars hold the entries from `entry` on.
__global__ void padded_blocks_kernel(uint64_t n, uint32_t first_row, uint32_t end_row, uint64_t entry,
                                     const uint64_t* __restrict__ rs, const uint32_t* __restrict__ cols, const double* __restrict__ scalars,
                                     const uint32_t* __restrict__ out_starts, uint32_t* __restrict__ out,
                                     double* __restrict__ vals) {
  constexpr uint32_t kNone = 0xffffffffu;  // past a row's end
  const uint32_t lane = threadIdx.x & 31, b = first_row + blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= end_row) return;
  uint64_t at[3], end[3];  // within cols and scalars
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    const uint64_t r = 3 * (uint64_t)b + p;
    at[p] = r < n ? rs[r] - entry : 0;
    end[p] = r < n ? rs[r + 1] - entry : 0;
  }
  bool own = 3 * (uint64_t)b + 3 > n;  // the padding's diagonal block is still to come
  const size_t base = out_starts ? out_starts[b] : 0;
  uint32_t count = 0;
  while (own || at[0] < end[0] || at[1] < end[1] || at[2] < end[2]) {
    uint32_t col[3], block[3], limit = kNone;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      col[p] = at[p] + lane < end[p] ? cols[at[p] + lane] : kNone;
      block[p] = col[p] == kNone ? kNone : col[p] / 3;
      const uint32_t last = __shfl_sync(0xffffffffu, block[p], 31);
      if (at[p] + 32 < end[p]) limit = min(limit, last);
    }
    unsigned lead[3];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint32_t before = __shfl_up_sync(0xffffffffu, block[p], 1);
      bool first = block[p] < limit && (lane == 0 || before != block[p]);
#pragma unroll
      for (int q = 0; q < p; ++q) {
        const uint32_t k = lanes_below(block[q], block[p]);
        if (__shfl_sync(0xffffffffu, block[q], k & 31) == block[p] && k < 32) first = false;
      }
      lead[p] = __ballot_sync(0xffffffffu, first);
    }
    const bool own_now = own && b < limit;
    const bool own_lead =
        own_now && !__any_sync(0xffffffffu, block[0] == b || block[1] == b || block[2] == b);
    // the place of block `key` (every lane asks together)
    auto place = [&](uint32_t key) {
      uint32_t k = count + (own_lead && b < key);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const uint32_t below = lanes_below(block[q], key);
        k += __popc(below < 32 ? lead[q] & ((1u << below) - 1u) : lead[q]);
      }
      return k;
    };
    if (out_starts) {
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const size_t k = base + place(block[p]);
        if (block[p] < limit) {
          if (lead[p] >> lane & 1u) out[k] = block[p];
          vals[k * 9 + 3 * p + col[p] % 3] = scalars[at[p] + lane];
        }
      }
      if (own_now) {
        const size_t k = base + place(b);
        if (lane == 0) {
          if (own_lead) out[k] = b;
          for (int p = 0; p < 3; ++p)
            if (3 * (uint64_t)b + p >= n) vals[k * 9 + 4 * p] = 1.0;
        }
      }
    }
    count += __popc(lead[0]) + __popc(lead[1]) + __popc(lead[2]) + own_lead;
#pragma unroll
    for (int p = 0; p < 3; ++p) at[p] += __popc(__ballot_sync(0xffffffffu, block[p] < limit));
    if (own_now) own = false;
  }
  if (!out_starts && lane == 0) out[b] = count;
}

// Copies listed blocks out of (gather) or back into (scatter) a block array.
__global__ void gather_blocks_kernel(size_t count, int len, const uint32_t* __restrict__ idx,
                                     const double* __restrict__ in, double* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count * len; i += (size_t)gridDim.x * blockDim.x)
    out[i] = in[(size_t)idx[i / len] * len + i % len];
}
__global__ void scatter_blocks_kernel(size_t count, int len, const uint32_t* __restrict__ idx,
                                      const double* __restrict__ in, double* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count * len; i += (size_t)gridDim.x * blockDim.x)
    out[(size_t)idx[i / len] * len + i % len] = in[i];
}
__global__ void set_values_kernel(size_t count, const uint32_t* __restrict__ idx, const double* __restrict__ vals,
                                  double* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
    out[idx[i]] = vals[i];
}

}  // namespace

sf_status setup_padded_blocks(cudaStream_t st, uint64_t n, uint32_t first, uint32_t end, uint64_t entry,
                              const uint64_t* rs, const uint32_t* cols, const double* scalars,
                              const uint32_t* out_starts, uint32_t* out, double* vals) {
  if (end <= first) return SF_OK;
  padded_blocks_kernel<<<(end - first + 3) / 4, 128, 0, st>>>(n, first, end, entry, rs, cols, scalars, out_starts, out,
                                                              vals);
  return cuda_check(cudaGetLastError(), "padded blocks");
}

sf_status setup_gather_blocks(cudaStream_t st, size_t count, int len, const uint32_t* idx, const double* in,
                              double* out) {
  if (count == 0) return SF_OK;
  gather_blocks_kernel<<<grid_for(count * len), kT, 0, st>>>(count, len, idx, in, out);
  return cuda_check(cudaGetLastError(), "gather blocks");
}

sf_status setup_scatter_blocks(cudaStream_t st, size_t count, int len, const uint32_t* idx, const double* in,
                               double* out) {
  if (count == 0) return SF_OK;
  scatter_blocks_kernel<<<grid_for(count * len), kT, 0, st>>>(count, len, idx, in, out);
  return cuda_check(cudaGetLastError(), "scatter blocks");
}

sf_status setup_set_values(cudaStream_t st, size_t count, const uint32_t* idx, const double* vals, double* out) {
  if (count == 0) return SF_OK;
  set_values_kernel<<<grid_for(count), kT, 0, st>>>(count, idx, vals, out);
  return cuda_check(cudaGetLastError(), "set values");
}

sf_status setup_inverse_diagonal(cudaStream_t st, uint32_t rows, int rb, const uint32_t* starts, const uint32_t* cols,
                                 const double* vals, double* inv, unsigned long long* bad, double* pivots) {
  if (rows == 0) return SF_OK;
  if (rb == 3)
    inverse_diagonal_kernel<3><<<grid_for(rows), kT, 0, st>>>(rows, starts, cols, vals, inv, bad, pivots);
  else
    inverse_diagonal_kernel<6><<<grid_for(rows), kT, 0, st>>>(rows, starts, cols, vals, inv, bad, pivots);
  return cuda_check(cudaGetLastError(), "inverse diagonal");
}

sf_status setup_block_norms(cudaStream_t st, size_t blocks, int len, const double* vals, double* out) {
  if (blocks == 0) return SF_OK;
  if (len == 9)
    block_norms_kernel<9><<<grid_for(blocks), kT, 0, st>>>(blocks, vals, out);
  else
    block_norms_kernel<36><<<grid_for(blocks), kT, 0, st>>>(blocks, vals, out);
  return cuda_check(cudaGetLastError(), "block norms");
}

sf_status setup_power_step(cudaStream_t st, uint32_t rows, int rb, const uint32_t* starts, const uint32_t* cols,
                           const double* vals, const double* inv, const double* v, double* s2) {
  if (rows == 0) return SF_OK;
  if (rb == 3)
    power_step_kernel<3><<<grid_for((size_t)rows * 32 / 10), kT, 0, st>>>(rows, starts, cols, vals, inv, v, s2);
  else
    power_step_kernel<6><<<grid_for((size_t)rows * 32 / 5), kT, 0, st>>>(rows, starts, cols, vals, inv, v, s2);
  return cuda_check(cudaGetLastError(), "power step");
}

size_t setup_norm_scratch(size_t n) {
  const size_t chunks = (n + kNormChunk - 1) / kNormChunk;
  return 256 + chunks * (sizeof(Increment) + 8 + 4);
}

sf_status setup_start_vector(cudaStream_t st, size_t n, double* v) {
  if (n == 0) return SF_OK;
  start_vector_kernel<<<grid_for(n), kT, 0, st>>>(n, v);
  return cuda_check(cudaGetLastError(), "start vector");
}

sf_status setup_normalize(cudaStream_t st, size_t n, const double* src, void* scratch, double* norm, double* v) {
  if (n == 0) return SF_OK;
  const uint32_t chunks = (uint32_t)((n + kNormChunk - 1) / kNormChunk);
  if (chunks <= kSmallChunks) {
    small_normalize_kernel<<<1, 32 * kSmallChunks, 0, st>>>(n, chunks, src, norm, v);
    return cuda_check(cudaGetLastError(), "normalize");
  }
  unsigned* tickets = (unsigned*)scratch;
  Increment* pairs = (Increment*)((char*)scratch + 256);
  double* sums = (double*)(pairs + chunks);
  int* binades = (int*)(sums + chunks);
  const unsigned grid = (chunks + kNormThreads / 32 - 1) / (kNormThreads / 32);
  norm_sums_kernel<<<grid, kNormThreads, 0, st>>>(n, chunks, src, sums, binades, tickets);
  norm_terms_kernel<<<grid, kNormThreads, 0, st>>>(n, chunks, src, binades, pairs, tickets + 1, norm);
  scale_kernel<<<grid_for(n), kT, 0, st>>>(n, src, norm, v);
  return cuda_check(cudaGetLastError(), "normalize");
}

sf_status setup_union_rows(cudaStream_t st, uint32_t rows, uint32_t width, const uint32_t* outer_starts,
                           const uint32_t* outer_idx, bool self, const uint32_t* inner_starts,
                           const uint32_t* inner_cols, const uint32_t* out_starts, uint32_t* out) {
  const uint32_t words = (width + 31) / 32;
  const size_t per_warp = (size_t)std::max<uint32_t>(words, 1) * 4;
  const size_t limit = 200 * 1024;
  if (per_warp > limit) return fail(SF_INVALID_ARGUMENT, "union pattern wider than one warp's bitmap");
  const int warps = (int)std::max<size_t>(1, std::min<size_t>(8, limit / per_warp));
  const size_t smem = per_warp * warps;
  if (rows == 0) return SF_OK;
  const void* k = (const void*)union_rows_kernel;
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
  const int grid = (int)std::max<size_t>(1, std::min<size_t>((rows + warps - 1) / warps, 148 * 16));
  union_rows_kernel<<<grid, 32 * warps, smem, st>>>(rows, words, outer_starts, outer_idx, self ? 1 : 0, inner_starts,
                                                    inner_cols, out_starts, out);
  return cuda_check(cudaGetLastError(), "union pattern");
}

// Strong neighbours by geometry (aggregate.rs:53-69): a thread per row takes the squared distance
// to each other column term for term (no contraction, as on the host), the row's closest one, and
// keeps the columns within reach^2 times it. out_starts null: each row's count into out and its
// closest distance into closest; else the strong columns in column order at out[out_starts[row]].
__global__ void strength_kernel(uint32_t rows, const uint32_t* __restrict__ starts, const uint32_t* __restrict__ cols,
                                const double* __restrict__ pos, double limit_scale, double* __restrict__ closest,
                                const uint32_t* __restrict__ out_starts, uint32_t* __restrict__ out) {
  for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < rows; row += gridDim.x * blockDim.x) {
    const double* p = pos + 3 * (size_t)row;
    const uint32_t a0 = starts[row], a1 = starts[row + 1];
    double c = 1.7976931348623157e308;
    for (uint32_t at = a0; at < a1; ++at) {
      const uint32_t col = cols[at];
      if (col == row) continue;
      const double* q = pos + 3 * (size_t)col;
      const double dx = q[0] - p[0], dy = q[1] - p[1], dz = q[2] - p[2];
      const double d = dx * dx + dy * dy + dz * dz;
      c = d < c ? d : c;  // std::min(c, d)
    }
    const double limit = limit_scale * c;
    uint32_t n = 0;
    for (uint32_t at = a0; at < a1; ++at) {
      const uint32_t col = cols[at];
      if (col == row) continue;
      const double* q = pos + 3 * (size_t)col;
      const double dx = q[0] - p[0], dy = q[1] - p[1], dz = q[2] - p[2];
      if (dx * dx + dy * dy + dz * dz <= limit) {
        if (out_starts) out[out_starts[row] + n] = col;
        ++n;
      }
    }
    if (!out_starts) {
      closest[row] = c;
      out[row] = n;
    }
  }
}

sf_status setup_strength(cudaStream_t st, uint32_t rows, const uint32_t* starts, const uint32_t* cols, const double* pos,
                         double limit_scale, double* closest, const uint32_t* out_starts, uint32_t* out) {
  if (rows == 0) return SF_OK;
  strength_kernel<<<grid_for(rows), kT, 0, st>>>(rows, starts, cols, pos, limit_scale, closest, out_starts, out);
  return cuda_check(cudaGetLastError(), "strength");
}

sf_status setup_entry_rows(cudaStream_t st, uint32_t rows, const uint32_t* starts, uint32_t* out) {
  if (rows == 0) return SF_OK;
  entry_rows_kernel<<<grid_for(rows), kT, 0, st>>>(rows, starts, out);
  return cuda_check(cudaGetLastError(), "entry rows");
}

sf_status setup_column_counts(cudaStream_t st, size_t entries, const uint32_t* cols, uint32_t* counts) {
  if (entries == 0) return SF_OK;
  column_counts_kernel<<<grid_for(entries), kT, 0, st>>>(entries, cols, counts);
  return cuda_check(cudaGetLastError(), "column counts");
}

sf_status setup_transpose_pattern(cudaStream_t st, size_t entries, const uint32_t* cols, const uint32_t* entry_row,
                                  uint32_t width, uint32_t longest, const uint32_t* t_starts, uint32_t* cursors,
                                  uint32_t* t_at, uint32_t* t_rows) {
  if (entries == 0) return SF_OK;
  transpose_fill_kernel<<<grid_for(entries), kT, 0, st>>>(entries, cols, cursors, t_at);
  transpose_sort_kernel<<<std::min<uint32_t>(width, 148 * 16), 128, longest * 4, st>>>(width, t_starts, entry_row, t_at,
                                                                                       t_rows);
  return cuda_check(cudaGetLastError(), "transpose pattern");
}

sf_status setup_rigid_modes(cudaStream_t st, uint32_t rows, const uint32_t* row_node, const double* nodes,
                            const double center[3], double scale, double* modes) {
  if (rows == 0) return SF_OK;
  rigid_modes_kernel<<<(rows + 255) / 256, 256, 0, st>>>(rows, row_node, nodes, center[0], center[1], center[2], scale,
                                                         modes);
  return cuda_check(cudaGetLastError(), "rigid modes");
}

sf_status setup_dense_inverse(cudaStream_t st, uint32_t rows, int rb, const uint32_t* starts, const uint32_t* cols,
                              const double* vals, size_t n, double* work, double* li, double* inverse,
                              unsigned long long* bad, double* pivot) {
  if (n == 0) return SF_OK;
  cudaMemsetAsync(work, 0, n * n * 8, st);
  cudaMemsetAsync(li, 0, n * n * 8, st);
  dense_from_blocks_kernel<<<(rows + 127) / 128, 128, 0, st>>>(rows, rb, rb, starts, cols, vals, n, work, li);
  for (size_t j0 = 0; j0 < n; j0 += kPanel) {
    const size_t j1 = std::min(n, j0 + kPanel), below = n - j1;
    const unsigned row_blocks = (unsigned)((below + kDenseThreads - 1) / kDenseThreads);
    const unsigned col_blocks = (unsigned)((j1 + kDenseThreads - 1) / kDenseThreads);
    dense_panel_kernel<<<row_blocks + col_blocks, kDenseThreads, 0, st>>>(n, j0, row_blocks, work, li, bad, pivot);
    if (below)
      dense_update_kernel<<<dim3((unsigned)((n + 31) / 32), (unsigned)((below + 31) / 32)), 256, 0, st>>>(n, j0, work, li,
                                                                                                        bad);
  }
  const unsigned tiles = (unsigned)((n + 31) / 32);
  gram_inverse_kernel<<<dim3(tiles, tiles), 256, 0, st>>>(n, li, inverse);
  return cuda_check(cudaGetLastError(), "dense inverse");
}

sf_status setup_tentative(cudaStream_t st, size_t aggregates, int rb, size_t max_members, const uint32_t* member_starts,
                          const uint32_t* members, const double* near_null, double* t, double* coarse) {
  if (aggregates == 0) return SF_OK;
  const size_t smem = max_members * (size_t)rb * 6 * sizeof(double);
  if (smem > kTentativeMaxSmem) return fail(SF_INVALID_ARGUMENT, "an aggregate too large for the tentative kernel");
  static std::atomic<uint64_t> opted{0};  // the opt-in above 48 KB, once per device
  int dev = 0;
  cudaGetDevice(&dev);
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (smem > 48 * 1024 && (!bit || !(opted.load() & bit))) {
    cudaFuncSetAttribute(tentative_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTentativeMaxSmem);
    opted.fetch_or(bit);
  }
  tentative_kernel<<<(unsigned)aggregates, 32, smem, st>>>((uint32_t)aggregates, rb, member_starts, members, near_null,
                                                           t, coarse);
  return cuda_check(cudaGetLastError(), "tentative");
}

sf_status setup_smooth(cudaStream_t st, int rb, size_t entries, const uint32_t* entry_row, const uint32_t* p_cols,
                       const uint32_t* a_starts, const uint32_t* a_cols, const double* a_vals, const uint32_t* n_starts,
                       const uint32_t* n_cols, const uint32_t* aggregate, const double* t_vals, const double* inv,
                       double omega, double* p_vals) {
  if (entries == 0) return SF_OK;
  if (rb == 3)
    smooth_kernel<3><<<grid_for(entries), kT, 0, st>>>(entries, entry_row, p_cols, a_starts, a_cols, a_vals, n_starts,
                                                       n_cols, aggregate, t_vals, inv, omega, p_vals);
  else
    smooth_kernel<6><<<grid_for(entries), kT, 0, st>>>(entries, entry_row, p_cols, a_starts, a_cols, a_vals, n_starts,
                                                       n_cols, aggregate, t_vals, inv, omega, p_vals);
  return cuda_check(cudaGetLastError(), "smooth");
}

sf_status setup_product(cudaStream_t st, int rb, size_t entries, const uint32_t* entry_row, const uint32_t* ap_cols,
                        const uint32_t* a_starts, const uint32_t* a_cols, const double* a_vals, const uint32_t* p_starts,
                        const uint32_t* p_cols, const double* p_vals, double* ap_vals) {
  if (entries == 0) return SF_OK;
  if (rb == 3)
    product_kernel<3><<<grid_for(entries), kT, 0, st>>>(entries, entry_row, ap_cols, a_starts, a_cols, a_vals,
                                                        p_starts, p_cols, p_vals, ap_vals);
  else
    product_kernel<6><<<grid_for(entries), kT, 0, st>>>(entries, entry_row, ap_cols, a_starts, a_cols, a_vals,
                                                        p_starts, p_cols, p_vals, ap_vals);
  return cuda_check(cudaGetLastError(), "product");
}

sf_status setup_galerkin(cudaStream_t st, int rb, size_t entries, const uint32_t* entry_row, const uint32_t* c_cols,
                         const uint32_t* pt_starts, const uint32_t* pt_rows, const uint32_t* pt_at, const double* p_vals,
                         const uint32_t* ap_starts, const uint32_t* ap_cols, const double* ap_vals, double* c_vals) {
  if (entries == 0) return SF_OK;
  // Six threads a block up to so many blocks, one beyond. 3-row fine blocks: 10,332 blocks 360 us with
  // six and 580 with one, 75,678 blocks 1,910 and 1,180, 307,995 blocks 1,330 and 850, 677,221 blocks
  // 16.4 and 9.3 ms (102,624 and 412,254 blocks of plates the same either way); six threads of 32,768
  // blocks are about what the device holds at once. 6-row fine blocks always: 11,095 blocks 810 us with
  // six and 1,490 with one, 71,122 blocks 220 and 317, and deeper levels have no more.
  constexpr size_t kSplit = 32768;
  auto launch = [&](auto kernel, size_t threads) {
    kernel<<<grid_for(threads), kT, 0, st>>>(entries, entry_row, c_cols, pt_starts, pt_rows, pt_at, p_vals, ap_starts,
                                             ap_cols, ap_vals, c_vals);
  };
  if (rb == 3)
    entries <= kSplit ? launch(galerkin_kernel<3, 1>, 6 * entries) : launch(galerkin_kernel<3, 6>, entries);
  else
    launch(galerkin_kernel<6, 1>, 6 * entries);
  return cuda_check(cudaGetLastError(), "galerkin");
}

template <typename S>
sf_status setup_convert(cudaStream_t st, size_t n, const double* in, S* out) {
  if (n == 0) return SF_OK;
  convert_kernel<S><<<grid_for(n), kT, 0, st>>>(n, in, out);
  return cuda_check(cudaGetLastError(), "convert");
}
template sf_status setup_convert<float>(cudaStream_t, size_t, const double*, float*);
template sf_status setup_convert<double>(cudaStream_t, size_t, const double*, double*);

template <typename S>
sf_status setup_transpose_blocks(cudaStream_t st, size_t blocks, int rb, int cb, const uint32_t* src, const double* in,
                                 S* out) {
  if (blocks == 0) return SF_OK;
  transpose_blocks_kernel<S><<<grid_for(blocks), kT, 0, st>>>(blocks, rb, cb, src, in, out);
  return cuda_check(cudaGetLastError(), "transpose blocks");
}
template sf_status setup_transpose_blocks<float>(cudaStream_t, size_t, int, int, const uint32_t*, const double*, float*);
template sf_status setup_transpose_blocks<double>(cudaStream_t, size_t, int, int, const uint32_t*, const double*, double*);

template <typename S>
sf_status setup_sell_fill(cudaStream_t st, size_t slots, int len, const uint32_t* sell_rows, const uint32_t* sell_len,
                          const uint32_t* sell_start, uint32_t nrows, const uint32_t* starts, const uint32_t* cols,
                          const double* in, uint32_t* out_cols, S* out) {
  if (slots == 0) return SF_OK;
  switch (len) {
    case 9:
      sell_fill_kernel<S, 9><<<grid_for(slots), kT, 0, st>>>(slots, sell_rows, sell_len, sell_start, nrows, starts, cols,
                                                            in, out_cols, out);
      break;
    case 18:
      sell_fill_kernel<S, 18><<<grid_for(slots), kT, 0, st>>>(slots, sell_rows, sell_len, sell_start, nrows, starts, cols,
                                                             in, out_cols, out);
      break;
    case 36:
      sell_fill_kernel<S, 36><<<grid_for(slots), kT, 0, st>>>(slots, sell_rows, sell_len, sell_start, nrows, starts, cols,
                                                             in, out_cols, out);
      break;
    default: return fail(SF_INVALID_ARGUMENT, "unsupported block size for the SELL layout");
  }
  return cuda_check(cudaGetLastError(), "SELL fill");
}
template <typename S>
sf_status setup_split_fill(cudaStream_t st, size_t slots, int cb, const uint32_t* sell_rows, const uint32_t* sell_len,
                           const uint32_t* sell_start, uint32_t nrows, const uint32_t* starts, const uint32_t* cols,
                           const double* in, uint32_t* out_cols, S* out) {
  if (slots == 0) return SF_OK;
  if (cb == 3)
    split_fill_kernel<S, 3><<<grid_for(slots), kT, 0, st>>>(slots, sell_rows, sell_len, sell_start, nrows, starts, cols,
                                                           in, out_cols, out);
  else if (cb == 6)
    split_fill_kernel<S, 6><<<grid_for(slots), kT, 0, st>>>(slots, sell_rows, sell_len, sell_start, nrows, starts, cols,
                                                           in, out_cols, out);
  else
    return fail(SF_INVALID_ARGUMENT, "unsupported block size for the split-row layout");
  return cuda_check(cudaGetLastError(), "split fill");
}
template sf_status setup_split_fill<float>(cudaStream_t, size_t, int, const uint32_t*, const uint32_t*, const uint32_t*,
                                           uint32_t, const uint32_t*, const uint32_t*, const double*, uint32_t*, float*);
template sf_status setup_split_fill<double>(cudaStream_t, size_t, int, const uint32_t*, const uint32_t*, const uint32_t*,
                                            uint32_t, const uint32_t*, const uint32_t*, const double*, uint32_t*, double*);

template sf_status setup_sell_fill<float>(cudaStream_t, size_t, int, const uint32_t*, const uint32_t*, const uint32_t*,
                                          uint32_t, const uint32_t*, const uint32_t*, const double*, uint32_t*, float*);
template sf_status setup_sell_fill<double>(cudaStream_t, size_t, int, const uint32_t*, const uint32_t*, const uint32_t*,
                                           uint32_t, const uint32_t*, const uint32_t*, const double*, uint32_t*, double*);

}  // namespace sf
