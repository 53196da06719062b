// The solver on the device: the conjugate gradient's iteration and its CUDA graph, device memory
// and pinned buffers, the operator layouts, batched iterations, kernel timing and the energy
// products. The kernels are in solve_kernels.cuh, the V-cycle's launch sequence in cycle.cuh.
#include "solve_kernels.cuh"

namespace sf {

thread_local std::vector<LaunchRecord>* g_recorder = nullptr;

namespace {

// z = M r for the solver's r (f64) into z (f64) or z32.
void enqueue_precondition(DeviceSolver& s, const double* r, double* z, float* z32, const int* status) {
  if (!s.multigrid) {
    launch_body<jacobi_kernel>(grid_for_elems(s.n), kThreads, 0, s.stream, s.n, s.jacobi, r, z, status);
    s.launches_per_iteration++;
    return;
  }
  if (!s.storage_single)
    Cycle<double, double>::precondition(s, r, z, status);
  else if (!s.vector_single)
    Cycle<float, double>::precondition(s, r, z, status);
  else
    Cycle<float, float>::precondition(s, r, z32, status);
}

template <int LPR>
void launch_pcg_spmv_lpr(DeviceSolver& s) {
  Op<double> A = op_of<double>(s.system);
  Shape sh = shape_of(A, true);
  // (outside a batch the grid is the block count)
  auto fixed = [&](LaunchRecord& r) {
    r.capacity = (unsigned)sh.capacity;
    r.fixed_blocks = true;
  };
  launch_body<pcg_spmv_dot_kernel<LPR>>(sh.grid, sh.threads, sh.smem, s.stream, (uint32_t)sh.grid, A, s.p, s.ap, s.partials, s.state);
  if (g_recorder) fixed(g_recorder->back());
  launch_body<pcg_update_kernel>(grid_for_reduction(s.n), kReduceThreads, 0, s.stream, s.n, s.p, s.ap, s.x, s.r, s.partials, s.state);
  launch_body<pcg_check_kernel<LPR>>(sh.grid, sh.threads, sh.smem, s.stream, (uint32_t)sh.grid, A, s.x, s.rhs, s.r,
                                     s.partials, s.state);
  if (g_recorder) fixed(g_recorder->back());
}

}  // namespace

sf_status cuda_check(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return SF_OK;
  char msg[200];
  std::snprintf(msg, sizeof(msg), "%s: %s", what, cudaGetErrorString(e));
  if (e == cudaErrorMemoryAllocation) return fail(SF_DEVICE_MEMORY_BUDGET, msg);
  return fail(SF_CUDA_ERROR, msg);
}

// Device memory comes from the device's stream-ordered pool: an allocation or a free is ordered on
// the solver's stream and never waits for the rest of the device (cudaFree would synchronize the
// whole device, stalling every other study in flight). The pool keeps freed memory for reuse
// instead of returning it at each synchronization.
void pool_setup(int device) {
  static std::mutex mu;
  static bool done[64] = {};
  std::lock_guard<std::mutex> lock(mu);
  if (device < 0 || device >= 64 || done[device]) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
    uint64_t keep = UINT64_MAX;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    // Reserve a first slab now (an eighth of the free memory, at most 8 GiB), once: growing the
    // pool later maps new memory inside a study's build, and such a call was measured blocking
    // the host for up to 0.8 s.
    size_t free_bytes = 0, total = 0;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    if (cudaMemGetInfo(&free_bytes, &total) == cudaSuccess) {
      const size_t slab = std::min<size_t>(free_bytes / 8, (size_t)8 << 30);
      cudaStream_t st = nullptr;
      void* p = nullptr;
      if (slab && cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess) {
        if (cudaMallocAsync(&p, slab, st) == cudaSuccess) cudaFreeAsync(p, st);
        cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
      }
      cudaGetLastError();
    }
    cudaSetDevice(prev);
  }
  done[device] = true;
}

sf_status dev_alloc(DeviceSolver& s, void** ptr, size_t bytes) {
  // 64 bytes of slack: the staged loads read whole 16-byte chunks past an array's last value.
  size_t padded = bytes + 64;
  pool_setup(s.device);
  cudaError_t e = cudaMallocAsync(ptr, padded, s.stream);
  if (e != cudaSuccess) return cuda_check(e, "cudaMallocAsync");
  cudaMemsetAsync(*ptr, 0, padded, s.stream);
  s.owned.push_back({*ptr, padded});
  s.bytes += padded;
  return SF_OK;
}

bool wants_sell(const DevBsr& m, uint64_t sell_min_rows) {
  // A warp stages two row groups at once; a group is at least one row, so an operator with rows
  // too long to stage (the transposes of wide prolongators) runs one thread per row instead.
  const size_t slot = ((m.group_bytes + 31) & ~15u) + ((m.group_blocks * 4 + 31) & ~15u) +
                      (((m.group_rows + 1) * 4 + 31) & ~15u);
  return m.rows >= sell_min_rows || 2 * slot > kMaxStagePerWarp;
}

bool wants_split(const DevBsr& m, bool uniform_lanes) {
  return !uniform_lanes && m.rb == 6 && (m.cb == 3 || m.cb == 6) && m.rows >= kSplitMinRows;
}

void dev_free(DeviceSolver& s, void* ptr) {
  if (!ptr) return;
  for (size_t i = 0; i < s.owned.size(); ++i)
    if (s.owned[i].first == ptr) {
      cudaFreeAsync(ptr, s.stream);
      s.bytes -= s.owned[i].second;
      s.owned[i] = s.owned.back();
      s.owned.pop_back();
      return;
    }
}

void dev_free_all(DeviceSolver& s) {
  if (s.graph_exec) cudaGraphExecDestroy(s.graph_exec);
  if (s.graph) cudaGraphDestroy(s.graph);
  if (s.run_exec) cudaGraphExecDestroy(s.run_exec);
  if (s.run_graph) cudaGraphDestroy(s.run_graph);
  s.graph_exec = s.run_exec = nullptr;
  s.graph = s.run_graph = nullptr;
  for (auto& p : s.owned) cudaFreeAsync(p.first, s.stream);
  s.owned.clear();
  s.bytes = 0;
}

sf_status make_row_groups(DeviceSolver& s, DevBsr& m, const uint32_t* starts, size_t value_bytes, bool one_pass) {
  // Rows per group: as many mean rows as fit kGroupTarget bytes (1 to 8, a power of two). The
  // warp splits into that many teams of 32 / teams lanes, one row each, so a warp works on several
  // light rows at once (their x gathers and epilogue loads overlap) and on a heavy row whole.
  double mean = m.rows ? (double)starts[m.rows] / m.rows : 0.0;
  // Batchable studies take a nominal row length per block shape (about 25 blocks on a 3x3
  // stiffness level, 4 on a prolongator, 30 on a coarse level or a transpose), so the choice, and
  // with it the kernel, is the same for every study of that shape.
  if (s.uniform_lanes) mean = (m.rb == 3 && m.cb == 3) ? 25.0 : (m.cb == 6 && m.rb == 3) ? 4.0 : 30.0;
  double row_bytes = std::max(1.0, mean * (double)value_bytes);
  int teams = 1;
  while (teams < 8 && (teams * 2) * row_bytes <= kGroupTarget) teams *= 2;
  m.lanes_per_row = 32 / teams;
  size_t target = std::min<size_t>(kGroupTarget, (size_t)(teams * row_bytes * 1.15));
  std::vector<uint4> g;
  g.reserve(m.rows / 2 + 2);
  uint32_t max_bytes = 0, max_blocks = 0, max_rows = 0;
  uint32_t r = 0;
  while (r < m.rows) {
    uint32_t e = r + 1;
    size_t bytes = (size_t)(starts[e] - starts[r]) * value_bytes;
    while (e < m.rows && (!one_pass || e - r < (uint32_t)teams) && bytes + (size_t)(starts[e + 1] - starts[e]) * value_bytes <= target) {
      bytes += (size_t)(starts[e + 1] - starts[e]) * value_bytes;
      ++e;
    }
    max_bytes = std::max<uint32_t>(max_bytes, (uint32_t)bytes);
    max_blocks = std::max<uint32_t>(max_blocks, starts[e] - starts[r]);
    max_rows = std::max<uint32_t>(max_rows, e - r);
    g.push_back(make_uint4(r, e, starts[r], starts[e]));
    r = e;
  }
  m.ngroups = (uint32_t)g.size();
  m.group_bytes = max_bytes;
  m.group_blocks = max_blocks;
  m.group_rows = max_rows;
  m.longest_row = 0;
  for (uint32_t i = 0; i < m.rows; ++i) m.longest_row = std::max(m.longest_row, starts[i + 1] - starts[i]);
  if (sf_status e = dev_alloc(s, (void**)&m.groups, std::max<size_t>(1, g.size()) * sizeof(uint4))) return e;
  if (!g.empty()) copy_h2d(s, m.groups, g.data(), g.size() * sizeof(uint4));
  return cuda_check(cudaStreamSynchronize(s.stream), "row groups");
}

namespace {

struct SellLayout {
  uint32_t nslices = 0;
  std::vector<uint32_t> rows, len, start;
};

// Rows by descending block count inside windows of kSellWindow rows, equal lengths in row order:
// a counting sort per window (the order a stable sort by descending length gives).
std::vector<uint32_t> window_order(uint32_t nrows, const uint32_t* starts) {
  std::vector<uint32_t> order(nrows), count;
  for (uint32_t w0 = 0; w0 < nrows; w0 += kSellWindow) {
    const uint32_t w1 = std::min(nrows, w0 + kSellWindow);
    uint32_t longest = 0;
    for (uint32_t r = w0; r < w1; ++r) longest = std::max(longest, starts[r + 1] - starts[r]);
    count.assign(longest + 2, 0);
    for (uint32_t r = w0; r < w1; ++r) count[longest - (starts[r + 1] - starts[r]) + 1] += 1;
    for (uint32_t k = 1; k <= longest + 1; ++k) count[k] += count[k - 1];
    for (uint32_t r = w0; r < w1; ++r) order[w0 + count[longest - (starts[r + 1] - starts[r])]++] = r;
  }
  return order;
}

// Rows sorted by descending block count inside windows of kSellWindow rows (stable, so equal
// lengths keep row order), cut into slices of 32, slice widths padded to chunks of `chunk`
// blocks. Only this row order is host work; the blocks are placed on the device.
SellLayout sell_layout(uint32_t nrows, const uint32_t* starts, uint32_t chunk) {
  SellLayout L;
  L.nslices = (nrows + 31) / 32;
  std::vector<uint32_t> order = window_order(nrows, starts);
  auto rlen = [&](uint32_t r) { return starts[r + 1] - starts[r]; };
  L.rows.assign((size_t)L.nslices * 32, nrows);
  L.len.assign((size_t)L.nslices * 32, 0);
  L.start.assign(L.nslices + 1, 0);
  for (uint32_t i = 0; i < nrows; ++i) {
    L.rows[i] = order[i];
    L.len[i] = rlen(order[i]);
  }
  for (uint32_t sl = 0; sl < L.nslices; ++sl) {
    uint32_t width = 0;
    for (uint32_t t = 0; t < 32; ++t) width = std::max(width, L.len[sl * 32 + t]);
    width = (width + chunk - 1) / chunk * chunk;
    L.start[sl + 1] = L.start[sl] + 32 * width;
  }
  return L;
}

// Block rows ordered as sell_layout orders rows, kSplitRowsPerSlice to a slice, six lanes each
// (lane 6 m + p: scalar row p of the slice's block row m; lanes 30 and 31 idle), slice widths
// padded to chunks of `chunk` blocks.
SellLayout split_layout(uint32_t nrows, const uint32_t* starts, uint32_t chunk) {
  SellLayout L;
  L.nslices = (nrows + kSplitRowsPerSlice - 1) / kSplitRowsPerSlice;
  std::vector<uint32_t> order = window_order(nrows, starts);
  auto rlen = [&](uint32_t r) { return starts[r + 1] - starts[r]; };
  L.rows.assign((size_t)L.nslices * 32, nrows);
  L.len.assign((size_t)L.nslices * 32, 0);
  L.start.assign(L.nslices + 1, 0);
  for (uint32_t i = 0; i < nrows; ++i) {
    const size_t sl = i / kSplitRowsPerSlice, m = i % kSplitRowsPerSlice;
    for (uint32_t p = 0; p < 6; ++p) {
      L.rows[sl * 32 + 6 * m + p] = order[i];
      L.len[sl * 32 + 6 * m + p] = rlen(order[i]);
    }
  }
  for (uint32_t sl = 0; sl < L.nslices; ++sl) {
    uint32_t width = 0;
    for (uint32_t t = 0; t < 32; ++t) width = std::max(width, L.len[sl * 32 + t]);
    width = (width + chunk - 1) / chunk * chunk;
    L.start[sl + 1] = L.start[sl] + 32 * width;
  }
  return L;
}

sf_status upload_sell_layout(DeviceSolver& s, DevBsr& m, const SellLayout& L, size_t value_bytes, bool split) {
  m.nslices = L.nslices;
  sf_status e = SF_OK;
  if (!e) e = dev_alloc(s, (void**)&m.sell_rows, L.rows.size() * 4);
  if (!e) e = dev_alloc(s, (void**)&m.sell_len, L.len.size() * 4);
  if (!e) e = dev_alloc(s, (void**)&m.sell_start, L.start.size() * 4);
  const size_t slots = L.start[L.nslices];
  const size_t col_slots = split ? slots / 32 * kSplitRowsPerSlice : slots;
  if (!e) e = dev_alloc(s, (void**)&m.sell_cols, std::max<size_t>(1, col_slots) * 4);
  if (!e) e = dev_alloc(s, &m.sell_vals, std::max<size_t>(1, slots) * value_bytes);
  if (e) return e;
  copy_h2d(s, m.sell_rows, L.rows.data(), L.rows.size() * 4);
  copy_h2d(s, m.sell_len, L.len.data(), L.len.size() * 4);
  copy_h2d(s, m.sell_start, L.start.data(), L.start.size() * 4);
  return SF_OK;
}

}  // namespace

// The SELL copy of a matrix from its f64 values on the device, converted to S.
template <typename S>
sf_status make_sell_converted(DeviceSolver& s, DevBsr& m, const uint32_t* starts, const double* vals) {
  const int len = (int)(m.rb * m.cb);
  SellLayout L = sell_layout(m.rows, starts, (uint32_t)sell_chunk_blocks(len, (int)sizeof(S)));
  if (sf_status e = upload_sell_layout(s, m, L, (size_t)len * sizeof(S), false)) return e;
  sf_status e = setup_sell_fill<S>(s.stream, (size_t)L.nslices * 32, len, m.sell_rows, m.sell_len, m.sell_start, m.rows,
                                   m.starts, m.cols, vals, m.sell_cols, (S*)m.sell_vals);
  if (!e) e = cuda_check(cudaStreamSynchronize(s.stream), "SELL placement");
  m.sell = true;
  return e;
}

// The split-row copy of a 6 x cb matrix from its f64 values on the device, converted to S.
template <typename S>
sf_status make_split_converted(DeviceSolver& s, DevBsr& m, const uint32_t* starts, const double* vals) {
  SellLayout L = split_layout(m.rows, starts, (uint32_t)sell_chunk_blocks((int)m.cb, (int)sizeof(S)));
  if (sf_status e = upload_sell_layout(s, m, L, (size_t)m.cb * sizeof(S), true)) return e;
  sf_status e = setup_split_fill<S>(s.stream, (size_t)L.nslices * 32, (int)m.cb, m.sell_rows, m.sell_len, m.sell_start,
                                    m.rows, m.starts, m.cols, vals, m.sell_cols, (S*)m.sell_vals);
  if (!e) e = cuda_check(cudaStreamSynchronize(s.stream), "split-row placement");
  m.split = true;
  return e;
}

sf_status make_sell_from_device(DeviceSolver& s, DevBsr& m, const uint32_t* starts) {
  return make_sell_converted<double>(s, m, starts, (const double*)m.vals);
}

namespace {

// A level operator on the device from the setup's f64 values: the setup's device pattern, the
// values converted to S (or the f64 values themselves when S is double and `alias` holds), row
// groups, and a SELL copy when the operator has many rows.
template <typename S>
sf_status device_bsr(DeviceSolver& s, const Bsr& h, DevBsr& d, bool alias) {
  d.rows = (uint32_t)h.rows;
  d.rb = (uint32_t)h.rb;
  d.cb = (uint32_t)h.cb;
  d.blocks = h.starts.back();
  d.starts = h.dev_starts;
  d.cols = h.dev_cols;
  const size_t n = d.blocks * h.rb * h.cb;
  if (alias && sizeof(S) == 8) {
    d.vals = h.dev;
  } else {
    if (sf_status e = dev_alloc(s, &d.vals, std::max<size_t>(1, n) * sizeof(S))) return e;
    if (sf_status e = setup_convert<S>(s.stream, n, h.dev, (S*)d.vals)) return e;
  }
  // A level's products keep a group to the rows a warp takes in one pass: five or six short rows to
  // a group of four teams cost two passes, the second mostly idle. (The f64 system's groups also
  // order its dot products' sums, so they stay as they are.)
  if (sf_status e = make_row_groups(s, d, h.starts.data(), h.rb * h.cb * sizeof(S), true)) return e;
  if (wants_split(d, s.uniform_lanes)) {
    if (sf_status e = make_split_converted<S>(s, d, h.starts.data(), h.dev)) return e;
  } else if (wants_sell(d, s.sell_min_rows)) {
    if (sf_status e = make_sell_converted<S>(s, d, h.starts.data(), h.dev)) return e;
  }
  return cuda_check(cudaGetLastError(), "level operator");
}

template <typename S>
sf_status upload_level(DeviceSolver& s, const std::vector<HostLevel>& levels, size_t li, DevLevel& L) {
  const HostLevel& h = levels[li];
  const bool alias = true;
  if (li == 0 && sizeof(S) == 8) {
    L.a = s.system;  // the f64 system matrix is the finest operator
  } else if (sf_status e = device_bsr<S>(s, h.a, L.a, alias)) {
    return e;
  }
  const size_t nd = h.a.rows * h.a.rb * h.a.rb;
  if (sizeof(S) == 8) {
    L.dinv = h.inverse_diagonal;
  } else {
    if (sf_status e = dev_alloc(s, &L.dinv, nd * sizeof(S))) return e;
    if (sf_status e = setup_convert<S>(s.stream, nd, h.inverse_diagonal, (S*)L.dinv)) return e;
  }
  L.has_p = h.has_p;
  if (h.has_p) {
    if (sf_status e = device_bsr<S>(s, h.p, L.p, alias)) return e;
    // The explicit transpose (the reference's GPU layout stores the same one for gather restriction,
    // gpu/layout.rs:254-291), its pattern as the Galerkin product made it.
    Bsr t;
    t.rows = levels[li + 1].a.rows;
    t.rb = h.p.cb;
    t.cb = h.p.rb;
    t.starts = h.t_starts;
    t.dev_starts = h.dev_t_starts;
    t.dev_cols = h.dev_t_rows;
    const size_t blocks = t.starts.back();
    sf_status e = dev_alloc(s, (void**)&t.dev, std::max<size_t>(1, blocks) * t.rb * t.cb * 8);
    if (e) return e;
    e = setup_transpose_blocks<double>(s.stream, blocks, (int)h.p.rb, (int)h.p.cb, h.dev_t_at, h.p.dev, t.dev);
    if (!e) e = device_bsr<S>(s, t, L.r, alias);
    if (!e) e = cuda_check(cudaStreamSynchronize(s.stream), "transpose");
    dev_free(s, h.dev_t_at);
    if (sizeof(S) != 8) dev_free(s, t.dev);  // the converted copy is the one kept
    if (e) return e;
  }
  return SF_OK;
}

}  // namespace

sf_status solver_upload_hierarchy(DeviceSolver& s, const std::vector<HostLevel>& levels, uint64_t degree) {
  size_t V = s.vector_single ? 4 : 8;
  s.levels.assign(levels.size(), DevLevel());
  for (size_t li = 0; li < levels.size(); ++li) {
    const HostLevel& h = levels[li];
    DevLevel& L = s.levels[li];
    L.n = (uint32_t)(h.a.rows * h.a.rb);
    sf_status e = s.storage_single ? upload_level<float>(s, levels, li, L) : upload_level<double>(s, levels, li, L);
    if (e) return e;
    L.has_factor = h.has_factor;
    if (h.has_factor) {
      L.coarse_inverse = h.dev_coarse_inverse;  // made on the device by the setup, owned by this solver
    }
    // ChebyshevCoefficients (gpu/layout.rs:443-465), the recurrence of cycle.rs:578-626.
    double theta = 0.5 * (h.lambda_max + h.lambda_min);
    double delta = 0.5 * (h.lambda_max - h.lambda_min);
    double sigma = theta / delta;
    double rho = 1.0 / sigma;
    L.theta = theta;
    L.steps.clear();
    for (uint64_t k = 1; k < degree; ++k) {
      double next = 1.0 / (2.0 * sigma - rho);
      L.steps.push_back({next * rho, 2.0 * next / delta});
      rho = next;
    }
    void** vecs[] = {&L.b, &L.x, &L.res, &L.d0, &L.d1, &L.post_x, &L.tmp};
    for (void** v : vecs)
      if (sf_status e = dev_alloc(s, v, (size_t)L.n * V)) return e;
  }
  if (s.vector_single)
    if (sf_status e = dev_alloc(s, (void**)&s.z32, (size_t)s.n * 4)) return e;
  // The coarse tail: the last smoothed level (6-row blocks) and the factored coarsest level,
  // small enough that one cluster beats a launch per phase. Batchable studies keep per-phase
  // launches (their kernel sequence must not depend on sizes).
  s.tail_level = -1;
  s.tail_cluster = 0;
  s.tail_smem = 0;
  if (s.coarse_tail && !s.uniform_lanes && s.levels.size() >= 3) {
    const size_t li = s.levels.size() - 2;
    const DevLevel& L = s.levels[li];
    const DevLevel& C = s.levels[li + 1];
    if (L.has_p && C.has_factor && L.a.rb == 6 && L.a.cb == 6 && L.p.rb == 6 && L.p.cb == 6 && L.r.rb == 6 &&
        L.r.cb == 6 && L.a.rows <= kTailMaxRows && C.n <= kTailMaxCoarse && L.steps.size() <= (size_t)kTailMaxSteps) {
      size_t smem = 0;
      const HostLevel &hs = levels[li], &hc = levels[li + 1];
      unsigned c = !s.storage_single ? Cycle<double, double>::tail_cluster(hs, hc, &smem)
                   : !s.vector_single ? Cycle<float, double>::tail_cluster(hs, hc, &smem)
                                      : Cycle<float, float>::tail_cluster(hs, hc, &smem);
      if (c) {
        s.tail_level = (int)li;
        s.tail_cluster = c;
        s.tail_smem = smem;
      }
    }
  }
  return cuda_check(cudaStreamSynchronize(s.stream), "hierarchy upload");
}

sf_status solver_init_pcg(DeviceSolver& s, double tolerance, uint64_t max_iterations) {
  PcgState h;
  std::memset(&h, 0, sizeof(h));
  h.tolerance = tolerance;
  h.max_iterations = max_iterations ? max_iterations : 10ull * s.n + 1000ull;
  h.flexible = s.flexible ? 1 : 0;
  h.status = ST_ACTIVE;
  copy_h2d(s, s.state, &h, sizeof(h));
  int one_active = ST_ACTIVE;
  copy_h2d(s, s.always_active, &one_active, sizeof(int));
  launch_body<pcg_init_kernel>(grid_for_reduction(s.n), kReduceThreads, 0, s.stream, s.n, s.rhs, s.x, s.r, s.partials, s.state);
  return solver_enqueue_reset(s);
}

sf_status solver_enqueue_reset(DeviceSolver& s) {
  const int grid = grid_for_reduction(s.n), wide = grid_for_elems(s.n);
  if (!s.multigrid) {
    // Jacobi: z = r / diag is formed where it is read, in both kernels.
    launch_body<jacobi_dot_rz_kernel>(grid, kReduceThreads, 0, s.stream, s.n, s.r, s.jacobi, s.ap, s.partials, s.state);
    launch_body<jacobi_update_p_kernel>(wide, kThreads, 0, s.stream, s.n, s.r, s.jacobi, s.p, s.state);
  } else {
    enqueue_precondition(s, s.r, s.z, s.z32, &s.state->status);
    if (s.vector_single) {
      launch_body<pcg_dot_rz_kernel<float>>(grid, kReduceThreads, 0, s.stream, s.n, s.r, s.z32, s.ap, s.partials, s.state);
      launch_body<pcg_update_p_kernel<float>>(wide, kThreads, 0, s.stream, s.n, s.z32, s.p, s.state);
    } else {
      launch_body<pcg_dot_rz_kernel<double>>(grid, kReduceThreads, 0, s.stream, s.n, s.r, s.z, s.ap, s.partials, s.state);
      launch_body<pcg_update_p_kernel<double>>(wide, kThreads, 0, s.stream, s.n, s.z, s.p, s.state);
    }
  }
  s.launches_per_iteration += 2;
  return cuda_check(cudaGetLastError(), "reset direction");
}

sf_status solver_enqueue_iteration(DeviceSolver& s) {
  cudaStream_t st = s.stream;
  s.launches_per_iteration = 0;
  if (s.system.sell) {
    SellOp<double> A = sell_of<double>(s.system);
    int grid = std::min(grid_for_slices(s.system.nslices), kReduceBlocks * 2);
    launch_body<sell_pcg_spmv_dot_kernel>(grid, kThreads, 0, st, A, s.p, s.ap, s.partials, s.state);
    launch_body<pcg_update_kernel>(grid_for_reduction(s.n), kReduceThreads, 0, st, s.n, s.p, s.ap, s.x, s.r, s.partials, s.state);
    launch_body<sell_pcg_check_kernel>(grid, kThreads, 0, st, A, s.x, s.rhs, s.r, s.partials, s.state);
  } else switch (product_lanes(s.system)) {
    case 8: launch_pcg_spmv_lpr<8>(s); break;
    case 16: launch_pcg_spmv_lpr<16>(s); break;
    default: launch_pcg_spmv_lpr<32>(s); break;
  }
  s.launches_per_iteration += 3;
  return solver_enqueue_reset(s);
}

// ------------------------------------------------------------ batched iterations
// Records one conjugate gradient iteration of every instance, checks that they launch the same
// kernels in the same order with the same block shapes, and captures one graph whose every node
// is a single grid over all instances: grid.x is the largest instance's, grid.y the instance
// count, and each launch site's argument packs sit in one device table (the per-instance offset
// table: each pack holds that instance's operator, vectors, scalars and status word).
sf_status batch_build(const std::vector<DeviceSolver*>& inst, cudaStream_t stream, BatchIteration& out) {
  out = BatchIteration();
  out.stream = stream;
  out.count = inst.size();
  if (inst.empty()) return fail(SF_INVALID_ARGUMENT, "an empty batch");
  std::vector<std::vector<LaunchRecord>> rec(inst.size());
  for (size_t i = 0; i < inst.size(); ++i) {
    g_recorder = &rec[i];
    sf_status e = solver_enqueue_iteration(*inst[i]);
    g_recorder = nullptr;
    if (e) return e;
  }
  const size_t sites = rec[0].size();
  for (size_t i = 1; i < inst.size(); ++i) {
    const char* why = nullptr;
    size_t at = 0;
    if (rec[i].size() != sites) why = "a different number of kernels per iteration";
    for (size_t j = 0; !why && j < sites; ++j) {
      at = j;
      if (rec[i][j].batched != rec[0][j].batched) why = "a different kernel";
      else if (rec[i][j].pack.size() != rec[0][j].pack.size()) why = "different arguments";
      else if (rec[i][j].cluster != rec[0][j].cluster) why = "a different cluster size";
    }
    if (why) {
      char msg[200];
      std::snprintf(msg, sizeof msg, "the studies of a batch must share their launch structure: study %zu has %s (launch %zu)",
                    i, why, at);
      return fail(SF_INVALID_ARGUMENT, msg);
    }
  }
  struct Site {
    const void* kernel;
    dim3 grid, block;
    size_t smem;
    void* table;
    unsigned cluster;
  };
  std::vector<Site> list(sites);
  for (size_t j = 0; j < sites; ++j) {
    Site& t = list[j];
    t.kernel = rec[0][j].batched;
    t.block = rec[0][j].block;
    t.grid = dim3(1, (unsigned)inst.size(), 1);
    t.smem = 0;
    t.cluster = rec[0][j].cluster;
    const size_t bytes = rec[0][j].pack.size();
    std::vector<unsigned char> host(bytes * inst.size());
    // Block sizes may differ (a row-group kernel's warps per block follow its largest group); the
    // bodies work with any block size and place each warp's staging slot by their own operator,
    // so the batch takes the largest block and the largest per-warp slot.
    size_t per_warp = 0, blocks = 0;
    unsigned capacity = ~0u;
    for (size_t i = 0; i < inst.size(); ++i) {
      blocks += rec[i][j].grid.x;
      capacity = std::min(capacity, rec[i][j].capacity);
      t.grid.x = std::max(t.grid.x, rec[i][j].grid.x);
      t.block.x = std::max(t.block.x, rec[i][j].block.x);
      per_warp = std::max(per_warp, rec[i][j].smem / std::max(1u, rec[i][j].block.x / 32));
      if (t.cluster) t.smem = std::max(t.smem, rec[i][j].smem);
      std::memcpy(host.data() + i * bytes, rec[i][j].pack.data(), bytes);
    }
    if (t.cluster) {
      // a cluster kernel keeps its block (launch bounds) and the largest instance's shared memory
    } else if (per_warp > 0) {
      // Fewer warps per block when the largest slot would not fit 200 KB of shared memory.
      size_t warps = std::max<size_t>(1, std::min<size_t>(t.block.x / 32, (200 * 1024) / per_warp));
      t.block.x = (unsigned)(32 * warps);
    }
    if (!t.cluster) t.smem = per_warp * (t.block.x / 32);
    // A row-group walk of more blocks than the device holds takes what it holds, shared among the
    // instances: a warp then walks several groups, each staged while the one before is multiplied,
    // instead of one group a warp whose staging nothing hides (16 cantilevers of 9,720 to 11,178
    // unknowns: 305 -> 270 us an iteration, the groups' single pass included).
    // The bodies with sums run the blocks these are formed for (the largest instance's, as before) in
    // turn, so their bits stay.
    if (rec[0][j].fixed_blocks) {
      const uint32_t count = t.grid.x;
      for (size_t i = 0; i < inst.size(); ++i) std::memcpy(host.data() + i * bytes, &count, sizeof(count));
    }
    if (capacity && blocks > capacity)
      t.grid.x = std::min<unsigned>(t.grid.x, (capacity + (unsigned)inst.size() - 1) / (unsigned)inst.size());
    if (t.smem > 200 * 1024) {
      batch_destroy(out);
      return fail(SF_INVALID_ARGUMENT, "a study of the batch needs more shared memory per warp than one SM holds");
    }
    pool_setup(inst[0]->device);
    cudaError_t e = cudaMallocAsync(&t.table, std::max<size_t>(host.size(), 16), stream);
    if (e != cudaSuccess) {
      batch_destroy(out);
      return cuda_check(e, "batch table");
    }
    out.tables.push_back(t.table);
    e = cudaMemcpyAsync(t.table, host.data(), host.size(), cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess && t.smem > 48 * 1024)
      e = cudaFuncSetAttribute(t.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) {
      batch_destroy(out);
      return cuda_check(e, "batch table");
    }
  }
  out.sites = sites;
  cudaError_t e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    batch_destroy(out);
    return cuda_check(e, "begin batch capture");
  }
  cudaError_t launch = cudaSuccess;
  for (Site& t : list) {
    cudaLaunchAttribute attr[1];
    if (t.cluster) {
      // one cluster per instance: grid.x is the cluster, blockIdx.y the instance
      t.grid.x = t.cluster;
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = t.cluster;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
    } else {
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[0].val.programmaticStreamSerializationAllowed = 1;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = t.grid;
    cfg.blockDim = t.block;
    cfg.dynamicSmemBytes = t.smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* argv[1] = {&t.table};
    cudaError_t le = cudaLaunchKernelExC(&cfg, t.kernel, argv);
    if (le != cudaSuccess && launch == cudaSuccess) launch = le;
  }
  e = cudaStreamEndCapture(stream, &out.graph);
  if (launch != cudaSuccess || e != cudaSuccess) {
    batch_destroy(out);
    return cuda_check(launch != cudaSuccess ? launch : e, "batch capture");
  }
  e = cudaGraphInstantiate(&out.exec, out.graph, 0);
  if (e != cudaSuccess) {
    batch_destroy(out);
    return cuda_check(e, "batch instantiate");
  }
  return SF_OK;
}

sf_status batch_replay(BatchIteration& b, uint64_t iterations) {
  for (uint64_t i = 0; i < iterations; ++i) {
    cudaError_t e = cudaGraphLaunch(b.exec, b.stream);
    if (e != cudaSuccess) return cuda_check(e, "batch replay");
  }
  return SF_OK;
}

void batch_destroy(BatchIteration& b) {
  if (b.exec) cudaGraphExecDestroy(b.exec);
  if (b.graph) cudaGraphDestroy(b.graph);
  for (void* t : b.tables) cudaFreeAsync(t, b.stream);
  b.exec = nullptr;
  b.graph = nullptr;
  b.tables.clear();
}

sf_status solver_restart(DeviceSolver& s, double tolerance, uint64_t max_iterations) {
  s.launches_per_iteration = 0;
  sf_status e = solver_init_pcg(s, tolerance, max_iterations);
  s.launches += s.launches_per_iteration + 1;
  return e;
}

sf_status solver_time_kernel(DeviceSolver& s, int kernel, uint64_t repeats, double* ms, double* bytes) {
  if (repeats == 0) return fail(SF_INVALID_ARGUMENT, "repeats must be positive");
  if (kernel == SF_KERNEL_SYSTEM_PRODUCT) {
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaEventRecord(a, s.stream);
    for (uint64_t i = 0; i < repeats; ++i)
      launch_bsr<double, double, 3, 3, OP_SET>(s.system, s.p, s.ap, nullptr, s.always_active, s.stream);
    cudaEventRecord(b, s.stream);
    cudaError_t e = cudaEventSynchronize(b);
    float t = 0;
    cudaEventElapsedTime(&t, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    *ms = t / (double)repeats;
    *bytes = (double)s.system.rows * 4 + (double)s.system.blocks * 76 + (double)s.n * 16;
    s.launches += repeats;
    return cuda_check(e, "time kernel");
  }
  if (!s.multigrid || s.levels.empty()) return fail(SF_INVALID_ARGUMENT, "the study has no multigrid hierarchy");
  if (kernel == SF_KERNEL_RESTRICTION && !s.levels[0].has_p) return fail(SF_INVALID_ARGUMENT, "one-level hierarchy");
  if (kernel < 0 || kernel > SF_KERNEL_RESTRICTION) return fail(SF_INVALID_ARGUMENT, "unknown kernel");
  if (!s.storage_single) return Cycle<double, double>::time_kernel(s, kernel, repeats, ms, bytes);
  if (!s.vector_single) return Cycle<float, double>::time_kernel(s, kernel, repeats, ms, bytes);
  return Cycle<float, float>::time_kernel(s, kernel, repeats, ms, bytes);
}

sf_status solver_level_stage(DeviceSolver& s, size_t level, int stage, const double* in0, const double* in1,
                             double* out0, double* out1) {
  if (!s.multigrid || level >= s.levels.size()) return fail(SF_INVALID_ARGUMENT, "no such multigrid level");
  if (!s.storage_single) return Cycle<double, double>::stage(s, level, stage, in0, in1, out0, out1);
  if (!s.vector_single) return Cycle<float, double>::stage(s, level, stage, in0, in1, out0, out1);
  return Cycle<float, float>::stage(s, level, stage, in0, in1, out0, out1);
}

sf_status solver_precondition(DeviceSolver& s, const double* d_in, double* d_out) {
  enqueue_precondition(s, d_in, d_out, s.z32, s.always_active);
  if (s.vector_single && s.multigrid)
    launch_body<convert_kernel<float, double>>(grid_for_elems(s.n), kThreads, 0, s.stream, s.n, s.z32, d_out, s.always_active);
  return cuda_check(cudaStreamSynchronize(s.stream), "precondition");
}

sf_status solver_system_multiply(DeviceSolver& s, const double* d_in, double* d_out) {
  launch_bsr<double, double, 3, 3, OP_SET>(s.system, d_in, d_out, nullptr, s.always_active, s.stream);
  return cuda_check(cudaStreamSynchronize(s.stream), "system multiply");
}

sf_status solver_read_state(DeviceSolver& s, PcgState* out) {
  copy_d2h(s, out, s.state, sizeof(PcgState));
  return cuda_check(cudaStreamSynchronize(s.stream), "read state");
}

// ------------------------------------------------------------ energy products, allocating nothing
// A variant of the conjugate gradient's system product (pcg_spmv_dot_kernel and
// sell_pcg_spmv_dot_kernel): for each of `count` vectors x_k of caller-owned device memory it
// writes y_k = A x_k and the energy e_k = x_k . y_k. Rows are summed exactly as the system product
// sums them; up to four vectors go through one walk of the operator, five to eight through two. The
// reduction's scratch is not the solver's: it is the file-scope array below, whose address is looked
// up once per device, so a call allocates no memory at all.
//
// Scratch layout (g_energy_scratch, 262,400 bytes per device):
//   bytes [0, 256):   arrival tickets (unsigned): the first for a call on a SELL system, one per walk
//                     on a row-group system. Each ticket must be zero when a launch starts. Static
//                     device storage is zero when the module loads, and the last block to take a
//                     ticket puts it back to zero before it exits, so the tickets are zero again
//                     after every completed call.
//   bytes [256, ...): kEnergyMaxBlocks slots of partial sums per vector. No initial value is needed:
//                     every block writes its slots before it takes its ticket.
// One array serves every study on a device, so two calls whose kernels can run at the same time
// (different streams, different studies, different host threads) race on it.
constexpr int kEnergyMaxVectors = 8;
constexpr int kEnergyMaxBlocks = 4096;  // blocks per vector of one launch
constexpr int kEnergyOneBlocks = 1024;  // of a launch for one vector, whose sums the others repeat
constexpr size_t kEnergyTicketBytes = 256;
constexpr size_t kEnergyScratchBytes = kEnergyTicketBytes + (size_t)kEnergyMaxVectors * kEnergyMaxBlocks * sizeof(double);
constexpr int kEnergyMaxDevices = 64;
static_assert(kEnergyMaxVectors * sizeof(unsigned) <= kEnergyTicketBytes, "tickets fit their header");

static __device__ __align__(256) unsigned char g_energy_scratch[kEnergyScratchBytes];

namespace {

__device__ __forceinline__ void energy_finish(double local, unsigned char* scratch, double* energy) {
  unsigned* ticket = reinterpret_cast<unsigned*>(scratch);
  double* partials = reinterpret_cast<double*>(scratch + kEnergyTicketBytes);
  double v[1] = {local}, total[1];
  if (finish_partials<1>(v, partials, ticket, total) && threadIdx.x == 0) energy[0] = total[0];
}

// SELL-32 system, one vector: one thread per row, rows summed as sell_kernel sums them. Bound by
// the operator's stream: 78 us a call on the gate plate where the walk below takes 83 us with one
// vector (its blocks finish their energies by themselves, 1,571 partials instead of 786).
__global__ void __launch_bounds__(kThreads) sell_energy_one_kernel(SellOp<double> A, const double* __restrict__ x,
                                                                   double* __restrict__ y,
                                                                   double* __restrict__ energy, unsigned char* scratch) {
  SellDot epi;
  epi.p = x;
  epi.ap = y;
  epi.local = 0.0;
  sell_rows<double, double, 3, 3, false>(A, x, epi, OpenGate{});
  energy_finish(epi.local, scratch, energy);
}

// SELL-32 system, several vectors: one thread per row and K vectors at once, each row of each vector summed as
// sell_kernel sums it, so the operator's stream (76 bytes a block) is read from memory once for
// all the vectors. A block is W slices by G groups of K vectors, a warp each: the G warps of a
// slice read its stream from L1. The x gathers bound it (3 K loads a block of about 25 sectors,
// L2 latency), so more than four vectors run as two groups of half the accumulators: 12 resident warps
// of K = 4 hide more of it than 8 of K = 8. Gate plate (201,000 rows, 394 MB of operator), 8 vectors:
// 487 us a call with a grid row per vector (the operator read eight times), 340 us with K = 8 in
// one thread, 208 us with two groups of four (the floor of its bytes is 72 us); 4 vectors 234 -> 116
// us, 2 vectors 119 -> 86 us (one call after another).
template <int K, int G, int W>
__global__ void __launch_bounds__(32 * W * G) sell_energy_kernel(SellOp<double> A, const double* __restrict__ x,
                                                             double* __restrict__ y, uint32_t n, int count,
                                                             uint32_t blocks, double* __restrict__ energy,
                                                             unsigned char* scratch) {
  constexpr int SHARES = kWarps / W;  // blocks to a virtual block
  constexpr int LEN = 9, U = sell_chunk_blocks(LEN, 8), VEC = 2, NV = U * LEN / VEC;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = (int)(warp / W) * K;  // this warp's vectors: first .. first + K - 1, those below count
  const double* xg[K];
#pragma unroll
  for (int k = 0; k < K; ++k) xg[k] = x + (size_t)min(first + k, count - 1) * n;
  double local[K];
#pragma unroll
  for (int k = 0; k < K; ++k) local[k] = 0.0;
  const uint32_t vb = blockIdx.x / SHARES, share = blockIdx.x % SHARES;
  for (uint32_t s = vb * kWarps + share + SHARES * (warp % W); s < A.nslices; s += blocks * kWarps) {
    const uint32_t slot = s * 32 + lane;
    const uint32_t row = A.rows[slot], len = A.len[slot], base = A.start[s];
    double acc[K][3];
#pragma unroll
    for (int k = 0; k < K; ++k) acc[k][0] = acc[k][1] = acc[k][2] = 0.0;
    // Values one chunk ahead, columns two, as in sell_rows.
    uint32_t cn[U], cf[U];
    double vn[U * LEN];
    if (len > 0) {
      load_cols_shared<U>(A.cols + base + lane * U, cn);
      const double2* vp = reinterpret_cast<const double2*>(A.vals + (size_t)base * LEN) + lane;
#pragma unroll
      for (int q = 0; q < NV; ++q) Vec16<double>::split(__ldg(vp + 32 * q), vn + q * VEC);
    }
    if (U < len) load_cols_shared<U>(A.cols + base + 32 * U + lane * U, cf);
    for (uint32_t k0 = 0; k0 < len; k0 += U) {
      uint32_t c[U];
      double v[U * LEN];
#pragma unroll
      for (int u = 0; u < U; ++u) c[u] = cn[u];
#pragma unroll
      for (int i = 0; i < U * LEN; ++i) v[i] = vn[i];
      if (k0 + U < len) {
        const uint32_t q1 = base + 32 * (k0 + U);
#pragma unroll
        for (int u = 0; u < U; ++u) cn[u] = cf[u];
        const double2* vp = reinterpret_cast<const double2*>(A.vals + (size_t)q1 * LEN) + lane;
#pragma unroll
        for (int q = 0; q < NV; ++q) Vec16<double>::split(__ldg(vp + 32 * q), vn + q * VEC);
        if (k0 + 2 * U < len) load_cols_shared<U>(A.cols + q1 + 32 * U + lane * U, cf);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (k0 + u >= len) break;
        double xv[K][3];
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
          for (int q = 0; q < 3; ++q) xv[k][q] = __ldg(xg[k] + (size_t)c[u] * 3 + q);
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
          for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int q = 0; q < 3; ++q) acc[k][p] += v[u * LEN + p * 3 + q] * xv[k][q];
      }
    }
    if (row < A.nrows)
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (first + k < count)
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            const size_t i = (size_t)row * 3 + p;
            y[(size_t)(first + k) * n + i] = acc[k][p];
            local[k] += xg[k][i] * acc[k][p];
          }
  }
  // The energies in the order of finish_partials over `blocks` blocks of kWarps warps: each warp's sum
  // by shuffles; the sums of a block's warps (every SHARES-th one of its virtual block's) in pairs as
  // block_sum pairs them, one partial per block and vector; the last block of the call then pairs the
  // shares and sums each vector's blocks, a warp per vector in the place of its kThreads threads. So an
  // energy does not depend on the number of vectors in the call. One ticket (vector 0's) serves the call.
  __shared__ double sh[K * G][W];
  __shared__ bool last;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double v = local[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if (lane == 0) sh[first + k][warp % W] = v;
  }
  __syncthreads();
  double* partials = reinterpret_cast<double*>(scratch + kEnergyTicketBytes);
  if ((int)threadIdx.x < count) {
    const double* v = sh[threadIdx.x];
    double t;
    if constexpr (W == 2)
      t = v[0] + v[1];
    else
      t = (v[0] + v[2]) + (v[1] + v[3]);
    __stcg(partials + (size_t)threadIdx.x * kEnergyMaxBlocks + blockIdx.x, t);
    __threadfence();
  }
  __syncthreads();
  unsigned* ticket = reinterpret_cast<unsigned*>(scratch);
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int k = (int)warp; k < count; k += W * G) {
    const double* part = partials + (size_t)k * kEnergyMaxBlocks;
    double v[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v[w] = 0.0;
    for (uint32_t b0 = lane; b0 < blocks; b0 += kThreads) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {  // past the last block: zeros, which change nothing
        const uint32_t b = b0 + 32 * w;
        double t[SHARES];
#pragma unroll
        for (int i = 0; i < SHARES; ++i) t[i] = b < blocks ? __ldcg(part + (size_t)b * SHARES + i) : 0.0;
        if constexpr (SHARES == 4)
          v[w] += (t[0] + t[2]) + (t[1] + t[3]);
        else
          v[w] += t[0] + t[1];
      }
    }
#pragma unroll
    for (int w = 0; w < kWarps; ++w)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[w] += __shfl_xor_sync(kFull, v[w], o);
    if (lane == 0) energy[k] = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

// Row-group system, one vector: LPR lanes per row, rows summed as bsr_kernel sums them.
template <int LPR>
__global__ void __launch_bounds__(kThreads) energy_kernel(Op<double> A, const double* __restrict__ x,
                                                           double* __restrict__ y, double* __restrict__ energy,
                                                           unsigned char* scratch) {
  extern __shared__ __align__(16) char smem[];
  char* wbase = smem + (threadIdx.x >> 5) * 2 * slot_bytes(A);
  EpiDot<LPR> epi;
  epi.p = x;
  epi.ap = y;
  epi.local = 0.0;
  run_groups<double, double, 3, 3, LPR, false>(A, x, wbase, epi, OpenGate{}, blockIdx.x, gridDim.x);
  energy_finish(epi.local, scratch, energy);
}

// Row-group system, several vectors: K of them in one walk (blockIdx.y picks the K), so a group's
// staged values are read once for all of them and each x gather round is K times as wide; rows are
// summed as bsr_kernel sums them. One staging slot a warp (a warp has one group or few) on energy_kernel's
// grid, whose warps, blocks and sums these are: an energy does not depend on the number of vectors.
// 26,010 rows, 8 vectors: 109 -> 68 us a call, 3 vectors 45 -> 38; 3,240 rows, 8 vectors: 29 -> 21
// (with a grid row per vector before; one call after another).
template <int LPR, int K>
__global__ void __launch_bounds__(kThreads) energy_groups_kernel(Op<double> A, const double* __restrict__ x,
                                                                  double* __restrict__ y, uint32_t n, int count,
                                                                  double* __restrict__ energy, unsigned char* scratch) {
  extern __shared__ __align__(16) char smem[];
  constexpr int TEAMS = 32 / LPR;
  const int lane = threadIdx.x & 31, team = lane / LPR, tl = lane % LPR;
  char* base = smem + (threadIdx.x >> 5) * slot_bytes(A);
  const int first = (int)blockIdx.y * K;
  const double* xg[K];
#pragma unroll
  for (int k = 0; k < K; ++k) xg[k] = x + (size_t)min(first + k, count - 1) * n;
  double local[K];
#pragma unroll
  for (int k = 0; k < K; ++k) local[k] = 0.0;
  const uint32_t warps = blockDim.x >> 5;
  for (uint32_t g = blockIdx.x * warps + (threadIdx.x >> 5); g < A.ngroups; g += gridDim.x * warps) {
    const uint4 d = A.groups[g];
    const int vo = stage_async(A.vals + (size_t)d.z * 9, (d.w - d.z) * 72u, base, lane);
    const int co = stage_async(A.cols + d.z, (d.w - d.z) * 4u, base + A.vbuf, lane);
    const int so = stage_async(A.starts + d.x, (d.y - d.x + 1) * 4u, base + A.vbuf + A.cbuf, lane);
    cp_async_commit();
    cp_async_wait_all();
    __syncwarp();
    const double* vals = reinterpret_cast<const double*>(base + vo);
    const uint32_t* cols = reinterpret_cast<const uint32_t*>(base + A.vbuf + co);
    const uint32_t* rst = reinterpret_cast<const uint32_t*>(base + A.vbuf + A.cbuf + so);
    const uint32_t nrows = d.y - d.x;
    for (uint32_t rb = 0; rb < nrows; rb += TEAMS) {
      const uint32_t lr = rb + team;
      const bool live = lr < nrows;
      double acc[K][3];
#pragma unroll
      for (int k = 0; k < K; ++k) acc[k][0] = acc[k][1] = acc[k][2] = 0.0;
      const uint32_t b1 = live ? rst[lr + 1] - d.z : 0;
      for (uint32_t j = live ? rst[lr] - d.z + tl : 0; j < b1; j += LPR) {
        const size_t c = (size_t)cols[j] * 3;
        double xv[K][3];
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
          for (int q = 0; q < 3; ++q) xv[k][q] = __ldg(xg[k] + c + q);
        const double* v = vals + (size_t)j * 9;
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
          for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int q = 0; q < 3; ++q) acc[k][p] += v[p * 3 + q] * xv[k][q];
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int o = LPR / 2; o > 0; o >>= 1) acc[k][p] += __shfl_xor_sync(kFull, acc[k][p], o);
      if (live && tl < 3) {
        const size_t i = (size_t)(d.x + lr) * 3 + tl;
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (first + k < count) {
            const double sum = pick<double, 3>(acc[k], tl);
            y[(size_t)(first + k) * n + i] = sum;
            local[k] += xg[k][i] * sum;
          }
      }
    }
    __syncwarp();
  }
  double total[K];
  double* partials = reinterpret_cast<double*>(scratch + kEnergyTicketBytes) + (size_t)first * kEnergyMaxBlocks;
  if (finish_partials<K>(local, partials, reinterpret_cast<unsigned*>(scratch) + blockIdx.y, total) && threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (first + k < count) energy[first + k] = total[k];
}

template <int LPR>
cudaError_t energy_groups_opt_in(int smem) {
  const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(energy_groups_kernel<LPR, 2>, attr, smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(energy_groups_kernel<LPR, 3>, attr, smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(energy_groups_kernel<LPR, 4>, attr, smem);
  return e;
}

std::mutex g_energy_mutex;
unsigned char* g_energy_address[kEnergyMaxDevices] = {};

// Once per device, with that device current: the scratch's device address and the row-group
// variants' shared-memory opt-in. Neither allocates memory; the first lookup on a device can load
// this library's device code there.
sf_status energy_setup(int device, unsigned char** out) {
  std::lock_guard<std::mutex> lock(g_energy_mutex);
  if (device < 0 || device >= kEnergyMaxDevices) return fail(SF_INVALID_ARGUMENT, "device ordinal out of range");
  if (!g_energy_address[device]) {
    unsigned char* ptr = nullptr;
    if (sf_status e = cuda_check(cudaGetSymbolAddress((void**)&ptr, g_energy_scratch), "cudaGetSymbolAddress"))
      return e;
    const int smem = 200 * 1024;
    cudaError_t e = cudaFuncSetAttribute(energy_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(energy_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(energy_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(energy_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = energy_groups_opt_in<4>(smem);
    if (e == cudaSuccess) e = energy_groups_opt_in<8>(smem);
    if (e == cudaSuccess) e = energy_groups_opt_in<16>(smem);
    if (e == cudaSuccess) e = energy_groups_opt_in<32>(smem);
    if (sf_status st = cuda_check(e, "cudaFuncSetAttribute")) return st;
    g_energy_address[device] = ptr;
  }
  *out = g_energy_address[device];
  return SF_OK;
}

unsigned energy_one_blocks(uint32_t nslices) { return (unsigned)std::min(grid_for_slices(nslices), kEnergyOneBlocks); }

template <int K, int G>
void launch_energy_sell(const SellOp<double>& A, const double* x, double* y, uint32_t n, int count, double* energy,
                        unsigned char* scratch, cudaStream_t st) {
  // A block per W slices (of the blocks of sell_energy_one_kernel, whose sums are formed), so the SMs
  // that finish early take the next ones.
  constexpr int W = G == 1 ? 4 : 2;  // 128 threads, three resident blocks at about 166 registers
  static_assert(kWarps == 8 && kWarps / 2 * kEnergyOneBlocks <= kEnergyMaxBlocks, "a partial per block");
  const unsigned blocks = energy_one_blocks(A.nslices);
  sell_energy_kernel<K, G, W><<<blocks * (kWarps / W), 32 * W * G, 0, st>>>(A, x, y, n, count, blocks, energy, scratch);
}

template <int LPR>
void launch_energy_lpr(const DevBsr& m, const double* x, double* y, double* energy, unsigned char* scratch,
                       cudaStream_t st) {
  Op<double> A = op_of<double>(m);
  Shape sh = shape_of(A, true);
  energy_kernel<LPR><<<std::min(sh.grid, kEnergyOneBlocks), sh.threads, sh.smem, st>>>(A, x, y, energy, scratch);
}

template <int LPR, int K>
void launch_energy_groups(const DevBsr& m, const double* x, double* y, uint32_t n, double* energy, int count,
                          unsigned char* scratch, cudaStream_t st) {
  Op<double> A = op_of<double>(m);
  const Shape sh = shape_of(A, true);  // the blocks of energy_kernel, whose sums are formed
  const dim3 grid((unsigned)std::min(sh.grid, kEnergyOneBlocks), (unsigned)((count + K - 1) / K));
  energy_groups_kernel<LPR, K><<<grid, sh.threads, sh.smem / 2, st>>>(A, x, y, n, count, energy, scratch);
}

// Two to four vectors in one walk, five to eight in two of three or four.
template <int LPR>
void launch_energy_rows(const DevBsr& m, const double* x, double* y, uint32_t n, double* energy, uint64_t count,
                        unsigned char* scratch, cudaStream_t st) {
  const int k = (int)count;
  if (k == 1) launch_energy_lpr<LPR>(m, x, y, energy, scratch, st);
  else if (k == 2) launch_energy_groups<LPR, 2>(m, x, y, n, energy, k, scratch, st);
  else if (k == 3 || k == 5 || k == 6) launch_energy_groups<LPR, 3>(m, x, y, n, energy, k, scratch, st);
  else launch_energy_groups<LPR, 4>(m, x, y, n, energy, k, scratch, st);
}

}  // namespace

uint64_t solver_energy_max_vectors() { return kEnergyMaxVectors; }

sf_status solver_energy_products(DeviceSolver& s, const double* x, double* y, double* energy, uint64_t count) {
  if (count > (uint64_t)kEnergyMaxVectors) {
    char msg[160];
    std::snprintf(msg, sizeof msg, "count %llu exceeds the %d vectors the energy scratch holds",
                  (unsigned long long)count, kEnergyMaxVectors);
    return fail(SF_INVALID_ARGUMENT, msg);
  }
  if (count == 0) return SF_OK;
  unsigned char* scratch = nullptr;
  if (sf_status e = energy_setup(s.device, &scratch)) return e;
  const DevBsr& m = s.system;
  if (m.sell) {
    SellOp<double> A = sell_of<double>(m);
    const int k = (int)count;
    if (k == 1) sell_energy_one_kernel<<<energy_one_blocks(m.nslices), kThreads, 0, s.stream>>>(A, x, y, energy, scratch);
    else if (k == 2) launch_energy_sell<2, 1>(A, x, y, s.n, k, energy, scratch, s.stream);
    else if (k == 3) launch_energy_sell<3, 1>(A, x, y, s.n, k, energy, scratch, s.stream);
    else if (k == 4) launch_energy_sell<4, 1>(A, x, y, s.n, k, energy, scratch, s.stream);
    else if (k <= 6) launch_energy_sell<3, 2>(A, x, y, s.n, k, energy, scratch, s.stream);
    else launch_energy_sell<4, 2>(A, x, y, s.n, k, energy, scratch, s.stream);
  } else {
    switch (m.lanes_per_row) {
      case 4: launch_energy_rows<4>(m, x, y, s.n, energy, count, scratch, s.stream); break;
      case 8: launch_energy_rows<8>(m, x, y, s.n, energy, count, scratch, s.stream); break;
      case 16: launch_energy_rows<16>(m, x, y, s.n, energy, count, scratch, s.stream); break;
      default: launch_energy_rows<32>(m, x, y, s.n, energy, count, scratch, s.stream); break;
    }
  }
  s.launches += 1;
  return cuda_check(cudaGetLastError(), "energy products");
}

}  // namespace sf
