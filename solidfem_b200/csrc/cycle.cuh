// The V-cycle's launch sequence (cycle.rs:461-651) over the kernels of solve_kernels.cuh, the
// inspection of its stages and the timing of its finest level's kernels.
#pragma once

#include "solve_kernels.cuh"

namespace sf {

namespace {

template <typename S, typename V>
StartArgs<S, V> start_args(const DevLevel& L, V* b_out, V* x) {
  StartArgs<S, V> a;
  a.dinv = (const S*)L.dinv;
  a.b_out = b_out;
  a.r = (V*)L.res;
  a.d = (V*)L.d0;
  a.x = x;
  a.theta = (V)L.theta;
  return a;
}

// The smoother from a zero guess on right-hand side b into x (cycle.rs:570-651). `outer`, when
// given, receives x += (smoothed x) at the last step instead of storing x.
template <typename S, typename V, typename B>
void enqueue_smooth(DeviceSolver& s, DevLevel& L, const B* b_in, V* b_out, V* x, V* outer, const int* status,
                    bool started = false) {
  cudaStream_t st = s.stream;
  V* r = (V*)L.res;
  V* d[2] = {(V*)L.d0, (V*)L.d1};
  if (!started) {  // else the product that made b_in did the start
    if (L.a.rb == 3)
      launch_cheb_start<S, V, B, 3>(L, b_in, b_out, r, d[0], x, L.theta, status, st);
    else
      launch_cheb_start<S, V, B, 6>(L, b_in, b_out, r, d[0], x, L.theta, status, st);
    s.launches_per_iteration++;
  }
  for (size_t k = 0; k < L.steps.size(); ++k) {
    bool last = k + 1 == L.steps.size();
    V* o = last ? outer : nullptr;
    if (L.a.rb == 3)
      launch_cheb_step<S, V, 3>(L, d[k & 1], d[(k + 1) & 1], r, x, o, L.steps[k].first, L.steps[k].second, status, st);
    else
      launch_cheb_step<S, V, 6>(L, d[k & 1], d[(k + 1) & 1], r, x, o, L.steps[k].first, L.steps[k].second, status, st);
    s.launches_per_iteration++;
  }
  if (outer && L.steps.empty()) {
    launch_body<add_kernel<V>>(grid_for_elems(L.n), kThreads, 0, st, L.n, outer, x, status);
    s.launches_per_iteration++;
  }
}

template <typename S>
TailMat<S> tail_mat(const DevBsr& m) {
  TailMat<S> t;
  t.starts = m.starts;
  t.cols = m.cols;
  t.vals = (const S*)m.vals;
  t.rows = m.rows;
  t.lanes = m.lanes_per_row;
  return t;
}

// Levels li and li + 1 (the coarsest, factored) as one cluster launch of tail_kernel.
template <typename S, typename V>
void enqueue_tail(DeviceSolver& s, size_t li, const int* status) {
  DevLevel& L = s.levels[li];
  DevLevel& C = s.levels[li + 1];
  TailArgs<S, V> t = {};
  t.a = tail_mat<S>(L.a);
  t.r = tail_mat<S>(L.r);
  t.p = tail_mat<S>(L.p);
  t.dinv = (const S*)L.dinv;
  t.inv = C.coarse_inverse;
  t.nc = C.n;
  t.nsteps = (uint32_t)L.steps.size();
  t.theta = (V)L.theta;
  for (size_t k = 0; k < L.steps.size(); ++k) {
    t.keep[k] = (V)L.steps[k].first;
    t.step[k] = (V)L.steps[k].second;
  }
  t.b = (const V*)L.b;
  t.x = (V*)L.x;
  t.status = status;
  launch_body_cluster<tail_kernel<S, V>, tail_threads<V>()>(dim3(s.tail_cluster), s.tail_smem, s.stream, t);
  s.launches_per_iteration++;
}

// CTAs of the tail's cluster on this device and their shared memory: 16 (a non-portable size)
// when each CTA's share fits kTailMaxSmem and the device can place such a cluster, else 8, else
// 0 (no tail). `hs` is the fused level, `hc` the coarsest.
template <typename S, typename V>
unsigned tail_cluster_size(const HostLevel& hs, const HostLevel& hc, size_t* smem) {
  typedef BodyTraits<decltype(&tail_kernel<S, V>)> T;
  const void* single = T::template single_n<tail_kernel<S, V>, tail_threads<V>()>();
  const void* batched = T::template batched_n<tail_kernel<S, V>, tail_threads<V>()>();
  const uint32_t nc = (uint32_t)(hc.a.rows * hc.a.rb);
  cudaFuncSetAttribute(single, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaFuncSetAttribute(batched, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  for (unsigned c : {16u, 8u}) {
    size_t bytes = 0;
    for (unsigned i = 0; i < c; ++i)
      bytes = std::max(bytes, tail_cta_bytes(hs.a.starts, hs.p.starts, hs.t_starts, nc, c, i, sizeof(S), sizeof(V)));
    if (bytes > kTailMaxSmem) continue;
    cudaFuncSetAttribute(single, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    cudaFuncSetAttribute(batched, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = c;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(tail_threads<V>());
    cfg.dynamicSmemBytes = bytes;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, single, &cfg) == cudaSuccess && clusters > 0) {
      *smem = bytes;
      return c;
    }
    cudaGetLastError();
  }
  return 0;
}

// One V-cycle from level `li` (cycle.rs:461-539). B is the type of the right-hand side; an f64
// right-hand side reaching an f32 level is rounded into b_store first.
template <typename S, typename V, typename B>
void enqueue_cycle(DeviceSolver& s, size_t li, const B* rhs, V* b_store, V* x, const int* status,
                   bool started = false) {
  if ((int)li == s.tail_level) {
    enqueue_tail<S, V>(s, li, status);
    return;
  }
  DevLevel& L = s.levels[li];
  cudaStream_t st = s.stream;
  if (!L.has_p) {
    if (L.has_factor) {
      const V* bv = (const V*)rhs;
      if (b_store) {
        launch_body<convert_kernel<B, V>>(grid_for_elems(L.n), kThreads, 0, st, L.n, rhs, b_store, status);
        s.launches_per_iteration++;
        bv = b_store;
      }
      launch_body<coarse_solve_kernel<V>>(grid_for_rows(L.n), kThreads, 0, st, L.n, L.coarse_inverse, bv, x, status);
      s.launches_per_iteration++;
    } else {
      enqueue_smooth<S, V, B>(s, L, rhs, b_store, x, nullptr, status, started);
    }
    return;
  }
  enqueue_smooth<S, V, B>(s, L, rhs, b_store, x, nullptr, status, started);
  const V* b = b_store ? (const V*)b_store : (const V*)rhs;
  DevLevel& C = s.levels[li + 1];
  bsr_dispatch<S, V, OP_RESIDUAL>(L.a, x, (V*)L.res, b, status, st);
  // The restriction; when the coarser level starts with its smoother, that start is fused in.
  const bool fuse = (int)(li + 1) != s.tail_level && (C.has_p || !C.has_factor);
  if (fuse)
    launch_start_product<S, V, OP_SET>(L.r, (const V*)L.res, (const V*)nullptr,
                                       start_args<S, V>(C, (V*)C.b, (V*)C.x), status, st);
  else
    bsr_dispatch<S, V, OP_SET>(L.r, (const V*)L.res, (V*)C.b, nullptr, status, st);
  s.launches_per_iteration += 2;
  enqueue_cycle<S, V, V>(s, li + 1, (const V*)C.b, nullptr, (V*)C.x, status, fuse);
  bsr_dispatch<S, V, OP_ADD>(L.p, (const V*)C.x, x, nullptr, status, st);
  // The residual b - A x with the post-smoother's start fused in (its right-hand side stays in
  // registers).
  launch_start_product<S, V, OP_RESIDUAL>(L.a, (const V*)x, b, start_args<S, V>(L, (V*)nullptr, (V*)L.post_x),
                                          status, st);
  s.launches_per_iteration += 2;
  enqueue_smooth<S, V, V>(s, L, (const V*)nullptr, nullptr, (V*)L.post_x, x, status, true);
}

template <typename S, typename V>
sf_status time_level0(DeviceSolver& s, int kernel, uint64_t repeats, double* ms, double* bytes) {
  DevLevel& L = s.levels[0];
  const int* on = s.always_active;
  double rows = L.a.rows, blocks = (double)L.a.blocks, rb = L.a.rb, sv = sizeof(V), ss = sizeof(S);
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  cudaEventRecord(a, s.stream);
  for (uint64_t i = 0; i < repeats; ++i) {
    if (kernel == SF_KERNEL_CHEBYSHEV_STEP) {
      V* d[2] = {(V*)L.d0, (V*)L.d1};
      launch_cheb_step<S, V, 3>(L, d[i & 1], d[(i + 1) & 1], (V*)L.res, (V*)L.x, nullptr, 0.5, 0.25, on, s.stream);
    } else if (kernel == SF_KERNEL_LEVEL_RESIDUAL) {
      launch_bsr<S, V, 3, 3, OP_RESIDUAL>(L.a, (const V*)L.x, (V*)L.tmp, (const V*)L.b, on, s.stream);
    } else {
      bsr_dispatch<S, V, OP_SET>(L.r, (const V*)L.res, (V*)s.levels[1].b, nullptr, on, s.stream);
    }
  }
  cudaEventRecord(b, s.stream);
  cudaError_t e = cudaEventSynchronize(b);
  float t = 0;
  cudaEventElapsedTime(&t, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  *ms = t / (double)repeats;
  double matrix = rows * 4 + blocks * (rb * rb * ss + 4);
  double vec = rows * rb * sv;
  if (kernel == SF_KERNEL_CHEBYSHEV_STEP)
    *bytes = matrix + vec /* d_old */ + 2 * vec /* r */ + rows * rb * rb * ss /* D^-1 */ + vec /* d_new */ + 2 * vec /* x */;
  else if (kernel == SF_KERNEL_LEVEL_RESIDUAL)
    *bytes = matrix + 3 * vec;
  else
    *bytes = (double)L.r.rows * 4 + (double)L.r.blocks * (L.r.rb * L.r.cb * ss + 4) + vec +
             (double)L.r.rows * L.r.rb * sv;
  s.launches += repeats;
  return cuda_check(e, "time kernel");
}

// One stage of level li's V-cycle on the level's own buffers, through the launches the cycle
// makes (same layouts, same fused epilogues): inputs in f64 device memory are rounded to the
// vector type first, outputs widened to f64. The stages and their buffers:
//   SMOOTH          b -> L.b;  smoother from zero into L.x
//   SMOOTH_ADD      b -> L.b, x -> L.tmp;  L.tmp += smoother (the post-smoother's last step)
//   START           b -> L.b;  the start kernel: L.x = (D^-1 b) / theta
//   RESIDUAL        b -> L.b, x -> L.x;  L.res = b - A x
//   RESTRICT        r -> L.res;  C.b = R r
//   PROLONG         e -> C.x, x -> L.x;  L.x += P e
//   RESTRICT_START  r -> L.res;  C.b = R r with the coarser level's start fused in (C.x)
//   RESIDUAL_START  b -> L.b, x -> L.x;  L.res = b - A x with the start fused in (L.post_x)
template <typename S, typename V>
sf_status level_stage(DeviceSolver& s, size_t li, int stage, const double* in0, const double* in1, double* out0,
                      double* out1) {
  DevLevel& L = s.levels[li];
  const bool coarse = li + 1 < s.levels.size();
  DevLevel* C = coarse ? &s.levels[li + 1] : nullptr;
  cudaStream_t st = s.stream;
  const int* on = s.always_active;
  auto to_v = [&](const double* src, void* dst, uint32_t n) {
    launch_body<convert_kernel<double, V>>(grid_for_elems(n), kThreads, 0, st, n, src, (V*)dst, on);
  };
  auto from_v = [&](const void* src, double* dst, uint32_t n) {
    launch_body<convert_kernel<V, double>>(grid_for_elems(n), kThreads, 0, st, n, (const V*)src, dst, on);
  };
  const bool smoothed = L.has_p || !L.has_factor;
  switch (stage) {
    case SF_STAGE_SMOOTH:
    case SF_STAGE_SMOOTH_ADD:
    case SF_STAGE_START:
      if (!smoothed) return fail(SF_INVALID_ARGUMENT, "the coarsest level is factored, not smoothed");
      to_v(in0, L.b, L.n);
      if (stage == SF_STAGE_START) {
        if (L.a.rb == 3)
          launch_cheb_start<S, V, V, 3>(L, (const V*)L.b, nullptr, (V*)L.res, (V*)L.d0, (V*)L.x, L.theta, on, st);
        else
          launch_cheb_start<S, V, V, 6>(L, (const V*)L.b, nullptr, (V*)L.res, (V*)L.d0, (V*)L.x, L.theta, on, st);
        from_v(L.x, out0, L.n);
      } else if (stage == SF_STAGE_SMOOTH) {
        enqueue_smooth<S, V, V>(s, L, (const V*)L.b, nullptr, (V*)L.x, nullptr, on);
        from_v(L.x, out0, L.n);
      } else {
        to_v(in1, L.tmp, L.n);
        enqueue_smooth<S, V, V>(s, L, (const V*)L.b, nullptr, (V*)L.post_x, (V*)L.tmp, on);
        from_v(L.tmp, out0, L.n);
      }
      break;
    case SF_STAGE_RESIDUAL:
    case SF_STAGE_RESIDUAL_START:
      to_v(in0, L.b, L.n);
      to_v(in1, L.x, L.n);
      if (stage == SF_STAGE_RESIDUAL) {
        bsr_dispatch<S, V, OP_RESIDUAL>(L.a, (const V*)L.x, (V*)L.res, (const V*)L.b, on, st);
      } else {
        if (!smoothed) return fail(SF_INVALID_ARGUMENT, "the coarsest level is factored, not smoothed");
        launch_start_product<S, V, OP_RESIDUAL>(L.a, (const V*)L.x, (const V*)L.b,
                                                start_args<S, V>(L, (V*)nullptr, (V*)L.post_x), on, st);
        from_v(L.post_x, out1, L.n);
      }
      from_v(L.res, out0, L.n);
      break;
    case SF_STAGE_RESTRICT:
    case SF_STAGE_RESTRICT_START:
      if (!L.has_p) return fail(SF_INVALID_ARGUMENT, "the level has no coarser level");
      to_v(in0, L.res, L.n);
      if (stage == SF_STAGE_RESTRICT) {
        bsr_dispatch<S, V, OP_SET>(L.r, (const V*)L.res, (V*)C->b, nullptr, on, st);
      } else {
        if (!C->has_p && C->has_factor) return fail(SF_INVALID_ARGUMENT, "the coarser level is factored, not smoothed");
        launch_start_product<S, V, OP_SET>(L.r, (const V*)L.res, (const V*)nullptr,
                                           start_args<S, V>(*C, (V*)C->b, (V*)C->x), on, st);
        from_v(C->x, out1, C->n);
      }
      from_v(C->b, out0, C->n);
      break;
    case SF_STAGE_PROLONG:
      if (!L.has_p) return fail(SF_INVALID_ARGUMENT, "the level has no coarser level");
      to_v(in0, C->x, C->n);
      to_v(in1, L.x, L.n);
      bsr_dispatch<S, V, OP_ADD>(L.p, (const V*)C->x, (V*)L.x, nullptr, on, st);
      from_v(L.x, out0, L.n);
      break;
    default:
      return fail(SF_INVALID_ARGUMENT, "unknown stage");
  }
  s.launches += 4;
  return cuda_check(cudaStreamSynchronize(st), "level stage");
}

}  // namespace

template <typename S, typename V>
void Cycle<S, V>::precondition(DeviceSolver& s, const double* r, V* z, const int* status) {
  V* b_store = sizeof(V) == 4 ? (V*)s.levels[0].b : nullptr;
  enqueue_cycle<S, V, double>(s, 0, r, b_store, z, status);
}

template <typename S, typename V>
sf_status Cycle<S, V>::stage(DeviceSolver& s, size_t li, int stage, const double* in0, const double* in1, double* out0,
                             double* out1) {
  return level_stage<S, V>(s, li, stage, in0, in1, out0, out1);
}

template <typename S, typename V>
sf_status Cycle<S, V>::time_kernel(DeviceSolver& s, int kernel, uint64_t repeats, double* ms, double* bytes) {
  return time_level0<S, V>(s, kernel, repeats, ms, bytes);
}

template <typename S, typename V>
unsigned Cycle<S, V>::tail_cluster(const HostLevel& hs, const HostLevel& hc, size_t* smem) {
  return tail_cluster_size<S, V>(hs, hc, smem);
}

}  // namespace sf
