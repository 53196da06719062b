// The solve's iterations as CUDA graphs, and the loop that replays them (host code; the kernels an
// iteration enqueues are solve.cu's).
#include <algorithm>
#include <cmath>

#include "device.h"

namespace sf {

namespace {

// On a failure there is neither graph nor executable.
sf_status capture_iterations(DeviceSolver& s, uint64_t count, cudaGraph_t* graph, cudaGraphExec_t* exec) {
  cudaError_t e = cudaStreamBeginCapture(s.stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return cuda_check(e, "begin capture");
  sf_status st = SF_OK;
  for (uint64_t i = 0; i < count && !st; ++i) st = solver_enqueue_iteration(s);
  cudaGraph_t g = nullptr;
  e = cudaStreamEndCapture(s.stream, &g);
  if (!st) st = cuda_check(e, "end capture");
  if (!st) st = cuda_check(cudaGraphInstantiate(exec, g, 0), "graph instantiate");
  if (st) {
    if (g) cudaGraphDestroy(g);
    g = nullptr;
    *exec = nullptr;
  }
  *graph = g;
  return st;
}

// The longer graph is a gain, not a need: when it cannot be made or launched (a device full of
// resident studies) the solver goes on with the graph of one iteration, and does not try again.
void give_up_run(DeviceSolver& s) {
  if (s.run_exec) cudaGraphExecDestroy(s.run_exec);
  if (s.run_graph) cudaGraphDestroy(s.run_graph);
  s.run_exec = nullptr;
  s.run_graph = nullptr;
  s.run_failed = true;
  cudaGetLastError();
}

// Iterations still to come by the mean rate of the `last` ones (0 while that says little), at most
// `most`.
uint64_t expected_iterations(const PcgState& last, uint64_t most) {
  if (last.iterations < 12 || !(last.rel > last.tolerance && last.rel < 1.0) || !(last.tolerance > 0.0)) return 0;
  const double more = (double)last.iterations * std::log(last.rel / last.tolerance) / -std::log(last.rel);
  return more >= (double)most ? most : (uint64_t)more;
}

// Enqueues kRunIterations iterations as one graph; false when that is not to be had, or not worth
// its making yet: `expected` more iterations are in sight, or `opening` a step, when what the solver
// has run so far stands for what is to come.
bool launch_run(DeviceSolver& s, bool opening, uint64_t expected) {
  if (s.run_failed) return false;
  if (!s.run_exec) {
    const uint64_t worth = kRunWorthPerKernel * s.graph_kernels;
    if (expected < worth && !(opening && s.iterations_run >= worth)) return false;
    const sf_error kept = error_slot();  // a failure here is not the caller's
    if (capture_iterations(s, kRunIterations, &s.run_graph, &s.run_exec)) {
      error_slot() = kept;
      give_up_run(s);
      return false;
    }
  }
  if (cudaGraphLaunch(s.run_exec, s.stream) != cudaSuccess) {
    give_up_run(s);
    return false;
  }
  s.launches += kRunIterations * s.graph_kernels;
  return true;
}

}  // namespace

sf_status solver_capture_graph(DeviceSolver& s) {
  if (s.graph_exec) return SF_OK;
  if (sf_status e = capture_iterations(s, 1, &s.graph, &s.graph_exec)) return e;
  size_t nodes = 0;
  cudaGraphGetNodes(s.graph, nullptr, &nodes);
  s.graph_kernels = nodes;
  return SF_OK;
}

// Pcg::step (pcg.rs:167-190) on the device: up to max_iterations iterations, enqueued in chunks;
// every kernel of an iteration after the solve ends returns at once, so the state is read back
// once per chunk, with one chunk in flight ahead. `cancel` is read before every iteration.
sf_status run_iterations(DeviceSolver& d, bool use_graphs, uint64_t max_iterations, sf_cancel_fn cancel, void* user,
                         PcgState* pinned, PcgState& last, int& status, bool& cancelled) {
  uint64_t done = 0;
  const uint64_t chunk_max = 16;
  uint64_t chunk = 4;
  bool stop = false;
  while (!stop && done < max_iterations) {
    uint64_t k = std::min<uint64_t>(chunk, max_iterations - done);
    uint64_t launched = 0;
    while (launched < k) {
      // Whole runs of iterations where no cancel must be read between them.
      if (use_graphs && !cancel && k - launched >= kRunIterations && d.n <= kRunMaxUnknowns &&
          launch_run(d, done == 0, done ? expected_iterations(last, max_iterations - done) : 0)) {
        launched += kRunIterations;
        continue;
      }
      if (cancel && cancel(user)) {
        cancelled = true;
        stop = true;
        break;
      }
      sf_status e = SF_OK;
      if (use_graphs) {
        e = cuda_check(cudaGraphLaunch(d.graph_exec, d.stream), "graph launch");
        d.launches += d.graph_kernels;
      } else {
        e = solver_enqueue_iteration(d);
        d.launches += d.launches_per_iteration;
      }
      if (e) return e;
      ++launched;
    }
    done += launched;
    d.iterations_run += launched;
    copy_d2h(d, pinned, d.state, sizeof(PcgState));
    if (sf_status e = cuda_check(cudaStreamSynchronize(d.stream), "solver step")) return e;
    last = *pinned;
    status = last.status;
    if (status != ST_ACTIVE) stop = true;
    chunk = std::min(chunk_max, chunk * 2);
  }
  return SF_OK;
}

}  // namespace sf
