// run_iterations and its graphs on a stand-in runtime: `iterations <case>`. A "kernel" of an
// iteration counts itself in the solver's state.
#include "fake_cuda.h"

#include <cmath>

#include "device.h"

using namespace sf;

namespace {

struct FakeGraph {
  uint64_t iterations = 0;
};
FakeGraph* capturing = nullptr;
int graphs = 0, execs = 0;  // alive
int begins = 0;             // captures begun
uint64_t kernels = 5;       // an iteration's
int instantiations_left = 1 << 30, run_launches_left = 1 << 30, enqueues_left = 1 << 30;
uint64_t run_launches = 0, single_launches = 0;
PcgState* device_state = nullptr;
uint64_t converges_at = 400;

void iterate() {
  PcgState& s = *device_state;
  if (s.status != ST_ACTIVE) return;
  s.iterations += 1;
  s.rel = std::pow(s.tolerance, (double)s.iterations / (double)converges_at);
  if (s.iterations >= converges_at) s.status = ST_CONVERGED;
}

}  // namespace

extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  ++begins;
  capturing = new FakeGraph;
  ++graphs;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)capturing;
  capturing = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  if (instantiations_left-- <= 0) return fake::failed(cudaErrorMemoryAllocation);
  *e = (cudaGraphExec_t) new FakeGraph(*(FakeGraph*)g);
  ++execs;
  return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t*, size_t* n) {
  *n = kernels * ((FakeGraph*)g)->iterations;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  const uint64_t n = ((FakeGraph*)e)->iterations;
  if (n > 1 && run_launches_left-- <= 0) return fake::failed(cudaErrorMemoryAllocation);
  (n > 1 ? run_launches : single_launches) += 1;
  for (uint64_t i = 0; i < n; ++i) fake::stream.push_back(iterate);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete (FakeGraph*)g;
  --graphs;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete (FakeGraph*)e;
  --execs;
  return cudaSuccess;
}
}

namespace sf {
sf_error& error_slot() {
  static sf_error e{};
  return e;
}
sf_status solver_enqueue_iteration(DeviceSolver& s) {
  s.launches_per_iteration = kernels;
  if (enqueues_left-- <= 0) return SF_CUDA_ERROR;
  if (capturing)
    capturing->iterations += 1;
  else
    fake::stream.push_back(iterate);
  return SF_OK;
}
}  // namespace sf

namespace {

struct Solve {
  DeviceSolver d;
  PcgState state{}, pinned{}, last{};
  int status = ST_ACTIVE;
  bool cancelled = false;
  Solve() {
    d.n = 9720;
    d.state = device_state = &state;
    state.tolerance = 1e-9;
    CHECK(solver_capture_graph(d) == SF_OK && d.graph_kernels == kernels);
  }
  ~Solve() {  // as dev_free_all
    if (d.graph_exec) cudaGraphExecDestroy(d.graph_exec);
    if (d.graph) cudaGraphDestroy(d.graph);
    if (d.run_exec) cudaGraphExecDestroy(d.run_exec);
    if (d.run_graph) cudaGraphDestroy(d.run_graph);
  }
  sf_status run(uint64_t n) { return run_iterations(d, true, n, nullptr, nullptr, &pinned, last, status, cancelled); }
};

// A longer graph that cannot be made (or launched) leaves the solve to the one at hand, is not tried
// again, and leaves neither a graph nor an error behind.
void no_run_graph() {
  {
    Solve s;
    CHECK(s.run(203) == SF_OK);
    CHECK(s.last.iterations == 203 && s.d.iterations_run == 203);
    CHECK(s.d.launches == 5 * 203);
    CHECK(s.run(50) == SF_OK);
    CHECK(s.last.iterations == 253);
    CHECK(run_launches == 0 && single_launches == 253);
    CHECK(begins == 2 && graphs == 1 && execs == 1);
    CHECK(cudaGetLastError() == cudaSuccess);
  }
  CHECK(graphs == 0 && execs == 0);
}

// One solve of a new solver: whether the longer graph is made, and how many iterations it takes on.
void one_solve(uint64_t iterations, bool made) {
  converges_at = iterations;
  Solve s;
  CHECK(s.run(~0ull >> 1) == SF_OK && s.status == ST_CONVERGED && s.last.iterations == iterations);
  CHECK(begins == (made ? 2 : 1));
  CHECK(!made || kRunIterations * run_launches >= iterations - 2 * kRunWorthPerKernel);
}

// Short solves of a solver that stays: made at the start of one, once they add up.
void many_solves(uint64_t iterations) {
  converges_at = iterations;
  Solve s;
  for (uint64_t ran = 0, i = 0; i < 20; ++i) {
    const bool due = ran >= kRunWorthPerKernel * kernels;
    s.state.iterations = 0;
    s.state.status = s.status = ST_ACTIVE;
    s.state.rel = 1.0;
    const uint64_t before = run_launches;
    CHECK(s.run(~0ull >> 1) == SF_OK && s.last.iterations == iterations);
    CHECK(begins == (due ? 2 : 1) && (run_launches > before) == due);
    ran = s.d.iterations_run;
  }
  CHECK(begins == 2);
}

void whole_solve(uint64_t total) {
  {
    Solve s;
    CHECK(s.run(total) == SF_OK);
    CHECK(s.last.iterations == total && s.d.iterations_run == total);
    CHECK(run_launches > 0 && single_launches + kRunIterations * run_launches == total);
    CHECK(begins == 2 && graphs == 2 && execs == 2);
  }
  CHECK(graphs == 0 && execs == 0);
}

}  // namespace

int main(int argc, char** argv) {
  const std::string what = argv[1];
  if (what == "whole") whole_solve(203);
  if (what == "soon-over") one_solve(90, false);
  if (what == "long-enough") one_solve(100, true);
  if (what == "long") one_solve(211, true);
  if (what == "short-solves") {
    kernels = 14;
    many_solves(39);
  }
  if (what == "no-instantiation") {
    instantiations_left = 1;
    no_run_graph();
  }
  if (what == "no-capture") {
    enqueues_left = 2;
    no_run_graph();
  }
  if (what == "no-launch") {
    run_launches_left = 0;
    no_run_graph();
  }
  return 0;
}
