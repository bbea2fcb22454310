// lbm_issue.h — how a run of n steps is issued: loose launches, or CUDA graphs
// of them.  Host code over the runtime API only, templated on the domain, so
// that it builds without the kernels.
#pragma once
#include <cuda_runtime.h>

#include "../../include/lbm_b200.h"
#include "lbm_internal.h"

namespace lbm {

// steps per captured graph chunk (even, so that a chunk returns the lattices
// and the boundary planes to the parity it started from)
constexpr int kGraphSteps = 32;

// The captured steps of a domain, one graph per starting lattice (AA: layout):
// kGraphSteps plain steps, and the last rest_steps steps of a run with their
// outputs.
struct RunGraphs {
  cudaGraphExec_t chunk[2] = {nullptr, nullptr};
  cudaGraphExec_t rest[2] = {nullptr, nullptr};
  int rest_steps[2] = {0, 0};
  int rest_seen[2] = {0, 0};   // length of the last rest launched step by step
  int rest_times[2] = {0, 0};  // ... and how many times in a row
  bool ran = false;            // a run was issued
  cudaStream_t capture = nullptr;

  void drop_rest(int i) {
    if (rest[i]) cudaGraphExecDestroy(rest[i]);  // freed when its last launch is done
    rest[i] = nullptr;
    rest_steps[i] = rest_seen[i] = rest_times[i] = 0;
  }
  void drop_chunk(int i) {
    if (chunk[i]) cudaGraphExecDestroy(chunk[i]);
    chunk[i] = nullptr;
  }
  // forget the captured steps
  void drop() {
    for (int i = 0; i < 2; ++i) {
      drop_chunk(i);
      drop_rest(i);
    }
  }
};

// status of a launch; a refused one leaves no error behind for a later call
inline int launch_status(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return LBM_OK;
  cudaGetLastError();
  return set_error(e == cudaErrorMemoryAllocation ? LBM_ERR_OOM : LBM_ERR_CUDA,
                   "launch of %s failed: %s", what, cudaGetErrorString(e));
}

// Graph of what emit(stream) launches, or nullptr where a step of building it
// fails: a graph only saves launches, so the caller then launches one by one.
// A launch that fails leaves no graph, whether or not it broke the capture.
template <class Emit>
cudaGraphExec_t capture_graph(RunGraphs& g, Emit&& emit) {
  cudaGraphExec_t ex = nullptr;
  if (!g.capture && cudaStreamCreateWithFlags(&g.capture, cudaStreamNonBlocking) != cudaSuccess)
    g.capture = nullptr;
  if (g.capture &&
      cudaStreamBeginCapture(g.capture, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
    const cudaError_t le = emit(g.capture);
    cudaGraph_t graph = nullptr;
    const cudaError_t ee = cudaStreamEndCapture(g.capture, &graph);
    if (le == cudaSuccess && ee == cudaSuccess &&
        cudaGraphInstantiate(&ex, graph, 0) != cudaSuccess)
      ex = nullptr;
    if (graph) cudaGraphDestroy(graph);
  }
  if (!ex) cudaGetLastError();  // not the caller's error
  return ex;
}

// Issue n steps from the state (d->cur, d->step): step(stream, cur, k, left)
// launches step k from lattice cur (left: steps of the run still to come, 0 for
// its last one), finish(stream, cur, k) what follows the last step k.  d->cur and
// d->step advance with every launch that is accepted, so they say what the
// lattices hold also where a later one fails.
//
// Launched one by one a step costs the host 2 to 3 us, which is more than the
// GPU needs for a box below about 48^3 (or a third of a 64^3 one when several
// are stepped side by side), so the steps are launched as CUDA graphs, which
// cost one launch (even a single step: 16^3 FP32 pull, three side by side, one
// step a run 7.6 us -> 6.2, three steps 14.4 -> 6.5).  Building one costs as
// much as some 40 launches: the chunk is built for a run of at least kLongRun
// chunks or a domain that has run before, the rest once two runs from the same
// lattice have ended in rests of the same length (to replace one, once ten in
// a row have, none of them launched from the graph between), so that a single
// short run pays for neither.  Where a graph cannot be built or launched the
// steps are launched one by one, and so they are on a stream that is being
// captured (into that graph).
constexpr int kLongRun = 8;
constexpr int kRestFirst = 1, kRestReplace = 9;  // equal rests before a graph
template <class D, class Step, class Finish>
int issue_run(D* d, int n, Step&& step, Finish&& finish) {
  RunGraphs& g = d->graphs;
  const int full = n > 2 ? (n - 2) / kGraphSteps : 0, m = n - full * kGraphSteps;
  const int c0 = d->cur;  // a chunk has an even number of steps
  auto advance = [&](int i) {
    d->cur ^= i & 1;
    d->step += i;
    d->post_direct = false;
  };
  // launch a graph of i steps
  auto launch = [&](cudaGraphExec_t ex, int i) {
    if (!ex) return false;
    if (cudaGraphLaunch(ex, d->stream) == cudaSuccess) {
      advance(i);
      return true;
    }
    cudaGetLastError();
    return false;
  };
  auto loose = [&](int i, int left) {
    for (; i > 0; --i, --left) {
      if (const int rc = launch_status(step(d->stream, d->cur, d->step + 1, left - 1), "a step"))
        return rc;
      advance(1);
    }
    return static_cast<int>(LBM_OK);
  };
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  int rc = launch_status(cudaStreamIsCapturing(d->stream, &cs), "a run");
  if (rc) return rc;
  const bool graphs = cs == cudaStreamCaptureStatusNone;
  bool chunks = graphs && full > 0 && (full >= kLongRun || g.ran);
  if (chunks && !g.chunk[c0])
    g.chunk[c0] = capture_graph(g, [&](cudaStream_t st) {
      cudaError_t e = cudaSuccess;
      for (int i = 0; i < kGraphSteps && e == cudaSuccess; ++i)
        e = step(st, c0 ^ (i & 1), d->step + 1 + i, n - 1 - i);
      return e;
    });
  for (int i = 0; i < full; ++i) {
    if (chunks && !launch(g.chunk[c0], kGraphSteps)) {
      g.drop_chunk(c0);
      chunks = false;
    }
    if (!chunks && (rc = loose(kGraphSteps, n - i * kGraphSteps))) return rc;
  }
  bool rest = graphs && g.rest[c0] && g.rest_steps[c0] == m;
  if (graphs && !rest) {
    if (g.rest_seen[c0] == m && g.rest_times[c0] >= (g.rest[c0] ? kRestReplace : kRestFirst)) {
      g.drop_rest(c0);
      g.rest[c0] = capture_graph(g, [&](cudaStream_t st) {
        cudaError_t e = cudaSuccess;
        for (int i = 0; i < m && e == cudaSuccess; ++i)
          e = step(st, c0 ^ (i & 1), d->step + 1 + i, m - 1 - i);
        return e == cudaSuccess ? finish(st, c0 ^ (m & 1), d->step + m) : e;
      });
      g.rest_steps[c0] = m;
      rest = g.rest[c0] != nullptr;
    } else {
      g.rest_times[c0] = g.rest_seen[c0] == m ? g.rest_times[c0] + 1 : 1;
      g.rest_seen[c0] = m;
    }
  }
  g.ran = true;
  if (rest) {
    g.rest_times[c0] = 0;  // the loose rests before it are no longer in a row
    if (launch(g.rest[c0], m)) return LBM_OK;
    g.drop_rest(c0);
  }
  if ((rc = loose(m, m))) return rc;
  return launch_status(finish(d->stream, d->cur, d->step), "rho and u");
}

}  // namespace lbm
