// The part of the CUDA runtime that lbm_issue.h calls, on the host: a stream
// runs what it is given at once, a stream in capture records it, a graph replays
// it.  fail_at[call] = n makes the n-th call of that kind fail (n < 0: it and
// all later ones).
#pragma once
#include <functional>
#include <set>
#include <vector>

enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone = 0, cudaStreamCaptureStatusActive = 1 };
enum cudaStreamCaptureMode { cudaStreamCaptureModeThreadLocal = 1 };
constexpr unsigned cudaStreamNonBlocking = 1;

namespace fake {
enum Call { kCreate, kBegin, kEnd, kInstantiate, kGraphLaunch, kIsCapturing, kKernel, kCalls };
using Work = std::vector<std::function<void()>>;
struct Stream {
  bool capturing = false, broken = false;
  Work recorded;
};
inline int fail_at[kCalls], calls[kCalls];
inline bool kernel_breaks_capture = false;
inline cudaError_t last = cudaSuccess;
inline std::set<const Work*> execs, graphs;  // alive

inline cudaError_t call(Call c) {
  const int n = ++calls[c], f = fail_at[c];
  if (f > 0 ? n == f : (f < 0 && n >= -f)) return last = cudaErrorMemoryAllocation;
  return cudaSuccess;
}
// a kernel launch
inline cudaError_t launch(Stream* s, std::function<void()> w) {
  const cudaError_t e = call(kKernel);
  if (e != cudaSuccess) {
    if (s->capturing && kernel_breaks_capture) s->broken = true;
    return e;
  }
  if (s->capturing)
    s->recorded.push_back(w);
  else
    w();
  return cudaSuccess;
}
}  // namespace fake

using cudaStream_t = fake::Stream*;
using cudaGraph_t = fake::Work*;
using cudaGraphExec_t = fake::Work*;

inline const char* cudaGetErrorString(cudaError_t) { return "injected"; }
inline cudaError_t cudaGetLastError() {
  const cudaError_t e = fake::last;
  fake::last = cudaSuccess;
  return e;
}
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  const cudaError_t e = fake::call(fake::kCreate);
  if (e == cudaSuccess) *s = new fake::Stream();
  return e;
}
inline cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
  *st = s->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return fake::call(fake::kIsCapturing);
}
inline cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  if (s->capturing) return fake::last = cudaErrorUnknown;
  const cudaError_t e = fake::call(fake::kBegin);
  if (e != cudaSuccess) return e;
  s->capturing = true;
  s->broken = false;
  s->recorded.clear();
  return cudaSuccess;
}
inline cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  if (!s->capturing) return fake::last = cudaErrorUnknown;
  s->capturing = false;
  *g = nullptr;
  const cudaError_t e = fake::call(fake::kEnd);
  if (e != cudaSuccess) return e;
  if (s->broken) return fake::last = cudaErrorUnknown;
  *g = new fake::Work(s->recorded);
  fake::graphs.insert(*g);
  return cudaSuccess;
}
inline cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
  const cudaError_t e = fake::call(fake::kInstantiate);
  if (e != cudaSuccess) return e;
  *x = new fake::Work(*g);
  fake::execs.insert(*x);
  return cudaSuccess;
}
inline cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  if (!fake::graphs.erase(g)) return fake::last = cudaErrorUnknown;
  delete g;
  return cudaSuccess;
}
inline cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  if (!fake::execs.erase(x)) return fake::last = cudaErrorUnknown;
  delete x;
  return cudaSuccess;
}
inline cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  if (!fake::execs.count(x)) return fake::last = cudaErrorUnknown;
  const cudaError_t e = fake::call(fake::kGraphLaunch);
  if (e != cudaSuccess) return e;
  for (auto& w : *x) {
    if (s->capturing)
      s->recorded.push_back(w);
    else
      w();
  }
  return cudaSuccess;
}
