// Runs of a domain over a host stand-in for the CUDA runtime.
//   driver CALL N BREAKS RUN...   one call of kind CALL fails, the N-th (N < 0:
//                                 it and all later ones; 0: none); BREAKS: a
//                                 kernel that fails in capture breaks it
// A run whose launches are refused returns an error.  Otherwise every step has
// to be done, with its side outputs; in either case the domain's step and
// lattice have to say what was done.  Prints "runs failed=F graphs=G" and exits
// 1 with the reason where that does not hold.
#include "lbm_issue.h"

#include <cstdarg>
#include <cstdio>
#include <cstdlib>

namespace lbm {
int set_error(int code, const char*, ...) { return code; }
void clear_error() {}
}  // namespace lbm

struct Domain {
  lbm::RunGraphs graphs;
  int cur = 0;
  long long step = 0;
  bool post_direct = false;
  cudaStream_t stream = nullptr;
};

// what the lattices went through
struct Device {
  long long done = 0, fields = 0, finished = 0;
  int cur = 0;
  bool order = true;
} dev;

int main(int argc, char** argv) {
  if (argc < 5) return 2;
  fake::fail_at[atoi(argv[1])] = atoi(argv[2]);
  fake::kernel_breaks_capture = atoi(argv[3]);
  fake::Stream own;
  Domain d;
  d.stream = &own;
  int failed = 0;
  for (int i = 4; i < argc; ++i) {
    const long long before = d.step;
    const int n = atoi(argv[i]);
    const int rc = lbm::issue_run(
        &d, n,
        [&](cudaStream_t st, int cur, long long k, int left) {
          const int par = (int)(k & 1);
          return fake::launch(st, [=] {
            dev.order = dev.order && cur == dev.cur && par == ((dev.done + 1) & 1);
            dev.cur ^= 1;
            ++dev.done;
            if (left == 0) dev.fields = dev.done;
          });
        },
        [&](cudaStream_t st, int cur, long long) {
          return fake::launch(st, [=] {
            dev.order = dev.order && cur == dev.cur;
            dev.finished = dev.done;
          });
        });
    const char* why = nullptr;
    if (!dev.order) why = "a step from the wrong lattice";
    if (dev.done != d.step || dev.cur != d.cur) why = "step or lattice is not what was done";
    if (fake::last != cudaSuccess) why = "an error left for a later call";
    if (fake::execs.size() > 4 || !fake::graphs.empty()) why = "graphs left over";
    if (rc == LBM_OK && d.step != before + n) why = "steps missing";
    if (rc == LBM_OK && (dev.fields != dev.done || dev.finished != dev.done))
      why = "side outputs missing";
    failed += rc != LBM_OK;
    if (why) {
      std::printf("run %d (%d steps, rc %d): %s\n", i - 4, n, rc, why);
      return 1;
    }
  }
  std::printf("runs failed=%d graphs=%d\n", failed, fake::calls[fake::kInstantiate]);
  d.graphs.drop();
  return fake::execs.empty() ? 0 : 1;
}
