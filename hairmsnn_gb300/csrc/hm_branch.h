// Work on a second stream beside a stream's own.
#pragma once
#include <cuda_runtime_api.h>

namespace hm {

// What is enqueued on `side` after fork() comes after main's work up to there
// and runs beside main's later work; end() marks its end, join() makes main
// wait for that.  A branch that is left open, because something between the two
// returned early, is joined by the destructor: main's later work, which may use
// the branch's buffers again, never runs beside it.  side == main: nothing to
// do, the work is in order.
struct SideBranch {
  cudaStream_t main, side;
  cudaEvent_t forked, ended;
  bool open = false;

  SideBranch(cudaStream_t m, cudaStream_t s, cudaEvent_t f, cudaEvent_t e) : main(m), side(s), forked(f), ended(e) {}
  SideBranch(const SideBranch&) = delete;
  SideBranch& operator=(const SideBranch&) = delete;

  cudaError_t fork() {
    if (side == main) return cudaSuccess;
    cudaError_t e = cudaEventRecord(forked, main);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side, forked, 0);
    if (e == cudaSuccess) open = true;
    return e;
  }
  cudaError_t end() { return open ? cudaEventRecord(ended, side) : cudaSuccess; }
  cudaError_t join() {
    if (!open) return cudaSuccess;
    const cudaError_t e = cudaStreamWaitEvent(main, ended, 0);
    if (e == cudaSuccess) open = false;
    return e;
  }
  ~SideBranch() {
    if (!open) return;
    if (end() != cudaSuccess || join() != cudaSuccess) cudaStreamSynchronize(side);
  }
};

}  // namespace hm
