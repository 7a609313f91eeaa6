// ih_fork.cuh -- a second stream for part of a sequence of launches.
#pragma once
#include <cuda_runtime.h>

namespace ih {

// Work on `side` beside `main` from start() on.  Whatever way the scope is left -- a
// failed launch in between included -- main comes after the work on side, so that a
// caller who synchronises main, or runs the next call on it, does not meet that
// work still running.
class Fork {
 public:
  // side comes after what main holds now (event `begin`)
  cudaError_t start(cudaStream_t main, cudaStream_t side, cudaEvent_t begin, cudaEvent_t end) {
    cudaError_t e = cudaEventRecord(begin, main);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side, begin, 0);
    if (e != cudaSuccess) return e;
    main_ = main;
    side_ = side;
    end_ = end;
    open_ = true;
    return cudaSuccess;
  }
  // main comes after all of side; nothing where nothing was started
  cudaError_t join() {
    if (!open_) return cudaSuccess;
    open_ = false;
    cudaError_t e = cudaEventRecord(end_, side_);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(main_, end_, 0);
    return e;
  }
  ~Fork() { join(); }
  Fork() = default;
  Fork(const Fork &) = delete;
  Fork &operator=(const Fork &) = delete;

 private:
  cudaStream_t main_ = nullptr, side_ = nullptr;
  cudaEvent_t end_ = nullptr;
  bool open_ = false;
};

}  // namespace ih
