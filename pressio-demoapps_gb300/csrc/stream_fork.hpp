// A second stream's share of a call's work: it starts behind what the first
// stream has been given and is joined to that stream when the call ends,
// whichever way it ends.  A call that fails between the two would otherwise
// return while the second stream still writes buffers that its caller reuses
// or frees on the first.
#pragma once

#include <string>

#include <cuda_runtime_api.h>

#include "internal.hpp"

namespace pda {

class StreamFork {
 public:
  StreamFork(cudaStream_t main, cudaStream_t side, cudaEvent_t forkEvent, cudaEvent_t joinEvent)
      : main_(main), side_(side), join_(joinEvent) {
    check(cudaEventRecord(forkEvent, main_), "stream fork");
    check(cudaStreamWaitEvent(side_, forkEvent, 0), "stream fork");
  }
  StreamFork(const StreamFork &) = delete;
  StreamFork &operator=(const StreamFork &) = delete;
  cudaStream_t side() const { return side_; }
  // the first stream waits for the second's work so far
  void join() {
    open_ = false;
    const cudaError_t e = order();
    if (e != cudaSuccess) {
      cudaStreamSynchronize(side_);
      check(e, "stream join");
    }
  }
  // an exception on its way out
  ~StreamFork() {
    if (open_ && order() != cudaSuccess) cudaStreamSynchronize(side_);
  }

 private:
  static void check(cudaError_t e, const char *what) {
    if (e != cudaSuccess) throw Error(PDA_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  }
  cudaError_t order() {
    const cudaError_t e = cudaEventRecord(join_, side_);
    return e != cudaSuccess ? e : cudaStreamWaitEvent(main_, join_, 0);
  }
  cudaStream_t main_, side_;
  cudaEvent_t join_;
  bool open_ = true;
};

}  // namespace pda
