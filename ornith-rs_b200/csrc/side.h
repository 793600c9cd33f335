// Work beside the main chain of a call, on the context's side stream: forked behind a point of the main stream and
// joined before whatever needs it.  Every way out of the scope joins, an error's too: what follows on the main stream
// (the next call, which writes the same buffers, and orn_sync) waits for all that the side stream was given.
#pragma once

#include <cuda_runtime_api.h>

class SideWork {
 public:
  // side null: there is no second stream, and everything goes to `main`
  SideWork(cudaStream_t main, cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) : main_(main), side_(side), fork_(fork), join_(join) {}
  SideWork(const SideWork&) = delete;
  SideWork& operator=(const SideWork&) = delete;
  ~SideWork() {
    if (!open_ || (cudaEventRecord(join_, side_) == cudaSuccess && cudaStreamWaitEvent(main_, join_, 0) == cudaSuccess)) return;
    cudaStreamSynchronize(side_);
    cudaGetLastError();  // the caller has its error already
  }
  bool two() const { return side_ != nullptr; }
  bool open() const { return open_; }  // the side stream may have been given work
  cudaStream_t stream() const { return side_ != nullptr ? side_ : main_; }
  // the point of the main stream that the work may start behind
  cudaError_t mark() { return two() ? cudaEventRecord(fork_, main_) : cudaSuccess; }
  // the side stream waits for that point: launches on stream() from here on
  cudaError_t start() {
    if (!two() || open_) return cudaSuccess;
    open_ = true;
    return cudaStreamWaitEvent(side_, fork_, 0);
  }
  // the last of the work has been launched
  cudaError_t done() { return open_ ? cudaEventRecord(join_, side_) : cudaSuccess; }
  // the main stream waits for what done() closed
  cudaError_t join() {
    if (!open_) return cudaSuccess;
    const cudaError_t e = cudaStreamWaitEvent(main_, join_, 0);
    if (e == cudaSuccess) open_ = false;
    return e;
  }

 private:
  cudaStream_t main_, side_;
  cudaEvent_t fork_, join_;
  bool open_ = false;
};
