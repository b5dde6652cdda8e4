// libcm_fe: the order of work that uses a handle's buffers on several streams
// (host code).  Both classes keep their promise on every way out of a scope,
// error returns included: where an event cannot order the streams, the host
// waits for the work instead.
#pragma once

#include <cuda_runtime.h>

namespace cmfe {

// Uses of one set of buffers, on whatever streams, in call order: begin()
// makes the stream wait for the previous use, the destructor marks the end of
// what was queued since.
class HandleOrder {
 public:
  explicit HandleOrder(cudaStream_t st) : st_(st) {}
  HandleOrder(const HandleOrder&) = delete;
  // *ev is created on first use; the work must not be queued when this fails.
  cudaError_t begin(cudaEvent_t* ev) {
    cudaError_t e = cudaSuccess;
    if (!*ev) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st_, *ev, 0);
    if (e == cudaSuccess) ev_ = *ev;
    return e;
  }
  ~HandleOrder() {
    if (ev_ && cudaEventRecord(ev_, st_) != cudaSuccess) {
      cudaGetLastError();
      cudaStreamSynchronize(st_);
    }
  }

 private:
  cudaStream_t st_;
  cudaEvent_t ev_ = nullptr;
};

// Streams forked from st, at most MOST; st follows the work queued on them when
// the scope ends.  No allocation, so nothing here throws.
class Fork {
 public:
  static constexpr int MOST = 8;
  explicit Fork(cudaStream_t st) : st_(st) {}
  Fork(const Fork&) = delete;
  // side continues from the event `from` of st; `done` will mark its end.
  cudaError_t add(cudaStream_t side, cudaEvent_t from, cudaEvent_t done) {
    if (n_ == MOST) return cudaErrorInvalidValue;
    const cudaError_t e = cudaStreamWaitEvent(side, from, 0);
    if (e == cudaSuccess) sides_[n_++] = {side, done};
    return e;
  }
  ~Fork() {
    for (int i = 0; i < n_; ++i) {
      const Side& s = sides_[i];
      if (cudaEventRecord(s.done, s.stream) != cudaSuccess || cudaStreamWaitEvent(st_, s.done, 0) != cudaSuccess) {
        cudaGetLastError();
        cudaStreamSynchronize(s.stream);
      }
    }
  }

 private:
  struct Side {
    cudaStream_t stream;
    cudaEvent_t done;
  };
  cudaStream_t st_;
  int n_ = 0;
  Side sides_[MOST];
};

}  // namespace cmfe
