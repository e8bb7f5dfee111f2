// A second stream beside a time loop's own, for a kernel of a step that does
// not depend on the step's next kernel: fork() lets it start behind everything
// the main stream holds, join() keeps the main stream's next work behind it.
// Used in captured loops only, where it is a branch of the graph (a caller's
// own capture included): as direct launches the four event calls per step cost
// the host more than the overlap gives (first gradient of one shot of 333 x
// 217: 14.6 ms with, 13.7 without; replayed: 9.9 against 10.8).  One per
// simulation object, made with it, so that neither
// other objects nor other threads meet it; every loop joins before it ends.
#pragma once

#include <cuda_runtime.h>

#include "internal.h"

namespace swgb {

struct SideStream {
  cudaStream_t s = nullptr;
  cudaEvent_t there = nullptr, back = nullptr;
  bool open = false;  // work forked and not joined yet

  SideStream() = default;
  SideStream(const SideStream&) = delete;
  SideStream& operator=(const SideStream&) = delete;
  ~SideStream() {
    if (s) cudaStreamDestroy(s);
    if (there) cudaEventDestroy(there);
    if (back) cudaEventDestroy(back);
  }
  void create() {
    check_cuda(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "side stream");
    check_cuda(cudaEventCreateWithFlags(&there, cudaEventDisableTiming), "side stream event");
    check_cuda(cudaEventCreateWithFlags(&back, cudaEventDisableTiming), "side stream event");
  }
  static bool captured(cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    check_cuda(cudaStreamIsCapturing(st, &cs), "cudaStreamIsCapturing");
    return cs == cudaStreamCaptureStatusActive;
  }
  // the stream for the forked launch, ordered behind st's work so far
  cudaStream_t fork(cudaStream_t st) {
    check_cuda(cudaEventRecord(there, st), "side stream fork");
    check_cuda(cudaStreamWaitEvent(s, there, 0), "side stream fork");
    return s;
  }
  void forked() {
    check_cuda(cudaEventRecord(back, s), "side stream record");
    open = true;
  }
  void join(cudaStream_t st) {
    if (!open) return;
    check_cuda(cudaStreamWaitEvent(st, back, 0), "side stream join");
    open = false;
  }
};

}  // namespace swgb
