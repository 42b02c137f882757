// call.h — the stream, events and device memory of one self-contained call
// (an auction, a quadratic solve, a demand map, the register clustering).
//
// Creating and destroying a stream and two events, and device memory that
// CUDA maps and unmaps, took 100 to 300 us of each call. Streams and events
// are kept for the next call, at most kKept of each device; memory comes from a
// pool of the device that keeps at most kKeptBytes between calls and gives
// back the rest. Any number of threads may call: each has its own stream.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace tgp {

class Call {
 public:
  explicit Call(int device);   // makes the device current
  ~Call();                     // the call's work is done: after finish(), or nothing was queued
  Call(const Call&) = delete;
  Call& operator=(const Call&) = delete;

  bool ok() const { return stream_ != nullptr; }
  cudaStream_t stream() const { return stream_; }
  char* memory(size_t bytes);  // once; nullptr when there is none
  void start() { cudaEventRecord(e0_, stream_); }
  // waits for the stream; `ms`: the device time since start()
  bool finish(float* ms);

 private:
  int device_;
  cudaStream_t stream_ = nullptr;
  cudaEvent_t e0_ = nullptr, e1_ = nullptr;
  char* base_ = nullptr;
  size_t bytes_ = 0;    // of the device's kept pool
  bool sound_ = true;   // no error seen: the stream may serve another call
};

}  // namespace tgp
