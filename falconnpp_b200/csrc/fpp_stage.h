// fpp_stage.h — pageable host data to the device through pinned buffers that
// several threads fill.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace fpp {

// The driver copies pageable memory through its own pinned buffers on one
// thread: 80 MB in 6.4 ms.  Four threads with two buffers of 512 KB each take
// 3.0 ms (two threads: 3.6, eight: 3.0; buffers of 1 MB: 2.1, but more to pin).
// Pinning these 4 MB takes 3 ms, once per handle: copies below 64 MB go to the
// driver, and so does a handle's first one below 128 MB (one build and no
// more would gain nothing).
class HostStage {
 public:
  static constexpr size_t kMinBytes = size_t(64) << 20;
  static constexpr size_t kFirstBytes = size_t(128) << 20;
  // Like cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s) for any
  // host memory; src has been read when it returns.  One caller at a time.
  cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t s);
  void release();

 private:
  static constexpr int kThreads = 4;
  static constexpr size_t kBuffer = size_t(512) << 10;
  bool ready();
  unsigned char* pin_ = nullptr;
  bool seen_ = false;  // a copy of kMinBytes before this one
  cudaEvent_t ev_[2 * kThreads] = {};  // the last copy out of each buffer
};

}  // namespace fpp
