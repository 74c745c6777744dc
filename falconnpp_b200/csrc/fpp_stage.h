// fpp_stage.h — pageable host data to the device through pinned buffers that
// several threads fill.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace fpp {

// The driver copies pageable memory through its own pinned buffers on one
// thread: 80 MB in 6.4 ms.  Four threads with two buffers of 512 KB each take
// 3.0 ms (two threads: 3.6, eight: 3.0; buffers of 1 MB: 2.1, but more to pin).
// Pinning these 4 MB takes 3 ms and more, once per handle, which a copy of about
// 70 MB gains back: a handle that has not copied that much before pins from 128
// MB on (one build of less would gain nothing, and does not), one that has, and
// so builds again and again, from 64 MB on.
class HostStage {
 public:
  static constexpr size_t kMinBytes = size_t(64) << 20;
  static constexpr size_t kFirstBytes = size_t(128) << 20;
  // Like cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s) for any
  // host memory: pageable memory has been read when it returns, pinned memory
  // is read in the stream's order.  One caller at a time.
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
