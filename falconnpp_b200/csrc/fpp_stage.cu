// fpp_stage.cu — HostStage (fpp_stage.h).
#include "fpp_stage.h"

#include <string.h>

#include <algorithm>
#include <atomic>
#include <thread>

namespace fpp {

void HostStage::release() {
  for (auto& e : ev_)
    if (e) cudaEventDestroy(e);
  if (pin_) cudaFreeHost(pin_);
  *this = HostStage();
}

bool HostStage::ready() {
  if (pin_) return true;
  if (cudaHostAlloc(reinterpret_cast<void**>(&pin_), 2 * kThreads * kBuffer, cudaHostAllocDefault) != cudaSuccess) {
    pin_ = nullptr;
    cudaGetLastError();
    return false;
  }
  for (auto& e : ev_)
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      e = nullptr;
      cudaGetLastError();
      release();
      return false;
    }
  return true;
}

cudaError_t HostStage::copy(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  cudaPointerAttributes at;
  const bool known = cudaPointerGetAttributes(&at, src) == cudaSuccess;
  int dev = 0;
  const bool worth = bytes >= (seen_ ? kMinBytes : kFirstBytes);
  seen_ = seen_ || bytes >= kMinBytes;
  if (!worth || std::thread::hardware_concurrency() < kThreads || !known ||
      at.type != cudaMemoryTypeUnregistered || cudaGetDevice(&dev) != cudaSuccess || !ready()) {
    cudaGetLastError();
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
  }
  std::atomic<size_t> next{0};
  std::atomic<int> bad{(int)cudaSuccess};
  // pieces from a counter: whichever threads there are take all of them
  auto work = [&](int t) {
    cudaError_t e = cudaSetDevice(dev);
    for (int b = 0; e == cudaSuccess; b ^= 1) {
      const size_t at0 = next.fetch_add(kBuffer);
      if (at0 >= bytes) break;
      const size_t m = std::min(kBuffer, bytes - at0);
      unsigned char* p = pin_ + (size_t)(2 * t + b) * kBuffer;
      if ((e = cudaEventSynchronize(ev_[2 * t + b])) != cudaSuccess) break;
      memcpy(p, static_cast<const unsigned char*>(src) + at0, m);
      if ((e = cudaMemcpyAsync(static_cast<unsigned char*>(dst) + at0, p, m, cudaMemcpyHostToDevice, s)) != cudaSuccess)
        break;
      e = cudaEventRecord(ev_[2 * t + b], s);
    }
    if (e != cudaSuccess) bad.store((int)e);
  };
  std::thread th[kThreads - 1];
  for (int t = 1; t < kThreads; ++t) {
    try {
      th[t - 1] = std::thread(work, t);
    } catch (...) {  // no thread, or no memory for one
      break;         // the others take its pieces
    }
  }
  work(0);
  for (auto& x : th)
    if (x.joinable()) x.join();
  return (cudaError_t)bad.load();
}

}  // namespace fpp
