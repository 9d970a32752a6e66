// Device-to-host copies of results into ordinary (pageable) memory.
//
// cudaMemcpy into pageable memory passes through the driver's staging buffer
// on one host thread, which also takes the page faults of freshly allocated
// arrays: 4 to 5 GB/s (the 63 MB of gradients of a 97x97x33 grid: 13 ms, with
// these threads 4).
// HostCopy gives a few threads a part of the array each; a thread streams its
// part through two pinned slots of its own, the bus copy of one chunk under
// the host copy of the other.  The slots (4 MB in all) belong to the object,
// are made on the first large copy and freed with it.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

class HostCopy {
  static constexpr int kThreads = 4;
  static constexpr size_t kSlot = 512 << 10;
  // below this the first copy of an object, which makes the slots and streams
  // (about 5 ms), would not pay for them
  static constexpr size_t kLeast = 32 << 20;
  char* pinned_ = nullptr;
  cudaStream_t s_[kThreads] = {};
  cudaEvent_t ready_ = nullptr, done_[kThreads][2] = {};
  bool made_ = false;

  bool make() {
    if (made_) return true;
    bool ok = cudaMallocHost(&pinned_, 2 * kThreads * kSlot) == cudaSuccess &&
              cudaEventCreateWithFlags(&ready_, cudaEventDisableTiming) == cudaSuccess;
    for (int w = 0; w < kThreads && ok; w++) {
      ok = cudaStreamCreateWithFlags(&s_[w], cudaStreamNonBlocking) == cudaSuccess;
      for (int k = 0; k < 2 && ok; k++)
        ok = cudaEventCreateWithFlags(&done_[w][k], cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) {
      cudaGetLastError();
      release();
    }
    return made_ = ok;
  }
  // thread w's part [at, end) through its two slots
  cudaError_t part(int w, char* dst, const char* src, size_t at, size_t end) {
    char* slot[2] = {pinned_ + 2 * w * kSlot, pinned_ + (2 * w + 1) * kSlot};
    size_t from[2] = {0, 0}, len[2] = {0, 0};
    cudaError_t e = cudaStreamWaitEvent(s_[w], ready_, 0);
    for (int k = 0; e == cudaSuccess && (at < end || len[0] || len[1]); k ^= 1) {
      if (len[k]) {  // the slot's chunk has been on its way since two rounds
        e = cudaEventSynchronize(done_[w][k]);
        if (e == cudaSuccess) std::memcpy(dst + from[k], slot[k], len[k]);
        len[k] = 0;
      }
      if (e == cudaSuccess && at < end) {
        from[k] = at;
        len[k] = std::min(kSlot, end - at);
        at += len[k];
        e = cudaMemcpyAsync(slot[k], src + from[k], len[k], cudaMemcpyDeviceToHost, s_[w]);
        if (e == cudaSuccess) e = cudaEventRecord(done_[w][k], s_[w]);
      }
    }
    if (e != cudaSuccess) cudaStreamSynchronize(s_[w]);  // nothing in flight into the slots after an error
    return e;
  }

 public:
  HostCopy() = default;
  HostCopy(const HostCopy&) = delete;
  HostCopy& operator=(const HostCopy&) = delete;
  ~HostCopy() { release(); }
  void release() {
    for (int w = 0; w < kThreads; w++) {
      if (s_[w]) cudaStreamDestroy(s_[w]);
      s_[w] = nullptr;
      for (int k = 0; k < 2; k++) {
        if (done_[w][k]) cudaEventDestroy(done_[w][k]);
        done_[w][k] = nullptr;
      }
    }
    if (ready_) cudaEventDestroy(ready_);
    ready_ = nullptr;
    if (pinned_) cudaFreeHost(pinned_);
    pinned_ = nullptr;
    made_ = false;
  }
  // dst (any memory) <- src (device), after the work already in `stream`.
  // Pinned, device and small destinations take the runtime's copy, which is
  // in `stream` and may still be under way at return; otherwise dst is
  // complete at return.  The slots, streams and events are made on src's device
  // and used there whichever is current (a null stream is the current one's and
  // takes the threads only where that is src's).
  cudaError_t copy(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    cudaPointerAttributes a, from;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    int current = 0;
    const bool plain = bytes >= kLeast && cudaPointerGetAttributes(&a, dst) == cudaSuccess &&
                       a.type == cudaMemoryTypeUnregistered &&
                       cudaStreamIsCapturing(stream, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone &&
                       cudaPointerGetAttributes(&from, src) == cudaSuccess && cudaGetDevice(&current) == cudaSuccess &&
                       (stream || from.device == current);
    const int dev = plain ? from.device : 0;
    const bool threaded = plain && cudaSetDevice(dev) == cudaSuccess && make();
    cudaGetLastError();
    const cudaError_t e = threaded ? by_threads(dst, src, bytes, stream, dev)
                                   : cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, stream);
    if (plain && current != dev) cudaSetDevice(current);
    return e;
  }

 private:
  cudaError_t by_threads(void* dst, const void* src, size_t bytes, cudaStream_t stream, int dev) {
    const cudaError_t e = cudaEventRecord(ready_, stream);
    if (e != cudaSuccess) return e;
    std::atomic<int> err{(int)cudaSuccess};
    // parts of whole pages, so that no two threads fault the same one
    const size_t per = ((bytes + kThreads - 1) / kThreads + 4095) / 4096 * 4096;
    auto run = [&](int w) {
      const size_t at = std::min(bytes, w * per), end = std::min(bytes, at + per);
      cudaError_t r = at < end ? cudaSetDevice(dev) : cudaSuccess;
      if (r == cudaSuccess && at < end) r = part(w, static_cast<char*>(dst), static_cast<const char*>(src), at, end);
      if (r != cudaSuccess) err = (int)r;
    };
    std::thread th[kThreads];
    for (int w = 1; w < kThreads; w++) {
      try {
        th[w] = std::thread(run, w);
      } catch (const std::system_error&) {
        run(w);  // no thread to be had: its part here
      }
    }
    run(0);
    for (int w = 1; w < kThreads; w++)
      if (th[w].joinable()) th[w].join();
    return (cudaError_t)err.load();
  }
};
