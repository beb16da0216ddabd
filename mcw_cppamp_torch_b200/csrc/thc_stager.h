// Uploads from pageable memory.  The driver stages those through its own pinned buffers with one thread, 18 GB/s where the
// bus takes 55: a third of the time of a batch of images on its way through a classifier.  Here the caller and a second
// thread copy pieces into pinned slots and queue each piece as soon as it is there (67 MB: 4.4 - 5.6 -> 2.9 ms; the
// AlexNet-style classifier over 128 host images 7.3 - 8.1 -> 5.3 - 5.8 ms, the VGG-A-style one over 24 3.45 -> 3.3; four or
// eight threads were no steadier).  One process-wide set of threads and slots (kStagers * 2 * kPiece bytes), made at the
// first large upload and kept; a caller that finds it busy takes the driver's way.
//
// Needs the CUDA runtime only (the tests run it on the host over a stand-in for it).
#ifndef THC_STAGER_H
#define THC_STAGER_H

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>

namespace thc {

constexpr long kPiece = 512 * 1024;
constexpr int kStagers = 2;
constexpr long kStageFrom = 16 * kPiece;   // 4 - 8 MB measured the same either way: waking the thread costs what it saves
class Stager {
 public:
  static Stager &get() {
    static Stager *s = new Stager();   // never destroyed: its threads outlive every caller
    return *s;
  }
  // False: nothing was queued.  True: everything was, unless `err` says what went wrong.  `device` is the current one.
  bool upload(void *dst, const void *src, long bytes, int device, cudaStream_t stream, cudaError_t &err) {
    std::unique_lock<std::mutex> one(busy_, std::try_to_lock);
    if (!one.owns_lock() || !ready(device)) return false;
    dst_ = (char *)dst; src_ = (const char *)src; bytes_ = bytes; stream_ = stream; next_ = 0; error_ = cudaSuccess;
    const long helpers = std::min<long>(kStagers - 1, bytes / kPiece - 1);
    {
      std::lock_guard<std::mutex> l(m_);
      wanted_ = (int)helpers; working_ = 0; job_++;
    }
    cv_.notify_all();
    work(0);
    {
      std::unique_lock<std::mutex> l(m_);
      wanted_ = 0;   // who has not started yet need not
      done_.wait(l, [&] { return working_ == 0; });
    }
    err = (cudaError_t)error_.load();
    return true;
  }

 private:
  struct Slot { char *p[2] = {}; cudaEvent_t free[2] = {}; };
  // threads once, slots and events for the device last used
  bool ready(int device) {
    try {
      for (; threads_ < kStagers - 1; threads_++) std::thread([this, i = threads_ + 1] { loop(i); }).detach();
    } catch (const std::system_error &) {
      return false;   // the process may not have another thread now; the next upload asks again
    }
    if (device == device_) return true;
    device_ = -1;   // until every slot has its event: a failure half-way leaves no device whose events are gone
    for (Slot &s : slots_)
      for (int k = 0; k < 2; k++) {
        // upload() returns with its last pieces still on their way: the pinned slot is this device's once they have left
        if (s.free[k] && cudaEventSynchronize(s.free[k]) != cudaSuccess) { cudaGetLastError(); return false; }
        if (s.free[k]) { cudaEventDestroy(s.free[k]); s.free[k] = nullptr; }
        if (!s.p[k] && cudaHostAlloc((void **)&s.p[k], kPiece, cudaHostAllocPortable) != cudaSuccess) { cudaGetLastError(); return false; }
        if (cudaEventCreateWithFlags(&s.free[k], cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); return false; }
      }
    device_ = device;
    return true;
  }
  void work(int who) {
    Slot &s = slots_[who];
    for (int k = 0;; k ^= 1) {
      const long at = next_.fetch_add(kPiece);
      if (at >= bytes_ || error_ != cudaSuccess) break;
      const long n = std::min(kPiece, bytes_ - at);
      cudaError_t e = cudaEventSynchronize(s.free[k]);   // the slot's last piece has left
      std::memcpy(s.p[k], src_ + at, n);
      if (e == cudaSuccess) e = cudaMemcpyAsync(dst_ + at, s.p[k], n, cudaMemcpyHostToDevice, stream_);
      if (e == cudaSuccess) e = cudaEventRecord(s.free[k], stream_);
      if (e != cudaSuccess) { error_ = e; break; }
    }
  }
  void loop(int who) {
    long seen = 0;
    int device = -1;
    for (;;) {
      {
        std::unique_lock<std::mutex> l(m_);
        cv_.wait(l, [&] { return job_ != seen; });
        seen = job_;
        if (wanted_ <= 0) continue;
        wanted_--;
        working_++;
      }
      if (device != device_) { cudaSetDevice(device_); device = device_; }
      work(who);
      std::lock_guard<std::mutex> l(m_);
      if (--working_ == 0) done_.notify_all();
    }
  }
  std::mutex busy_, m_;
  std::condition_variable cv_, done_;
  int threads_ = 0;   // helpers started
  int device_ = -1, wanted_ = 0, working_ = 0;
  long job_ = 0, bytes_ = 0;
  char *dst_ = nullptr;
  const char *src_ = nullptr;
  cudaStream_t stream_ = nullptr;
  std::atomic<long> next_{0};
  std::atomic<int> error_{cudaSuccess};
  Slot slots_[kStagers];
};

}  // namespace thc

#endif
