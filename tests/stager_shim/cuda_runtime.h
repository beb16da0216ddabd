/* The few runtime calls of thc_stager.h on the host.  A stream is a queue of copies that run only when an event behind them or the
 * stream itself is waited for, i.e. as late as real ones may. */
#ifndef FAKE_CUDA_RUNTIME_H
#define FAKE_CUDA_RUNTIME_H

#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <mutex>

enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorInvalidResourceHandle = 400 };
enum { cudaMemcpyHostToDevice = 1, cudaHostAllocPortable = 1, cudaEventDisableTiming = 2 };

struct FakeCopy { void *dst; const void *src; size_t n; };
struct FakeStream { std::deque<FakeCopy> queue; long done = 0, queued = 0; };
struct FakeEvent { FakeStream *stream; long upto; };
typedef FakeStream *cudaStream_t;
typedef FakeEvent *cudaEvent_t;

inline std::mutex &fake_mutex() { static std::mutex m; return m; }
inline int &fake_fail_event_create() { static int n = 0; return n; }   // n > 0: the n-th creation from now on fails

inline void fake_run(FakeStream *s, long upto) {
  while (s->done < upto) {
    const FakeCopy c = s->queue.front();
    s->queue.pop_front();
    std::memcpy(c.dst, c.src, c.n);
    s->done++;
  }
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) { std::lock_guard<std::mutex> l(fake_mutex()); fake_run(s, s->queued); return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, int, cudaStream_t s) {
  std::lock_guard<std::mutex> l(fake_mutex());
  s->queue.push_back({dst, src, n});
  s->queued++;
  return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, int) {
  std::lock_guard<std::mutex> l(fake_mutex());
  if (fake_fail_event_create() > 0 && --fake_fail_event_create() == 0) return cudaErrorMemoryAllocation;
  *e = new FakeEvent{nullptr, 0};
  return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }   // returns at once, as the real one does
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::mutex> l(fake_mutex());
  if (!e) return cudaErrorInvalidResourceHandle;
  e->stream = s; e->upto = s->queued;
  return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  std::lock_guard<std::mutex> l(fake_mutex());
  if (!e) return cudaErrorInvalidResourceHandle;
  if (e->stream) fake_run(e->stream, e->upto);   // never recorded: complete
  return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void **p, size_t n, int) { *p = std::malloc(n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }

#endif
