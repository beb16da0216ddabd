// Staged uploads over the stand-in runtime: one scenario per argument, exit code 0 when the bytes arrived.
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "thc_stager.h"

#include <cerrno>
#include <dlfcn.h>
#include <pthread.h>

using thc::Stager;

// Takes the place of the C library's for the whole program, std::thread included.
static bool no_threads = false;
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x) noexcept {
  if (no_threads) return EAGAIN;
  return ((int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *))dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, x);
}

struct Upload {
  std::vector<char> src, dst;
  FakeStream *stream = new FakeStream;   // outlives the upload, as the stager's events may
  bool taken = false;
  cudaError_t err = cudaSuccess;
  Upload(long bytes, int seed) : src(bytes), dst(bytes, 0) { for (long i = 0; i < bytes; i++) src[i] = (char)(i * 31 + i / 4096 + seed * 7 + 1); }
  void run(int device) { taken = Stager::get().upload(dst.data(), src.data(), (long)src.size(), device, stream, err); }
  bool arrived() { cudaStreamSynchronize(stream); return taken && err == cudaSuccess && std::memcmp(src.data(), dst.data(), src.size()) == 0; }
};

int main(int, char **argv) {
  const std::string what = argv[1];
  const long n = 17 * thc::kPiece + 12345;
  if (what == "devices") {   // the last pieces for device 0 are still in flight when an upload to device 1 begins
    for (int round = 0; round < 8; round++) {
      Upload a(n, 2 * round), b(n, 2 * round + 1);
      a.run(0);
      b.run(1);
      if (!a.arrived() || !b.arrived()) { std::printf("round %d: device 0 %d, device 1 %d\n", round, a.arrived(), b.arrived()); return 1; }
    }
    return 0;
  }
  if (what == "event") {   // an event of the new device cannot be made: the driver's way this time, and no trace of it later
    for (int fail = 1; fail <= 4; fail++) {
      Upload a(n, 1), b(n, 2), c(n, 3), d(n, 4);
      a.run(0);
      fake_fail_event_create() = fail;
      b.run(1);
      fake_fail_event_create() = 0;
      c.run(0);
      d.run(1);
      if (!a.arrived() || b.taken || !c.arrived() || !d.arrived()) {
        std::printf("creation %d: %d %d %d (error %d) %d\n", fail, a.arrived(), b.taken, c.arrived(), (int)c.err, d.arrived());
        return 1;
      }
    }
    return 0;
  }
  if (what == "thread") {   // no thread to be had: the driver's way, until there is one
    Upload a(n, 1), b(n, 2);
    no_threads = true;
    a.run(0);
    no_threads = false;
    b.run(0);
    return !a.taken && b.arrived() ? 0 : 1;
  }
  return 2;
}
