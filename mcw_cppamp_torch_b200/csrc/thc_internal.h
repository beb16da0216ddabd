// Shared internals of libTHC (B200): error plumbing, per-thread device context, launch helpers.
#ifndef THC_INTERNAL_H
#define THC_INTERNAL_H

#include <cuda_runtime.h>
#include <algorithm>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>

#include "THC.h"

namespace thc {

struct Error : std::runtime_error {
  using std::runtime_error::runtime_error;
};

struct OutOfMemory : Error {   // the device has no room for a request; nothing else is wrong
  using Error::Error;
};

[[noreturn]] void fail(const char *fmt, ...);
void record_error(const char *msg);  // thread-local message + user handler

#define THC_CHECK(cond, ...) \
  do { if (!(cond)) ::thc::fail(__VA_ARGS__); } while (0)
// Mirrors THArgCheck(condition, argNumber, msg) of TH.
#define THC_ARG(cond, argn, msg) \
  do { if (!(cond)) ::thc::fail("Invalid argument %d: %s", (argn), (msg)); } while (0)
#define THC_CUDA(expr) \
  do { cudaError_t e__ = (expr); if (e__ != cudaSuccess) \
    ::thc::fail("CUDA error %s at %s:%d: %s", cudaGetErrorName(e__), __FILE__, __LINE__, cudaGetErrorString(e__)); } while (0)

// Every extern "C" entry point body sits between these: C++ exceptions never cross the C ABI.
#define THC_BEGIN try {
#define THC_END(...) } catch (const std::exception &e__) { ::thc::record_error(e__.what()); return __VA_ARGS__; } \
                     catch (...) { ::thc::record_error("unknown error"); return __VA_ARGS__; }

// What the tensor-core kernels get to report a pipeline stall (a bounded mbarrier wait that ran out).
namespace mm {
struct StallCtl {
  int *dev_flag;     // device memory; a kernel that finds it set on entry does no work
  int *host_flag;    // mapped pinned host memory (device alias); the host reads it after a synchronisation
  long long limit;   // SM cycles one wait may take
};
}  // namespace mm

// Scalar results (sums, maxima, single elements) travel to the host through one mapped pinned record: the kernel
// writes the value, then the sequence number the host polls for (scalar_expect / scalar_wait).
struct ScalarSlot {
  double value;
  unsigned long long seq;
};

constexpr long kSmallStage = 16384;

struct Context {
  int device = -1;            // current device of this host thread, -1 = not yet initialised
  cudaStream_t stream = nullptr;
  bool owns_stream = false;
  int sm_count = 0;
  int math_mode = 0;          // 0 fp32x3, 1 simt, 2 bf16
  long launches = 0;
  long products[3] = {};      // launches of the two-SM engine by mm::kTf32, kBf16, kPairs
  // small device scratch reused by reductions and the GEMM error flag (lazy, per device)
  void *scratch = nullptr;
  size_t scratch_bytes = 0;
  ScalarSlot *scalar_slot = nullptr;      // mapped pinned host record
  ScalarSlot *scalar_slot_dev = nullptr;  // its device alias
  float *small_stage = nullptr;           // kSmallStage floats of mapped pinned memory behind small downloads
  float *small_stage_dev = nullptr;
  unsigned long long scalar_seq = 0;      // number of the last scalar asked for
  // stall flags of the tensor-core kernels (see mm::StallCtl)
  int *stall_host = nullptr;      // mapped pinned host word
  int *stall_host_dev = nullptr;  // its device alias
  int *stall_dev = nullptr;       // device word
  long long stall_limit = 1ll << 27;
  // workspace arena of the entry points' temporaries (see ws_alloc)
  char *ws_base = nullptr;
  size_t ws_cap = 0, ws_used = 0;
  int ws_depth = 0;
  long ws_epoch = 0;             // bumped whenever the arena is replaced by a larger one
  void *ws_retired[8] = {};      // arenas outgrown inside the running entry point, freed when it returns
  int ws_nretired = 0;
  long allocs = 0;               // stream-ordered allocations requested from the driver (storages + arena growth)
  // item counters of the persistent matrix-multiply launches (see sched_counter)
  unsigned *sched_counters = nullptr;
  int sched_next = 0, sched_block = 0, sched_recorded = 0;
  cudaStream_t sched_stream = nullptr;
  void *plane_records[64] = {};    // see plane_record()
  long plane_epoch = 0;            // bumped whenever they are given back
};

Context &ctx();                   // initialises device 0 on first use; fails loudly without CUDA
cudaStream_t stream();
// Waits for the stream, then turns a stall raised by any kernel since the last check into an Error (clearing it).
// Every entry point that hands results to the host synchronises through this.
void sync_stream();
void check_stall();               // the check alone, for callers that have just synchronised themselves
// The next scalar's sequence number, for a kernel that ends in scalar_deliver(ctx().scalar_slot_dev, value, number);
// scalar_wait returns the value once the number has arrived (or fails with the stream's error).  Everything queued
// on the stream before that kernel is then complete too, and a pipeline stall is reported as by sync_stream.
unsigned long long scalar_expect();
double scalar_wait(unsigned long long seq);
#ifdef __CUDACC__
__device__ __forceinline__ void scalar_deliver(ScalarSlot *slot, double v, unsigned long long seq) {
  volatile ScalarSlot *s = slot;
  s->value = v;
  __threadfence_system();
  s->seq = seq;
}
#endif
mm::StallCtl stall_ctl();         // kernel parameter of the tensor-core kernels
// A zeroed device word for one persistent launch to hand out its work items from.  The words come from two blocks of
// 4096; when one has been used up the other is cleared on the stream and takes over (the launches that used it are ahead of
// the clearing in the same stream).  Launches that are being recorded take theirs from a third block, where each is cleared
// by a node of the recording.  (Two recordings share it, as they share the workspace arena: they run one after the other.)
unsigned *sched_counter();
// The same for other uses inside one entry point, `n` words side by side on a 32-byte boundary; they keep their values until
// some thousand further words have been handed out.
unsigned *zeroed_words(int n);
int device_if_initialised();       // -1 before the first CUDA use on this thread; never initialises
void *scratch(size_t bytes);      // grow-only device scratch of the reductions, zero-filled when (re)allocated
// Records for planes that outlive an entry point (mm::KeptRange; which belongs to whom is the caller's), allocated 64 at a time.
constexpr int kPlaneRecords = 4096, kPlaneChunks = 64;
constexpr size_t kPlaneRecordBytes = 8224;
void *plane_record(int i);
// Device words that are zero between launches: tickets of kernels that put them back to zero when they are done.  One
// block for all of them, since the launches of a context run one after the other on its stream.
constexpr int kZeroWords = 16384;
unsigned *zero_words();
void *dev_alloc(size_t bytes);    // stream-ordered allocation (caching pool): storages
void dev_free(void *p);
// Temporaries of one entry-point call (operand planes, split-K partials, repacked weights ...) come from a
// per-context arena instead of the driver: ws_alloc bumps a pointer, and the WsScope the entry point opened
// gives everything back when it is left.  Work on the context's stream is ordered, so the next call may reuse
// the bytes while this call's kernels are still queued.  The arena grows (a larger one replaces it; the old one
// is freed in stream order once the entry point returns) until it fits the largest call, then no entry point
// asks the driver for memory at all.
void *ws_alloc(size_t bytes);
// Whether the next requests of this scope, `bytes` in all, can be had; for callers with a way that takes less.
bool ws_reserve(size_t bytes);
struct WsScope {
  size_t mark;
  long epoch;
  WsScope();
  ~WsScope();
  WsScope(const WsScope &) = delete;
  WsScope &operator=(const WsScope &) = delete;
};
inline void count_launch() { ctx().launches++; }
void check_launch(const char *what);  // cudaGetLastError -> fail

inline int ceil_div(long a, long b) { return (int)((a + b - 1) / b); }

// ---- tensor helpers shared by the math / nn files ----
long nelem(const THGPUTensor *t);
bool is_contiguous(const THGPUTensor *t);
inline float *data_ptr(const THGPUTensor *t) { return t->storage ? t->storage->data + t->storageOffset : nullptr; }
void resize_nd(THGPUTensor *t, int nd, const long *size, const long *stride /*nullable*/);
THGPUStorage *storage_new();
void storage_free(THGPUStorage *s);
void storage_resize(THGPUStorage *s, long size);
// points `self` at `storage` (retained; may be null) with the given view; null size / stride keep / derive them
void tensor_raw_set(THGPUTensor *self, THGPUStorage *storage, long offset, int nd, const long *size, const long *stride);
// throwing internals behind the C ABI of the same names
THGPUTensor *tensor_new();
void tensor_free(THGPUTensor *t);
void tensor_copy(THGPUTensor *dst, THGPUTensor *src);
THGPUTensor *tensor_new_contiguous(THGPUTensor *t);   // retains t when it already is contiguous
THGPUTensor *tensor_new_sized(int nd, const long *size);
void tensor_resize_as(THGPUTensor *r, const THGPUTensor *t);
// Whether the memory from a tensor's first element to its last meets another's.  By address: two storages may borrow the same
// memory (THGPUStorage_newWithData).
bool overlap(const THGPUTensor *a, const THGPUTensor *b);

// Scope guard: one reference to a tensor, released when the scope is left by any route, so that a THC_CHECK that
// throws between THC_BEGIN and THC_END does not leak it.
struct TensorRef {
  THGPUTensor *t;
  explicit TensorRef(THGPUTensor *t_ = nullptr) : t(t_) {}
  TensorRef(const TensorRef &) = delete;
  TensorRef &operator=(const TensorRef &) = delete;
  ~TensorRef() { if (t) tensor_free(t); }
  void reset(THGPUTensor *t_ = nullptr) { if (t) tensor_free(t); t = t_; }
  operator THGPUTensor *() const { return t; }
  THGPUTensor *operator->() const { return t; }
};

// Collapsed strided description of up to 4 operands over one index space (used by the generic
// elementwise / copy kernels).  dims are merged wherever every operand allows it.
constexpr int kMaxDims = 8;
struct Strided {
  int nd;
  long size[kMaxDims];
  long stride[4][kMaxDims];
};
// Builds the description for operands that all have nelem equal; returns false if more than
// kMaxDims dims remain after collapsing.
bool collapse(int nops, const THGPUTensor *const *ops, Strided &out);

// SGD (with momentum when v is given) over flat buffers on an explicit stream
void sgd_update_async(float *w, const float *g, float *v, long n, float lr, float momentum, cudaStream_t s);

// device-side GEMM front (col-major BLAS semantics) shared by addmm / conv / Linear
void gemm(char transa, char transb, long m, long n, long k, float alpha, const float *a, long lda,
          const float *b, long ldb, float beta, float *c, long ldc, const float *row_bias = nullptr);   // bias[i] added to row i (beta 0)

#ifdef __CUDACC__
// Kernels of a stream follow one another as programmatic dependents: a kernel's blocks may take their places, and set up what is
// theirs alone, while the previous kernel drains, and wait in pdl_wait() for its results.  Every kernel launched this way
// executes the wait, which is what keeps the order transitive.  Worth about 1.5 us a launch (a step of 100 launches at 128
// images: 4.10 -> 4.02 ms).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() { pdl_wait(); pdl_trigger(); }
// `early` false: the ordinary order, the whole device free before the first block starts.
template <class... P, class... A>
void launch_on_stream(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A &&...args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream();
  cfg.attrs = &attr; cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);   // check_launch() picks an error up
}
template <class... P, class... A>
void pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A &&...args) {
  launch_on_stream(true, kernel, grid, block, smem, args...);
}
#endif

}  // namespace thc

#endif
