// Full reductions of torch.GPUTensor to one host scalar: sum / max / min / dot and the whole-tensor norms.
//
// One launch reads every element once.  Each block reduces a grid-strided slice (fp32 runs of 4 folded into a double
// accumulator per thread) and writes one partial; the last block to finish (atomic ticket) folds the partials in fixed
// order, so the result is deterministic and no block ever waits on another.  Tensors that one block finishes in a few
// loads skip the ticket.  The value goes straight to mapped pinned host memory, followed by a sequence number the host
// polls: a kernel that has delivered its number is the last thing the caller waits for, so neither a device-to-host
// copy nor a stream synchronisation follows (they cost three times the kernel on small tensors).
//
// The norms' terms (squares, powers, centred squares ...) are functors evaluated on the way, rounded to float as the CPU
// does, instead of a pass that writes them to a temporary of the tensor's size.
#ifndef THC_REDUCE_CUH
#define THC_REDUCE_CUH

#include "thc_apply.cuh"

namespace thc {

enum { RED_SUM = 0, RED_MAX = 1, RED_MIN = 2, RED_DOT = 3 };

struct RedScratch {
  double partial[1024];
  unsigned int ticket;
  unsigned int pad;
};

template <int MODE> struct RedTraits;
template <> struct RedTraits<RED_SUM> {
  __device__ static double init(float) { return 0.0; }
  __device__ static double fold4(float4 v) { return (double)((v.x + v.y) + (v.z + v.w)); }
  __device__ static double one(float v) { return (double)v; }
  __device__ static double comb(double a, double b) { return a + b; }
};
template <> struct RedTraits<RED_MAX> {
  __device__ static double init(float first) { return (double)first; }
  __device__ static double fold4(float4 v) { return (double)fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); }
  __device__ static double one(float v) { return (double)v; }
  __device__ static double comb(double a, double b) { return a > b ? a : b; }
};
template <> struct RedTraits<RED_MIN> {
  __device__ static double init(float first) { return (double)first; }
  __device__ static double fold4(float4 v) { return (double)fminf(fminf(v.x, v.y), fminf(v.z, v.w)); }
  __device__ static double one(float v) { return (double)v; }
  __device__ static double comb(double a, double b) { return a < b ? a : b; }
};

// The element itself: the term of sum / max / min.
struct IdTerm {
  static constexpr int NIN = 1;
  __device__ float operator()(const float *a) const { return a[0]; }
};

template <int MODE>
__device__ __forceinline__ double block_reduce(double v, double *smem) {
  typedef RedTraits<MODE> T;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = T::comb(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  if (warp == 0) {
    // lanes beyond the warp count re-use entry 0 for max/min (idempotent) and contribute 0 to sums
    v = lane < nwarps ? smem[lane] : (MODE == RED_SUM ? 0.0 : smem[0]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = T::comb(v, __shfl_xor_sync(0xffffffffu, v, o));
  }
  __syncthreads();
  return v;  // valid in warp 0
}

template <int MODE, class Term>
__global__ void __launch_bounds__(512) reduce_all_kernel(const float *__restrict__ x, const float *__restrict__ y, long n, bool vec,
                                                         RedScratch *s, Term term, ScalarSlot *slot, unsigned long long seq) {
  pdl_begin();
  constexpr bool DOT = MODE == RED_DOT;
  constexpr int BASE = DOT ? RED_SUM : MODE;
  constexpr int NIN = DOT ? 2 : Term::NIN;
  typedef RedTraits<BASE> T;
  __shared__ double smem[32];
  __shared__ bool is_last;
  const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x, nthreads = (long)gridDim.x * blockDim.x;
  auto one = [&](float a, float b) -> float {
    const float in[2] = {a, b};
    return term(in);
  };
  auto four = [&](const float4 &v, const float4 &w) -> double {
    // products are exact in double; keeps the dot product faithful to a double accumulator
    if (DOT) return (double)v.x * w.x + (double)v.y * w.y + (double)v.z * w.z + (double)v.w * w.w;
    return T::fold4(make_float4(one(v.x, w.x), one(v.y, w.y), one(v.z, w.z), one(v.w, w.w)));
  };
  double acc = T::init(x[0]);
  long done = 0;
  if (vec) {
    const long nvec = n >> 2;
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    const float4 *y4 = reinterpret_cast<const float4 *>(y);
    long i = tid;
    constexpr int U = NIN == 1 ? 4 : 2;   // four independent 16-byte loads per thread in flight
    for (; i + (U - 1) * nthreads < nvec; i += U * nthreads) {
      float4 v[U], w[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        v[u] = x4[i + u * nthreads];
        w[u] = NIN == 2 ? y4[i + u * nthreads] : v[u];
      }
#pragma unroll
      for (int u = 0; u < U; u += 2) acc = T::comb(acc, T::comb(four(v[u], w[u]), four(v[u + 1], w[u + 1])));
    }
    for (; i < nvec; i += nthreads) {
      const float4 v = x4[i];
      acc = T::comb(acc, four(v, NIN == 2 ? y4[i] : v));
    }
    done = nvec << 2;
  }
  for (long i = done + tid; i < n; i += nthreads) {
    if (DOT) acc += (double)x[i] * y[i];
    else acc = T::comb(acc, T::one(one(x[i], NIN == 2 ? y[i] : 0.f)));
  }
  acc = block_reduce<BASE>(acc, smem);
  if (gridDim.x > 1) {
    if (threadIdx.x == 0) {
      s->partial[blockIdx.x] = acc;
      __threadfence();
      const unsigned int t = atomicAdd(&s->ticket, 1u);
      is_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    acc = T::init(x[0]);
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) acc = T::comb(acc, ((volatile double *)s->partial)[i]);
    acc = block_reduce<BASE>(acc, smem);
    if (threadIdx.x == 0) s->ticket = 0;  // ready for the next launch on this stream
  }
  if (threadIdx.x == 0) scalar_deliver(slot, acc, seq);
}

// x (and y): n floats each, in any order the two share
template <int MODE, class Term>
double reduce_flat(const float *x, const float *y, long n, Term term) {
  constexpr int NIN = MODE == RED_DOT ? 2 : Term::NIN;
  Context &c = ctx();
  RedScratch *s = (RedScratch *)scratch(sizeof(RedScratch));
  // the ticket starts at 0 (scratch is zero-filled when allocated); each launch resets it
  const bool vec = aligned16(x) && (NIN == 1 || aligned16(y));
  const long work = vec ? (n + 3) / 4 : n;
  // one block up to eight loads per thread: below that the ticket's round trips cost more than a second block gains
  int blocks = work <= 8 * 512 ? 1 : (int)std::min<long>((work + 511) / 512, std::min(1024, c.sm_count * 4));   // 4 x 512 threads fill an SM
  const unsigned long long seq = scalar_expect();
  pdl_launch(reduce_all_kernel<MODE, Term>, blocks, 512, 0, x, y, n, vec, s, term, c.scalar_slot_dev, seq);
  check_launch("reduce_all");
  return scalar_wait(seq);
}

// A tensor whose elements occupy one gap-free block of memory in some dim order (contiguous, or a
// transposed / permuted view of a contiguous block): order-free reductions can run over the block.
bool is_dense_block(const THGPUTensor *t);
bool same_layout(const THGPUTensor *a, const THGPUTensor *b);

template <int MODE, class Term>
double reduce_all(THGPUTensor *t, THGPUTensor *u, Term term) {
  const long n = nelem(t);
  THC_ARG(n > 0, 1, "tensor must have one dimension");
  if (MODE == RED_DOT || Term::NIN == 2) {
    THC_ARG(nelem(u) == n, 2, "sizes do not match");
    if (is_dense_block(t) && same_layout(t, u)) return reduce_flat<MODE>(data_ptr(t), data_ptr(u), n, term);
    TensorRef tc(tensor_new_contiguous(t)), uc(tensor_new_contiguous(u));
    return reduce_flat<MODE>(data_ptr(tc), data_ptr(uc), n, term);
  }
  if (is_dense_block(t)) return reduce_flat<MODE>(data_ptr(t), nullptr, n, term);
  TensorRef tc(tensor_new_contiguous(t));
  return reduce_flat<MODE>(data_ptr(tc), nullptr, n, term);
}

}  // namespace thc

#endif
