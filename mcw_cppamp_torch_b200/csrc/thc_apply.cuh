// Elementwise kernel family shared by copy, tensor math and Threshold.
//
// One functor, three data paths, picked on the host from the operands' strides:
//   contiguous : float4 grid-stride streaming (the HBM-bound fast path)
//   tiled 2-D  : operands whose unit-stride dimension differs from the output's (transposed views):
//                4 x 4 blocks transposed in registers where 16-byte accesses are possible, else
//                64 x 64 shared-memory tiles, so that every global access stays coalesced; counts the
//                same algorithmic bytes as the contiguous case
//   strided    : anything else (and transposed operands of a few rows or columns), collapsed dims + div/mod indexing (correct, not fast)
// This replaces the reference pattern "newContiguous every operand, run, freeCopyTo the result"
// (gputorch/lib/THC/THCTensorMath.cpp:67-163) and its per-element div/mod copy kernel
// (gputorch/lib/THC/THCTensorCopy.cpp:170-218).
#ifndef THC_APPLY_CUH
#define THC_APPLY_CUH

#include "per_device.h"
#include "thc_internal.h"

#include <type_traits>

namespace thc {

template <int NIN>
struct Operands {
  float *out;
  const float *in[NIN > 0 ? NIN : 1];
};

template <typename Op, int NIN>
__global__ void __launch_bounds__(256) apply_contig_kernel(Operands<NIN> p, long n, bool vec, Op op) {
  pdl_begin();
  const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long nthreads = (long)gridDim.x * blockDim.x;
  long done = 0;
  if (vec) {
    const long nvec = n >> 2;
    long i = tid;
    // U independent 16-byte loads per operand in flight per thread before the first store: one load per thread left
    // the one-input operations at 0.86 of the copy rate the two-input ones reach with their two
    constexpr int U = NIN <= 1 ? 4 : 2;
    for (; i + (U - 1) * nthreads < nvec; i += U * nthreads) {
      float4 v[U][NIN > 0 ? NIN : 1];
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int k = 0; k < NIN; k++) v[u][k] = reinterpret_cast<const float4 *>(p.in[k])[i + u * nthreads];
#pragma unroll
      for (int u = 0; u < U; u++) {
        float a[NIN > 0 ? NIN : 1];
        float4 r;
#pragma unroll
        for (int k = 0; k < NIN; k++) a[k] = v[u][k].x;
        r.x = op(a);
#pragma unroll
        for (int k = 0; k < NIN; k++) a[k] = v[u][k].y;
        r.y = op(a);
#pragma unroll
        for (int k = 0; k < NIN; k++) a[k] = v[u][k].z;
        r.z = op(a);
#pragma unroll
        for (int k = 0; k < NIN; k++) a[k] = v[u][k].w;
        r.w = op(a);
        reinterpret_cast<float4 *>(p.out)[i + u * nthreads] = r;
      }
    }
    for (; i < nvec; i += nthreads) {
      float4 v[NIN > 0 ? NIN : 1];
#pragma unroll
      for (int k = 0; k < NIN; k++) v[k] = reinterpret_cast<const float4 *>(p.in[k])[i];
      float a[NIN > 0 ? NIN : 1];
      float4 r;
#pragma unroll
      for (int k = 0; k < NIN; k++) a[k] = v[k].x;
      r.x = op(a);
#pragma unroll
      for (int k = 0; k < NIN; k++) a[k] = v[k].y;
      r.y = op(a);
#pragma unroll
      for (int k = 0; k < NIN; k++) a[k] = v[k].z;
      r.z = op(a);
#pragma unroll
      for (int k = 0; k < NIN; k++) a[k] = v[k].w;
      r.w = op(a);
      reinterpret_cast<float4 *>(p.out)[i] = r;
    }
    done = nvec << 2;
  }
  for (long i = done + tid; i < n; i += nthreads) {
    float a[NIN > 0 ? NIN : 1];
#pragma unroll
    for (int k = 0; k < NIN; k++) a[k] = p.in[k][i];
    p.out[i] = op(a);
  }
}

struct StridedArgs {
  int nd;
  long size[kMaxDims];
  long stride[4][kMaxDims];
};

template <typename Op, int NIN>
__global__ void __launch_bounds__(256) apply_strided_kernel(Operands<NIN> p, StridedArgs s, long n, Op op) {
  pdl_begin();
  const long nthreads = (long)gridDim.x * blockDim.x;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nthreads) {
    long rem = i, off[NIN + 1];
#pragma unroll
    for (int k = 0; k <= NIN; k++) off[k] = 0;
    for (int d = s.nd - 1; d >= 0; d--) {
      const long q = rem / s.size[d], r = rem - q * s.size[d];
#pragma unroll
      for (int k = 0; k <= NIN; k++) off[k] += r * s.stride[k][d];
      rem = q;
    }
    float a[NIN > 0 ? NIN : 1];
#pragma unroll
    for (int k = 0; k < NIN; k++) a[k] = p.in[k][off[k + 1]];
    p.out[off[0]] = op(a);
  }
}

// Order in which the tiles of a transposing kernel are taken: strips of eight tiles along dim 0, inside a strip dim 0
// fastest.  The blocks that run together then cover a wide rectangle, so that both the rows they write (along dim 1)
// and the rows they read (transposed inputs, along dim 0) are runs of 2 KB and more instead of one 256-byte piece per
// DRAM page.
struct TileWalk {
  unsigned tiles0, tiles1;
  __host__ __device__ unsigned count() const { return tiles0 * tiles1; }
  __device__ __forceinline__ void at(unsigned t, unsigned &t0, unsigned &t1) const {
    constexpr unsigned G = 8;
    const unsigned strip = t / (G * tiles1), r = t - strip * G * tiles1;
    const unsigned h = tiles0 - strip * G < G ? tiles0 - strip * G : G;
    t1 = r / h;
    t0 = strip * G + (r - t1 * h);
  }
};
// strides of a 2-D index space: [operand][dim], operand 0 is the output
struct Strides2d {
  long s[4][2];
};
// How many of an operand set's inputs before `k` are staged in shared memory, i.e. the place of its tile.
__host__ __device__ constexpr int staged_before(unsigned via, int k) {
  int n = 0;
  for (int i = 0; i < k; i++) n += via >> i & 1u;
  return n;
}

// 2-D index space (n0, n1); the output has unit stride along dim 1.  Inputs flagged in VIA have unit stride along
// dim 0 and are transposed through 64 x 64 shared-memory tiles: for sizes, pitches or addresses that 16-byte accesses
// cannot serve.  Every global access of a warp is one contiguous 128-byte segment, eight per thread and operand in
// flight.  Bound by instruction issue, not by memory, as long as each element pays for its whole address and bounds tests (58
// instructions a warp access, half the issue slots, 3.5 TB/s on 3001 x 5003): hence steps from one pointer per tile (64 bits
// wide: any pitch; 32-bit ones measured no faster) and a path without tests for the tiles inside.  Three inputs (addcmul)
// need 64 registers: two blocks an SM (3001 x 5003: 51 us with one input transposed, 43 contiguous; element by element 128, the result transposed 465).
template <typename Op, int NIN, unsigned VIA>   // VIA: bit k = operand k is transposed
__global__ void __launch_bounds__(512, NIN == 3 ? 2 : 3) apply_tiled2d_kernel(Operands<NIN> p, int n0, int n1, const Strides2d st,
                                                                TileWalk walk, Op op) {
  pdl_begin();
  constexpr int T = 64, PITCH = T + 1, TY = 512 / T, NJ = T / TY;
  extern __shared__ float tile2d_smem[];   // one [T][PITCH] tile per staged operand
  const int tx = threadIdx.x % T, ty = threadIdx.x / T;
  const unsigned ntiles = walk.count();
  auto one_tile = [&](int b0, int b1, auto inside) {
    constexpr bool INSIDE = decltype(inside)::value;
    float direct[NIN > 1 ? NIN : 1][NIN > 1 ? NJ : 1];   // a single input is always the staged one
#pragma unroll
    for (int k = 0; k < NIN; k++) {
      if (VIA & (1u << k)) {   // rows of the tile run along dim 0
        const float *src = p.in[k] + (b0 + tx) + (b1 + ty) * st.s[k + 1][1];
        const long step = TY * st.s[k + 1][1];
        float *tile = tile2d_smem + staged_before(VIA, k) * T * PITCH + ty * PITCH + tx;
        float v[NJ];
#pragma unroll
        for (int j = 0; j < NJ; j++) v[j] = (INSIDE || (b0 + tx < n0 && b1 + ty + j * TY < n1)) ? src[j * step] : 0.f;
#pragma unroll
        for (int j = 0; j < NJ; j++) tile[j * TY * PITCH] = v[j];
      }
    }
    // operands that need no transposition are fetched into registers BEFORE the barrier, so that their loads fly
    // together with the staged ones instead of starting after them
#pragma unroll
    for (int k = 0; k < (NIN > 1 ? NIN : 0); k++) {
      if (!(VIA & (1u << k))) {
        const float *src = p.in[k] + (b0 + ty) * st.s[k + 1][0] + (b1 + tx) * st.s[k + 1][1];
        const long step = TY * st.s[k + 1][0];
#pragma unroll
        for (int j = 0; j < NJ; j++) direct[k][j] = (INSIDE || (b0 + ty + j * TY < n0 && b1 + tx < n1)) ? src[j * step] : 0.f;
      }
    }
    __syncthreads();
    float *dst = p.out + (b0 + ty) * st.s[0][0] + (b1 + tx);
    const long step = TY * st.s[0][0];
#pragma unroll
    for (int j = 0; j < NJ; j++) {
      float a[NIN];
#pragma unroll
      for (int k = 0; k < NIN; k++)
        a[k] = (VIA & (1u << k)) ? tile2d_smem[staged_before(VIA, k) * T * PITCH + tx * PITCH + ty + j * TY]
                                 : direct[NIN > 1 ? k : 0][NIN > 1 ? j : 0];
      if (INSIDE || (b0 + ty + j * TY < n0 && b1 + tx < n1)) dst[j * step] = op(a);
    }
    __syncthreads();
  };
  for (unsigned t = blockIdx.x; t < ntiles; t += gridDim.x) {
    unsigned t0, t1;
    walk.at(t, t0, t1);
    const int b0 = (int)t0 * T, b1 = (int)t1 * T;
    if (b0 + T <= n0 && b1 + T <= n1) one_tile(b0, b1, std::true_type());
    else one_tile(b0, b1, std::false_type());
  }
}

// The same index space with 16-byte accesses on both sides and no shared memory: a thread owns a 4 x 4 block, reads a
// transposed input as four 16-byte rows along dim 0, the others as four along dim 1, and transposes in registers.
// A warp covers 16 (dim 0) x 32 (dim 1): transposed inputs arrive in whole 64-byte segments whose other half the
// neighbouring warp of the block fetches, results leave in 128-byte segments.  No barrier, so loads of later
// tiles fly under the stores of earlier ones.  addcmul on 8192 x 8192: 160 us contiguous, 170 - 194 with any operands
// transposed (527 - 1346 element by element).  n0, n1 and all pitches multiples of 4, 16-byte aligned bases.
template <typename Op, int NIN, unsigned VIA>
__global__ void __launch_bounds__(256) apply_transpose4_kernel(Operands<NIN> p, int n0, int n1, const Strides2d st, TileWalk walk,
                                                               Op op) {
  pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int o0 = (warp & 3) * 16 + (lane & 3) * 4, o1 = (warp >> 2) * 32 + (lane >> 2) * 4;
  const unsigned ntiles = walk.count();
  for (unsigned t = blockIdx.x; t < ntiles; t += gridDim.x) {
    unsigned t0, t1;
    walk.at(t, t0, t1);
    const int i0 = (int)t0 * 64 + o0, i1 = (int)t1 * 64 + o1;
    if (i0 >= n0 || i1 >= n1) continue;
    float v[NIN][4][4];   // [operand][row of the access][element]
#pragma unroll
    for (int k = 0; k < NIN; k++) {
      const bool tr = (VIA & (1u << k)) != 0;
      const long step = tr ? st.s[k + 1][1] : st.s[k + 1][0];
      const float *b = p.in[k] + (tr ? i1 * step + i0 : i0 * step + i1);
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float4 q = *reinterpret_cast<const float4 *>(b + r * step);
        v[k][r][0] = q.x; v[k][r][1] = q.y; v[k][r][2] = q.z; v[k][r][3] = q.w;
      }
    }
    float *dst = p.out + i0 * st.s[0][0] + i1;
#pragma unroll
    for (int r = 0; r < 4; r++) {
      float o[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        float a[NIN];
#pragma unroll
        for (int k = 0; k < NIN; k++) a[k] = ((VIA & (1u << k)) != 0) ? v[k][c][r] : v[k][r][c];
        o[c] = op(a);
      }
      *reinterpret_cast<float4 *>(dst + r * st.s[0][0]) = make_float4(o[0], o[1], o[2], o[3]);
    }
  }
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// f(integral constant `via`) for via in [FIRST, END)
template <unsigned FIRST, unsigned END, class F> void with_via(unsigned via, F f) {
  if constexpr (FIRST < END) {
    if (via == FIRST) f(std::integral_constant<unsigned, FIRST>());
    else with_via<FIRST + 1, END>(via, f);
  }
}

// out = op(in...) over tensors of equal shape (already resized by the caller); out may alias an input.
template <int NIN, typename Op>
void apply(THGPUTensor *out, const THGPUTensor *in0, const THGPUTensor *in1, Op op, const char *name,
           const THGPUTensor *in2 = nullptr) {
  const long n = nelem(out);
  if (n == 0) return;
  const THGPUTensor *ops[4] = {out, in0, in1, in2};
  Operands<NIN> p;
  p.out = data_ptr(out);
  for (int k = 0; k < NIN; k++) p.in[k] = data_ptr(ops[k + 1]);
  const int max_blocks = ctx().sm_count * 8;
  bool all_contig = is_contiguous(out);
  for (int k = 0; k < NIN; k++) all_contig = all_contig && is_contiguous(ops[k + 1]);
  if (all_contig) {
    bool vec = aligned16(p.out);
    for (int k = 0; k < NIN; k++) vec = vec && aligned16(p.in[k]);
    long work = vec ? (n + 3) / 4 : n;
    int blocks = (int)((work + 255) / 256);
    if (blocks > max_blocks) blocks = max_blocks;
    pdl_launch(apply_contig_kernel<Op, NIN>, blocks, 256, 0, p, n, vec, op);
    check_launch(name);
    return;
  }
  Strided s;
  THC_CHECK(collapse(NIN + 1, ops, s), "%s: too many non-collapsible dimensions", name);
  if constexpr (NIN >= 1) {
    if (s.nd == 2) {
      // normalise so that the output's unit-stride dim is dim 1
      int a = 0, b = 1;
      if (s.stride[0][1] != 1 && s.stride[0][0] == 1) { a = 1; b = 0; }
      if (s.stride[0][b] == 1) {
        unsigned via = 0;
        for (int k = 0; k < NIN; k++)
          if (s.stride[k + 1][a] == 1 && s.stride[k + 1][b] != 1) via |= 1u << k;
        const bool fits = s.size[0] < (1l << 31) - 128 && s.size[1] < (1l << 31) - 128;   // 32-bit places
        const long n0 = s.size[a], n1 = s.size[b];
        const long tiles0 = (n0 + 63) / 64, tiles1 = (n1 + 63) / 64;
        Strides2d st = {};
        for (int k = 0; k <= NIN; k++) { st.s[k][0] = s.stride[k][a]; st.s[k][1] = s.stride[k][b]; }
        // 16-byte accesses on every operand: pitches and extents multiples of 4, aligned bases
        bool vec = aligned16(p.out) && n0 % 4 == 0 && n1 % 4 == 0 && st.s[0][0] % 4 == 0;
        for (int k = 0; k < NIN; k++)
          vec = vec && aligned16(p.in[k]) && ((via >> k & 1u) ? st.s[k + 1][1] % 4 == 0 : st.s[k + 1][1] == 1 && st.s[k + 1][0] % 4 == 0);
        // A few rows or columns fill a few of a tile's 64, and the tile takes as long.  33.5 M elements in 2 / 6 rows: cadd 1593 / 553
        // us through shared-memory tiles, 243 / 263 element by element (addcmul 2178 / 748 against 263 / 275, copy 1087 / 382
        // against 235 / 255); the former falls as one over the rows, which puts the line at 9 - 16.  Blocks turned in
        // registers, in 4 / 8 rows: copy 180 / 105 us, cadd 307 / 183, addcmul 324 / 194 against 235, 248 and 266.
        const bool wide = std::min(n0, n1) >= (vec ? (NIN == 3 ? 8 : 4) : 12);
        if (via && fits && wide && tiles0 * tiles1 < (1l << 30)) {
          const TileWalk walk{(unsigned)tiles0, (unsigned)tiles1};
          const unsigned blocks = std::min(walk.count(), (unsigned)max_blocks);
          const auto launch = [&](auto v) {
            constexpr unsigned VIA = decltype(v)::value;
            if (vec) {
              pdl_launch(apply_transpose4_kernel<Op, NIN, VIA>, blocks, 256, 0, p, (int)n0, (int)n1, st, walk, op);
            } else {
              constexpr size_t smem = (size_t)staged_before(VIA, NIN) * 64 * 65 * sizeof(float);
              if constexpr (smem > 48 * 1024) {   // three staged tiles
                static PerDevice allowed;
                allowed.get(ctx().device, [] {
                  THC_CUDA(cudaFuncSetAttribute(apply_tiled2d_kernel<Op, NIN, VIA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                  return 1;
                });
              }
              pdl_launch(apply_tiled2d_kernel<Op, NIN, VIA>, blocks, 512, smem, p, (int)n0, (int)n1, st, walk, op);
            }
          };
          with_via<1, (1u << NIN)>(via, launch);
          check_launch(name);
          return;
        }
      }
    }
  }
  StridedArgs sa;
  sa.nd = s.nd;
  for (int d = 0; d < kMaxDims; d++) {
    sa.size[d] = d < s.nd ? s.size[d] : 1;
    for (int k = 0; k < 4; k++) sa.stride[k][d] = d < s.nd ? s.stride[k][d] : 0;
  }
  int blocks = (int)((n + 255) / 256);
  if (blocks > max_blocks) blocks = max_blocks;
  pdl_launch(apply_strided_kernel<Op, NIN>, blocks, 256, 0, p, sa, n, op);
  check_launch(name);
}

}  // namespace thc

#endif
