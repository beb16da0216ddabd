// torch.GPUTensor math: elementwise, full reductions, dim-wise reductions, BLAS-backed products.
//
// Reference: gputorch/lib/THC/THCTensorMath.cpp (line ranges per function in include/THC.h) and its
// Bolt wrappers gputorch/lib/THC/THCBolt.cpp:96-412.  Numerics follow the CPU TH semantics the
// results are checked against (mcw_torch7_core/lib/TH/generic/THTensorMath.c): sums accumulate in
// double (TH's accreal), max/min use strict comparisons so the first extremum wins.
#include <cfloat>

#include "thc_reduce.cuh"

namespace thc {

// ------------------------------------------------------------------ elementwise functors
struct ConstOp { float v; __device__ float operator()(const float *) const { return v; } };
struct AddScalarOp { float v; __device__ float operator()(const float *a) const { return a[0] + v; } };
struct MulScalarOp { float v; __device__ float operator()(const float *a) const { return a[0] * v; } };
struct DivScalarOp { float v; __device__ float operator()(const float *a) const { return a[0] / v; } };
// t + value*src with the product rounded before the sum, like the C expression on the CPU
struct CaddOp { float v; __device__ float operator()(const float *a) const { return __fadd_rn(a[0], __fmul_rn(v, a[1])); } };
struct CmulOp { __device__ float operator()(const float *a) const { return a[0] * a[1]; } };
struct CdivOp { __device__ float operator()(const float *a) const { return a[0] / a[1]; } };

static void resize_as(THGPUTensor *r, const THGPUTensor *t) { tensor_resize_as(r, t); }

// ------------------------------------------------------------------ full reductions (thc_reduce.cuh)
bool is_dense_block(const THGPUTensor *t) {
  int order[kMaxDims * 4];
  int nd = 0;
  for (int d = 0; d < t->nDimension; d++)
    if (t->size[d] != 1) { if (nd >= kMaxDims * 4) return false; order[nd++] = d; }
  for (int i = 1; i < nd; i++)
    for (int j = i; j > 0 && t->stride[order[j]] < t->stride[order[j - 1]]; j--) {
      int z = order[j]; order[j] = order[j - 1]; order[j - 1] = z;
    }
  long z = 1;
  for (int i = 0; i < nd; i++) {
    if (t->stride[order[i]] != z) return false;
    z *= t->size[order[i]];
  }
  return true;
}

bool same_layout(const THGPUTensor *a, const THGPUTensor *b) {
  if (a->nDimension != b->nDimension) return false;
  for (int d = 0; d < a->nDimension; d++)
    if (a->size[d] != b->size[d] || (a->size[d] != 1 && a->stride[d] != b->stride[d])) return false;
  return true;
}

// ------------------------------------------------------------------ dim-wise reductions
// The source is described as out(o, j) <- reduce_r src[base + o*so + j*sj + r*sr].
//   row kernel   : sr == 1 (reduced dim is the unit-stride one).  One block per output, or one warp.
//   column kernel: sj == 1 (outputs are unit-stride neighbours).  Threads own 1 or 4 columns each, the
//                  reduced dim is additionally split over threadIdx.y and blockIdx.y; the last block of a
//                  column range folds the blockIdx.y partials in ascending order.
template <int MODE, class I = long> __device__ __forceinline__ bool better(float a, I ia, float b, I ib) {
  // true when (a, ia) should replace (b, ib): strictly better value, or equal value at a lower index
  if (MODE == RED_MAX) return a > b || (a == b && ia < ib);
  return a < b || (a == b && ia < ib);
}

template <int MODE>
__global__ void __launch_bounds__(256) reduce_rows_kernel(const float *__restrict__ src, long so, long R,
                                                          float *__restrict__ out, float *__restrict__ idx,
                                                          float scale, bool vec) {
  pdl_begin();
  __shared__ double sd[32];
  __shared__ float sv[32];
  __shared__ long si[32];
  const float *row = src + (long)blockIdx.x * so;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  if (MODE == RED_SUM) {
    double acc = 0;
    long done = 0;
    if (vec) {
      const float4 *r4 = reinterpret_cast<const float4 *>(row);
      const long n4 = R >> 2, bd = blockDim.x;
      long i = threadIdx.x;
      // four 16-byte loads in flight per thread before the first add (a row of 8192 floats is two such rounds)
      for (; i + 3 * bd < n4; i += 4 * bd) {
        const float4 v0 = r4[i], v1 = r4[i + bd], v2 = r4[i + 2 * bd], v3 = r4[i + 3 * bd];
        acc += (double)v0.x + (double)v0.y + (double)v0.z + (double)v0.w;
        acc += (double)v1.x + (double)v1.y + (double)v1.z + (double)v1.w;
        acc += (double)v2.x + (double)v2.y + (double)v2.z + (double)v2.w;
        acc += (double)v3.x + (double)v3.y + (double)v3.z + (double)v3.w;
      }
      for (; i < n4; i += bd) {
        const float4 v = r4[i];
        acc += (double)v.x + (double)v.y + (double)v.z + (double)v.w;
      }
      done = n4 << 2;
    }
    for (long i = done + threadIdx.x; i < R; i += blockDim.x) acc += (double)row[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) sd[warp] = acc;
    __syncthreads();
    if (warp == 0) {
      acc = lane < nwarps ? sd[lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) out[blockIdx.x] = (float)(acc * (double)scale);
    }
  } else {
    // positions fit 32 bits (checked by the launcher): half the integer work of 64-bit indices per element
    float bv = row[0];
    int bi = 0;
    long done = 0;
    if (vec) {
      const float4 *r4 = reinterpret_cast<const float4 *>(row);
      const long n4 = R >> 2, bd = blockDim.x;
      // the best of the four first (ties keep the lower position), then one comparison against the running best
      auto take = [&](const float4 &v, long i) {
        const int b = (int)(i << 2);
        float m = v.x; int mi = b;
        if (MODE == RED_MAX ? v.y > m : v.y < m) { m = v.y; mi = b + 1; }
        if (MODE == RED_MAX ? v.z > m : v.z < m) { m = v.z; mi = b + 2; }
        if (MODE == RED_MAX ? v.w > m : v.w < m) { m = v.w; mi = b + 3; }
        if (better<MODE, int>(m, mi, bv, bi)) { bv = m; bi = mi; }
      };
      long i = threadIdx.x;
      for (; i + 3 * bd < n4; i += 4 * bd) {   // four 16-byte loads in flight per thread
        const float4 v0 = r4[i], v1 = r4[i + bd], v2 = r4[i + 2 * bd], v3 = r4[i + 3 * bd];
        take(v0, i); take(v1, i + bd); take(v2, i + 2 * bd); take(v3, i + 3 * bd);
      }
      for (; i < n4; i += bd) take(r4[i], i);
      done = n4 << 2;
    }
    for (long i = done + threadIdx.x; i < R; i += blockDim.x)
      if (better<MODE, int>(row[i], (int)i, bv, bi)) { bv = row[i]; bi = (int)i; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better<MODE, int>(ov, oi, bv, bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { sv[warp] = bv; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
      bv = lane < nwarps ? sv[lane] : sv[0];
      bi = lane < nwarps ? (int)si[lane] : (int)si[0];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (better<MODE, int>(ov, oi, bv, bi)) { bv = ov; bi = oi; }
      }
      if (lane == 0) {
        out[blockIdx.x] = bv;
        if (idx) idx[blockIdx.x] = (float)(bi + 1);
      }
    }
  }
}

// Rows of a few hundred elements: a warp per row, eight rows per block (a block per row would leave most of its
// threads, or most of the SM's block slots, without work).
template <int MODE>
__global__ void __launch_bounds__(256) reduce_rows_warp_kernel(const float *__restrict__ src, long so, long J, int R,
                                                               float *__restrict__ out, float *__restrict__ idx, float scale) {
  pdl_begin();
  const long j = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (j >= J) return;
  const int lane = threadIdx.x & 31;
  const float *row = src + j * so;
  if (MODE == RED_SUM) {
    double acc = 0;
    int i = lane;
    for (; i + 96 < R; i += 128) {
      const float v0 = row[i], v1 = row[i + 32], v2 = row[i + 64], v3 = row[i + 96];
      acc += (double)v0 + (double)v1 + (double)v2 + (double)v3;
    }
    for (; i < R; i += 32) acc += (double)row[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) out[j] = (float)(acc * (double)scale);
  } else {
    float bv = row[0];
    int bi = 0;
#pragma unroll 4
    for (int i = lane; i < R; i += 32) {
      const float v = row[i];
      if (better<MODE, int>(v, i, bv, bi)) { bv = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better<MODE, int>(ov, oi, bv, bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) {
      out[j] = bv;
      if (idx) idx[j] = (float)(bi + 1);
    }
  }
}

// Where a column reduction leaves its results.  With more than one slice of the reduced dimension the partials of
// slice s go to psum / (pval, pidx)[(o * splits + s) * J + j], and the block that finishes last among the slices of its
// columns (tickets[o * gridDim.x + blockIdx.x], zero between launches) folds them in slice order: no second launch.
template <class I>   // positions along the reduced dimension
struct ColOut {
  double *psum;
  float *pval;
  I *pidx;
  unsigned *tickets;
  float *out, *idx;
  float scale;
};
template <int MODE, class I>
__device__ __forceinline__ void cols_emit(const ColOut<I> &w, long t, double acc, float v, I i) {
  if (MODE == RED_SUM) {
    w.out[t] = (float)(acc * (double)w.scale);
  } else {
    w.out[t] = v;
    if (w.idx) w.idx[t] = (float)(i + 1);
  }
}
// Called by all threads of the block once its partials are written; COLS columns from j0 on belong to the block.
template <int MODE, int COLS, class I>
__device__ __forceinline__ void cols_fold_if_last(const ColOut<I> &w, long J, long j0) {
  __shared__ bool is_last;
  const int tid = threadIdx.y * 32 + threadIdx.x, splits = gridDim.y;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    unsigned *ticket = w.tickets + (long)blockIdx.z * gridDim.x + blockIdx.x;
    is_last = atomicAdd(ticket, 1u) == (unsigned)splits - 1;
    if (is_last) *ticket = 0;   // ready for the next launch on this stream
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // `COLS` columns, 256 / COLS interleaved groups of slices per column, folded in group order
  __shared__ double fd[256];
  __shared__ float fv[256];
  __shared__ I fi[256];
  const int c = tid % COLS, grp = tid / COLS;
  constexpr int GROUPS = 256 / COLS;
  const long j = j0 + c, first = (long)blockIdx.z * splits * J + j;
  double acc = 0;
  float bv = 0;
  I bi = -1;
  if (j < J) {
    if (MODE == RED_SUM) {
#pragma unroll 8
      for (int s = grp; s < splits; s += GROUPS) acc += __ldcg(w.psum + first + (long)s * J);
    } else {
      for (int s0 = grp; s0 < splits; s0 += 8 * GROUPS) {
        float ov[8];
        I oi[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int s = s0 + u * GROUPS;
          ov[u] = s < splits ? __ldcg(w.pval + first + (long)s * J) : 0.f;
          oi[u] = s < splits ? __ldcg(w.pidx + first + (long)s * J) : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (oi[u] >= 0 && (bi < 0 || better<MODE, I>(ov[u], oi[u], bv, bi))) { bv = ov[u]; bi = oi[u]; }
      }
    }
  }
  if (MODE == RED_SUM) fd[tid] = acc;
  else { fv[tid] = bv; fi[tid] = bi; }
  __syncthreads();
  if (grp == 0 && j < J) {
    for (int k = 1; k < GROUPS; k++) {
      if (MODE == RED_SUM) {
        acc += fd[k * COLS + c];
      } else {
        const float ov = fv[k * COLS + c];
        const I oi = fi[k * COLS + c];
        if (oi >= 0 && (bi < 0 || better<MODE, I>(ov, oi, bv, bi))) { bv = ov; bi = oi; }
      }
    }
    cols_emit<MODE, I>(w, (long)blockIdx.z * J + j, acc, bv, bi);
  }
}

// grid (ceil(J/32), splits, O); block (32, 8).
template <int MODE, class I>
__global__ void __launch_bounds__(256) reduce_cols_kernel(const float *__restrict__ src, long so, long sr, long J, I R,
                                                          I rows_per_split, const ColOut<I> w) {
  pdl_begin();
  __shared__ double sd[8][33];
  __shared__ float sv[8][33];
  __shared__ I si[8][33];
  const long j = (long)blockIdx.x * 32 + threadIdx.x;
  const I r0 = blockIdx.y * rows_per_split, r1 = min(R, r0 + rows_per_split);
  const float *base = src + (long)blockIdx.z * so + j;
  double acc = 0;
  float bv = 0;
  I bi = -1;
  if (j < J) {
    I r = r0 + (I)threadIdx.y;
    for (; r + 56 < r1; r += 64) {  // eight independent loads in flight per thread
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = base[(long)(r + 8 * u) * sr];
      if (MODE == RED_SUM) {
        acc += (((double)v[0] + (double)v[1]) + ((double)v[2] + (double)v[3])) + (((double)v[4] + (double)v[5]) + ((double)v[6] + (double)v[7]));
      } else {
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (bi < 0 || better<MODE, I>(v[u], r + 8 * u, bv, bi)) { bv = v[u]; bi = r + 8 * u; }
      }
    }
    for (; r < r1; r += 8) {
      const float v = base[(long)r * sr];
      if (MODE == RED_SUM) acc += (double)v;
      else if (bi < 0 || better<MODE, I>(v, r, bv, bi)) { bv = v; bi = r; }
    }
  }
  if (MODE == RED_SUM) sd[threadIdx.y][threadIdx.x] = acc;
  else { sv[threadIdx.y][threadIdx.x] = bv; si[threadIdx.y][threadIdx.x] = bi; }
  __syncthreads();
  if (threadIdx.y == 0 && j < J) {
    if (MODE == RED_SUM) {
      for (int k = 1; k < 8; k++) acc += sd[k][threadIdx.x];
    } else {
      for (int k = 1; k < 8; k++) {
        const float ov = sv[k][threadIdx.x];
        const I oi = si[k][threadIdx.x];
        if (oi >= 0 && (bi < 0 || better<MODE, I>(ov, oi, bv, bi))) { bv = ov; bi = oi; }
      }
    }
    if (gridDim.y == 1) {
      cols_emit<MODE, I>(w, (long)blockIdx.z * J + j, acc, bv, bi);
    } else {
      const long o = ((long)blockIdx.z * gridDim.y + blockIdx.y) * J + j;
      if (MODE == RED_SUM) w.psum[o] = acc;
      else { w.pval[o] = bv; w.pidx[o] = bi; }
    }
  }
  if (gridDim.y > 1) cols_fold_if_last<MODE, 32, I>(w, J, (long)blockIdx.x * 32);
}

// The same with four adjacent columns per thread (16-byte loads: a warp fetches 512 contiguous bytes per row, and
// eight rows are requested before the first is used).  J % 4 == 0, 16-byte aligned rows.  grid (ceil(J/128), splits, O).
template <int MODE, class I>
__global__ void __launch_bounds__(256) reduce_cols4_kernel(const float *__restrict__ src, long so, long sr, long J, I R,
                                                           I rows_per_split, const ColOut<I> w) {
  pdl_begin();
  __shared__ double sd[8][129];
  __shared__ float sv[8][129];
  __shared__ I si[8][129];
  const long j = ((long)blockIdx.x * 32 + threadIdx.x) * 4;
  const I r0 = blockIdx.y * rows_per_split, r1 = min(R, r0 + rows_per_split);
  const float *base = src + (long)blockIdx.z * so + j;
  double acc[4] = {0, 0, 0, 0};
  float bv[4] = {0, 0, 0, 0};
  I bi[4] = {-1, -1, -1, -1};
  auto take = [&](const float4 &v, I r) {
    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int c = 0; c < 4; c++) {
      if (MODE == RED_SUM) acc[c] += (double)e[c];
      else if (bi[c] < 0 || better<MODE, I>(e[c], r, bv[c], bi[c])) { bv[c] = e[c]; bi[c] = r; }
    }
  };
  if (j < J) {
    I r = r0 + (I)threadIdx.y;
    for (; r + 56 < r1; r += 64) {
      float4 v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = *reinterpret_cast<const float4 *>(base + (long)(r + 8 * u) * sr);
#pragma unroll
      for (int u = 0; u < 8; u++) take(v[u], r + 8 * u);
    }
    for (; r < r1; r += 8) take(*reinterpret_cast<const float4 *>(base + (long)r * sr), r);
  }
#pragma unroll
  for (int c = 0; c < 4; c++) {
    if (MODE == RED_SUM) sd[threadIdx.y][threadIdx.x * 4 + c] = acc[c];
    else { sv[threadIdx.y][threadIdx.x * 4 + c] = bv[c]; si[threadIdx.y][threadIdx.x * 4 + c] = bi[c]; }
  }
  __syncthreads();
  // 128 columns of the block, folded over the eight row slices in slice order
  const int col = threadIdx.y * 32 + threadIdx.x;
  const long jc = (long)blockIdx.x * 128 + col;
  if (col < 128 && jc < J) {
    double a = 0;
    float v = 0;
    I i = -1;
    if (MODE == RED_SUM) {
      a = sd[0][col];
      for (int k = 1; k < 8; k++) a += sd[k][col];
    } else {
      v = sv[0][col];
      i = si[0][col];
      for (int k = 1; k < 8; k++) {
        const float ov = sv[k][col];
        const I oi = si[k][col];
        if (oi >= 0 && (i < 0 || better<MODE, I>(ov, oi, v, i))) { v = ov; i = oi; }
      }
    }
    if (gridDim.y == 1) {
      cols_emit<MODE, I>(w, (long)blockIdx.z * J + jc, a, v, i);
    } else {
      const long o = ((long)blockIdx.z * gridDim.y + blockIdx.y) * J + jc;
      if (MODE == RED_SUM) w.psum[o] = a;
      else { w.pval[o] = v; w.pidx[o] = i; }
    }
  }
  if (gridDim.y > 1) cols_fold_if_last<MODE, 128, I>(w, J, (long)blockIdx.x * 128);
}

template <int MODE>
static void reduce_dim(THGPUTensor *values, THGPUTensor *indices, THGPUTensor *src, long dim, float scale) {
  THC_ARG(dim >= 0 && dim < src->nDimension, 3, "dimension out of range");
  // output shape = src shape with size[dim] = 1 (kept), computed into a contiguous result
  long osize[kMaxDims * 4];
  THC_CHECK(src->nDimension <= kMaxDims * 4, "too many dimensions");
  for (int d = 0; d < src->nDimension; d++) osize[d] = src->size[d];
  osize[dim] = 1;
  const long R = src->size[dim];
  TensorRef src_keep;
  const THGPUTensor *orig = src;
  long O, J, so, sj, sr;
  const float *base;
  auto describe = [&](THGPUTensor *t) -> bool {
    // contiguous: [outer, R, inner]
    if (is_contiguous(t)) {
      O = 1; J = 1;
      for (int d = 0; d < dim; d++) O *= t->size[d];
      for (int d = (int)dim + 1; d < t->nDimension; d++) J *= t->size[d];
      so = R * J; sj = 1; sr = J;
      if (J == 1) { J = O; O = 1; sj = R; sr = 1; so = 0; }  // innermost dim: rows
      return true;
    }
    if (t->nDimension == 2) {  // strided 2-D view (e.g. a transpose): use its strides directly
      const int od = dim == 0 ? 1 : 0;
      O = 1; so = 0; J = t->size[od]; sj = t->stride[od]; sr = t->stride[dim];
      return sr == 1 || sj == 1;
    }
    return false;
  };
  THC_ARG(nelem(src) > 0, 3, "empty tensor");
  if (R == 1) {  // nothing to reduce: values = src, every index is 1
    THGPUTensor *c = tensor_new_contiguous(src);
    THGPUTensor *v = tensor_new_sized(src->nDimension, osize);
    tensor_copy(v, c);
    if (MODE == RED_SUM && scale != 1.f) apply<1>(v, v, nullptr, MulScalarOp{scale}, "mean");
    tensor_free(c);
    resize_nd(values, src->nDimension, osize, nullptr);
    tensor_copy(values, v);
    tensor_free(v);
    if (indices) {
      resize_nd(indices, src->nDimension, osize, nullptr);
      apply<0>(indices, nullptr, nullptr, ConstOp{1.f}, "ones");
    }
    return;
  }
  if (!describe(src)) {
    src_keep.reset(tensor_new_contiguous(src));
    src = src_keep;
    describe(src);
  }
  THC_CHECK(O <= 65535, "outer dimension too large for the column reducer");
  base = data_ptr(src);
  const int ond = src->nDimension;
  // Results go where they belong unless a destination shares memory with the source or the other destination, or is not
  // contiguous after resizing: then through a temporary.  Both are resized before either pointer is taken: two views of one
  // storage, the second of which makes it grow, must not leave the first with memory that is gone.
  auto apart = [&](const THGPUTensor *dst) { return !dst->storage || dst->storage != orig->storage; };
  const bool twins = indices && values->storage && values->storage == indices->storage;
  bool direct_v = !twins && apart(values), direct_i = indices && !twins && apart(indices);
  if (direct_v) resize_nd(values, ond, osize, nullptr);
  if (direct_i) resize_nd(indices, ond, osize, nullptr);
  direct_v = direct_v && !overlap(values, orig);
  direct_i = direct_i && !overlap(indices, orig) && !overlap(indices, values);
  auto place = [&](THGPUTensor *dst, bool direct, TensorRef &tmp) -> float * {
    if (!dst) return nullptr;
    if (direct && is_contiguous(dst)) return data_ptr(dst);
    tmp.reset(tensor_new_sized(ond, osize));
    return data_ptr(tmp);
  };
  TensorRef vtmp, itmp;
  float *out = place(values, direct_v, vtmp), *idx = place(indices, direct_i, itmp);
  if (sr == 1) {
    THC_CHECK(O == 1, "internal: row reduce with outer dim");
    THC_CHECK(R < (1l << 31), "reduced dimension too long");
    const bool vec = aligned16(base) && (sj % 4 == 0);
    if (R < 512) {
      pdl_launch(reduce_rows_warp_kernel<MODE>, (unsigned)((J + 7) / 8), 256, 0, base, sj, J, (int)R, out, idx, scale);
    } else {
      const int threads = R >= 4096 ? 256 : 128;
      pdl_launch(reduce_rows_kernel<MODE>, (unsigned)J, threads, 0, base, sj, R, out, idx, scale, vec);
    }
    check_launch("reduce_rows");
  } else {
    THC_CHECK(sj == 1, "internal: column reduce needs unit stride");
    const bool vec4 = J % 4 == 0 && sr % 4 == 0 && so % 4 == 0 && aligned16(base) && J >= 128;
    const long colblocks = vec4 ? (J + 127) / 128 : (J + 31) / 32;
    const long want = (long)ctx().sm_count * 8;
    // slices of at least 64 rows (a thread's eight loads in flight), and none for what one block reads in four rounds
    long splits = R <= 256 ? 1 : std::max(1l, std::min(std::min(want / (colblocks * O), (R + 63) / 64), 512l));
    const long rows_per_split = (R + splits - 1) / splits;
    splits = (R + rows_per_split - 1) / rows_per_split;
    const size_t nparts = splits > 1 ? (size_t)O * splits * J : 0;
    WsScope ws_scope;
    const dim3 grid((unsigned)colblocks, (unsigned)splits, (unsigned)O), block(32, 8);
    auto launch = [&](auto position) {
      typedef decltype(position) I;
      ColOut<I> w = {};
      if (splits > 1) {
        char *scr = (char *)ws_alloc(nparts * std::max(sizeof(double), sizeof(I) + sizeof(float)));
        w.psum = (double *)scr;
        w.pidx = (I *)scr;
        w.pval = (float *)(scr + nparts * sizeof(I));
        THC_CHECK(colblocks * O <= kZeroWords, "internal: too many column ranges to split");
        w.tickets = zero_words();
      }
      w.out = out; w.idx = idx; w.scale = scale;
      if (vec4) pdl_launch(reduce_cols4_kernel<MODE, I>, grid, block, 0, base, so, sr, J, (I)R, (I)rows_per_split, w);
      else pdl_launch(reduce_cols_kernel<MODE, I>, grid, block, 0, base, so, sr, J, (I)R, (I)rows_per_split, w);
    };
    if (R < (1l << 31) - 4096) launch(0);   // a thread steps at most 64 rows past the end
    else launch(0l);
    check_launch("reduce_cols");
  }
  if (vtmp.t) { resize_nd(values, ond, osize, nullptr); tensor_copy(values, vtmp); }
  if (itmp.t) { resize_nd(indices, ond, osize, nullptr); tensor_copy(indices, itmp); }
}

}  // namespace thc

using namespace thc;

THC_API void THGPUTensor_add(THGPUTensor *self, THGPUTensor *src, float value) {
  THC_BEGIN resize_as(self, src); apply<1>(self, src, nullptr, AddScalarOp{value}, "add"); THC_END()
}
THC_API void THGPUTensor_mul(THGPUTensor *self, THGPUTensor *src, float value) {
  THC_BEGIN resize_as(self, src); apply<1>(self, src, nullptr, MulScalarOp{value}, "mul"); THC_END()
}
THC_API void THGPUTensor_div(THGPUTensor *self, THGPUTensor *src, float value) {
  THC_BEGIN resize_as(self, src); apply<1>(self, src, nullptr, DivScalarOp{value}, "div"); THC_END()
}
THC_API void THGPUTensor_cadd(THGPUTensor *self, THGPUTensor *src1, float value, THGPUTensor *src2) {
  THC_BEGIN
  THC_ARG(nelem(src1) == nelem(src2), 3, "size do not match");
  resize_as(self, src1);
  THC_ARG(THGPUTensor_isSameSizeAs(src1, src2), 3, "shapes do not match");
  apply<2>(self, src1, src2, CaddOp{value}, "cadd");
  THC_END()
}
THC_API void THGPUTensor_cmul(THGPUTensor *self, THGPUTensor *src1, THGPUTensor *src2) {
  THC_BEGIN
  THC_ARG(nelem(src1) == nelem(src2), 3, "size do not match");
  resize_as(self, src1);
  THC_ARG(THGPUTensor_isSameSizeAs(src1, src2), 3, "shapes do not match");
  apply<2>(self, src1, src2, CmulOp(), "cmul");
  THC_END()
}
THC_API void THGPUTensor_cdiv(THGPUTensor *self, THGPUTensor *src1, THGPUTensor *src2) {
  THC_BEGIN
  THC_ARG(nelem(src1) == nelem(src2), 3, "size do not match");
  resize_as(self, src1);
  THC_ARG(THGPUTensor_isSameSizeAs(src1, src2), 3, "shapes do not match");
  apply<2>(self, src1, src2, CdivOp(), "cdiv");
  THC_END()
}

THC_API float THGPUTensor_dot(THGPUTensor *self, THGPUTensor *src) { THC_BEGIN return (float)reduce_all<RED_DOT>(self, src, IdTerm()); THC_END(0.f) }
THC_API float THGPUTensor_minall(THGPUTensor *self) { THC_BEGIN return (float)reduce_all<RED_MIN>(self, nullptr, IdTerm()); THC_END(0.f) }
THC_API float THGPUTensor_maxall(THGPUTensor *self) { THC_BEGIN return (float)reduce_all<RED_MAX>(self, nullptr, IdTerm()); THC_END(0.f) }
THC_API float THGPUTensor_sumall(THGPUTensor *self) { THC_BEGIN return (float)reduce_all<RED_SUM>(self, nullptr, IdTerm()); THC_END(0.f) }
THC_API float THGPUTensor_meanall(THGPUTensor *self) {
  THC_BEGIN
  return (float)(reduce_all<RED_SUM>(self, nullptr, IdTerm()) / (double)nelem(self));
  THC_END(0.f)
}

THC_API void THGPUTensor_sum(THGPUTensor *self, THGPUTensor *src, long dim) {
  THC_BEGIN reduce_dim<RED_SUM>(self, nullptr, src, dim, 1.f); THC_END()
}
THC_API void THGPUTensor_mean(THGPUTensor *self, THGPUTensor *src, long dim) {
  THC_BEGIN
  THC_ARG(dim >= 0 && dim < src->nDimension, 3, "dimension out of range");
  reduce_dim<RED_SUM>(self, nullptr, src, dim, 1.f / (float)src->size[dim]);
  THC_END()
}
THC_API void THGPUTensor_max(THGPUTensor *values, THGPUTensor *indices, THGPUTensor *src, long dim) {
  THC_BEGIN reduce_dim<RED_MAX>(values, indices, src, dim, 1.f); THC_END()
}
THC_API void THGPUTensor_min(THGPUTensor *values, THGPUTensor *indices, THGPUTensor *src, long dim) {
  THC_BEGIN reduce_dim<RED_MIN>(values, indices, src, dim, 1.f); THC_END()
}

// ------------------------------------------------------------------ BLAS-backed products
// addmv (THCTensorMath.cpp:624-695): r = beta*t + alpha*mat*vec
THC_API void THGPUTensor_addmv(THGPUTensor *r_, float beta, THGPUTensor *t, float alpha, THGPUTensor *mat, THGPUTensor *vec) {
  THC_BEGIN
  THC_CHECK(mat->nDimension == 2 && vec->nDimension == 1, "matrix and vector expected");
  THC_CHECK(mat->size[1] == vec->size[0], "size mismatch");
  THC_CHECK(t->nDimension == 1 && t->size[0] == mat->size[0], "size mismatch");
  if (r_ != t) { resize_as(r_, t); tensor_copy(r_, t); }
  THGPUTensor *m = nullptr;
  if (mat->stride[0] == 1) {
    THGPUBlas_gemv('n', mat->size[0], mat->size[1], alpha, data_ptr(mat), mat->stride[1], data_ptr(vec), vec->stride[0],
                   beta, data_ptr(r_), r_->stride[0]);
  } else if (mat->stride[1] == 1) {
    THGPUBlas_gemv('t', mat->size[1], mat->size[0], alpha, data_ptr(mat), mat->stride[0], data_ptr(vec), vec->stride[0],
                   beta, data_ptr(r_), r_->stride[0]);
  } else {
    m = tensor_new_contiguous(mat);
    THGPUBlas_gemv('t', mat->size[1], mat->size[0], alpha, data_ptr(m), m->stride[0], data_ptr(vec), vec->stride[0],
                   beta, data_ptr(r_), r_->stride[0]);
    tensor_free(m);
  }
  THC_END()
}

// addr (THCTensorMath.cpp:809-860): r = beta*t + alpha * vec1 (x) vec2
THC_API void THGPUTensor_addr(THGPUTensor *r_, float beta, THGPUTensor *t, float alpha, THGPUTensor *vec1, THGPUTensor *vec2) {
  THC_BEGIN
  THC_CHECK(vec1->nDimension == 1 && vec2->nDimension == 1, "vector and vector expected");
  THC_CHECK(t->nDimension == 2, "size mismatch");
  THC_CHECK(t->size[0] == vec1->size[0] && t->size[1] == vec2->size[0], "size mismatch");
  if (r_ != t) { resize_as(r_, t); tensor_copy(r_, t); }
  if (beta != 1.f) apply<1>(r_, r_, nullptr, MulScalarOp{beta}, "mul");
  if (r_->stride[0] == 1) {
    THGPUBlas_ger(vec1->size[0], vec2->size[0], alpha, data_ptr(vec1), vec1->stride[0], data_ptr(vec2), vec2->stride[0],
                  data_ptr(r_), r_->stride[1]);
  } else if (r_->stride[1] == 1) {
    THGPUBlas_ger(vec2->size[0], vec1->size[0], alpha, data_ptr(vec2), vec2->stride[0], data_ptr(vec1), vec1->stride[0],
                  data_ptr(r_), r_->stride[0]);
  } else {
    THGPUTensor *c = tensor_new_sized(r_->nDimension, r_->size);
    tensor_copy(c, r_);
    THGPUBlas_ger(vec2->size[0], vec1->size[0], alpha, data_ptr(vec2), vec2->stride[0], data_ptr(vec1), vec1->stride[0],
                  data_ptr(c), c->stride[0]);
    tensor_copy(r_, c);
    tensor_free(c);
  }
  THC_END()
}

// addmm (THCTensorMath.cpp:697-807; CPU semantics mcw_torch7_core/lib/TH/generic/THTensorMath.c:458-561):
// r = beta*t + alpha*m1*m2.  Row-major results are computed as the transposed column-major product;
// transpose flags come from the operands' strides, so transposed views cost nothing.  A result with
// neither stride equal to 1 goes through a contiguous temporary and is copied back (the CPU
// behaviour; the reference GPU code wrote into the wrong buffer there).
THC_API void THGPUTensor_addmm(THGPUTensor *r_, float beta, THGPUTensor *t, float alpha, THGPUTensor *m1, THGPUTensor *m2) {
  THC_BEGIN
  THC_CHECK(m1->nDimension == 2 && m2->nDimension == 2, "matrix and matrix expected");
  THC_CHECK(t->nDimension == 2, "size mismatch");
  THC_CHECK(t->size[0] == m1->size[0] && t->size[1] == m2->size[1] && m1->size[1] == m2->size[0], "size mismatch");
  if (t != r_) { resize_as(r_, t); tensor_copy(r_, t); }
  char transpose_r, transpose_m1, transpose_m2;
  THGPUTensor *r__, *m1_, *m2_;
  if (r_->stride[0] == 1 && r_->stride[1] != 0) { transpose_r = 'n'; r__ = r_; }
  else if (r_->stride[1] == 1 && r_->stride[0] != 0) { THGPUTensor *sw = m2; m2 = m1; m1 = sw; transpose_r = 't'; r__ = r_; }
  else {
    transpose_r = 'n';
    const long tsize[2] = {r_->size[1], r_->size[0]};
    r__ = tensor_new_sized(2, tsize);
    { long z = r__->size[0]; r__->size[0] = r__->size[1]; r__->size[1] = z;
      z = r__->stride[0]; r__->stride[0] = r__->stride[1]; r__->stride[1] = z; }
    tensor_copy(r__, r_);
  }
  const int i0 = transpose_r == 'n' ? 0 : 1, i1 = transpose_r == 'n' ? 1 : 0;
  if (m1->stride[i0] == 1 && m1->stride[i1] != 0) { transpose_m1 = 'n'; m1_ = m1; }
  else if (m1->stride[i1] == 1 && m1->stride[i0] != 0) { transpose_m1 = 't'; m1_ = m1; }
  else { transpose_m1 = transpose_r == 'n' ? 't' : 'n'; m1_ = tensor_new_contiguous(m1); }
  if (m2->stride[i0] == 1 && m2->stride[i1] != 0) { transpose_m2 = 'n'; m2_ = m2; }
  else if (m2->stride[i1] == 1 && m2->stride[i0] != 0) { transpose_m2 = 't'; m2_ = m2; }
  else { transpose_m2 = transpose_r == 'n' ? 't' : 'n'; m2_ = tensor_new_contiguous(m2); }
  gemm(transpose_m1, transpose_m2, r__->size[i0], r__->size[i1], m1_->size[i1], alpha, data_ptr(m1_),
       transpose_m1 == 'n' ? m1_->stride[i1] : m1_->stride[i0], data_ptr(m2_),
       transpose_m2 == 'n' ? m2_->stride[i1] : m2_->stride[i0], beta, data_ptr(r__), r__->stride[i1]);
  if (m1_ != m1) tensor_free(m1_);
  if (m2_ != m2) tensor_free(m2_);
  if (r__ != r_) { tensor_copy(r_, r__); tensor_free(r__); }
  THC_END()
}
