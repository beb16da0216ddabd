// BLAS front-ends on raw device pointers (column-major Fortran convention), the layer the
// reference implemented in gputorch/lib/THC/THCBlas.cpp: gemm dispatch :249-288 over four 16x16
// tile kernels :10-246 (three of which ignored the leading dimensions), gemv :291-467, axpy
// :470-483, ger :486-502.  Here gemm maps onto the shared matrix-multiply engines (tcgen05 3xTF32
// by default: the two-SM one, or a warp-level one for small and narrow products), all leading dimensions are honoured and C is not read when beta == 0.
#include "mm_launch.cuh"

namespace thc {

struct ScaleOp { float v; __device__ float operator()(const float *a) const { return a[0] * v; } };

static __global__ void scale_matrix_kernel(float *c, long m, long n, long ldc, float beta) {
  pdl_begin();
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m * n) return;
  const long j = t / m, i = t - j * m;
  c[i + j * ldc] = beta == 0.f ? 0.f : beta * c[i + j * ldc];
}

// out[i + j * ldc] = bias[i]
static __global__ void broadcast_rows_kernel(float *c, long m, long n, long ldc, const float *__restrict__ bias) {
  pdl_begin();
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m * n) return;
  const long j = t / m, i = t - j * m;
  c[i + j * ldc] = bias[i];
}
// Up to two matrices copied to pitches that TMA can address (blockIdx.y: which): lines of `run` floats.
struct PackJob { const float *src; float *dst; long lines, run, src_ld, dst_ld; };
static __global__ void __launch_bounds__(256) pack_matrix_kernel(const PackJob a, const PackJob b) {
  pdl_begin();
  // a warp copies up to 1024 floats of a line, all its loads in flight before the first store
  const PackJob &j = blockIdx.y ? b : a;
  const int lane = threadIdx.x & 31;
  const long warps = (long)gridDim.x * (blockDim.x >> 5), parts = (j.run + 1023) / 1024;
  for (long w = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < j.lines * parts; w += warps) {
    const long l = w / parts, i0 = (w - l * parts) * 1024 + lane;
    const float *s = j.src + l * j.src_ld;
    float *d = j.dst + l * j.dst_ld;
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = i0 + 32 * i < j.run ? s[i0 + 32 * i] : 0.f;
#pragma unroll
    for (int i = 0; i < 32; i++)
      if (i0 + 32 * i < j.run) d[i0 + 32 * i] = v[i];
  }
}

// Tensor-core path over the matrices as they lie in memory (raw-operand engine): TMA reads either layout of
// either operand, so no pass over the operands precedes the product.
template <bool A_MN, bool B_MN>
static void gemm_raw_t(const float *a, long lda, const float *b, long ldb, long m, long n, long k, const mm::Epilogue &epi) {
  using namespace mm;
  Problem<RawOperand<A_MN>, RawOperand<B_MN>> p;
  p.epi = epi;
  p.M = m; p.N = n; p.K = k;
  launch_raw(p, [&](auto &q, int bn2) {
    attach_raw_map<kTf32>(q.a, a, m, k, lda, TC_BM);
    attach_raw_map<kTf32>(q.b, b, n, k, ldb, bn2 / 2);
  });
}
// One side of a product: element (r, l) at p[l + r * ld] (along_k) or p[r + l * ld].
struct GemmSide { const float *p; long ld; bool along_k; long rows; };
// Orientation of the 256-row tiles and the epilogue for D(i, j) at c[i + j * ldc]: the first side takes the rows unless it has
// no more than half a tile of them and the other has more.
static mm::Epilogue gemm_sides(GemmSide &x, GemmSide &y, float alpha, float beta, float *c, long ldc, const float *row_bias) {
  if (x.rows <= 128 && y.rows > x.rows) {
    std::swap(x, y);
    mm::Epilogue e{c, row_bias, alpha, beta, 1, ldc, 1};   // rows of the product are columns of c: out[m * ldc + n]
    return e;
  }
  mm::Epilogue e{c, nullptr, alpha, beta, LONG_MAX, 0, ldc};
  e.row_bias = row_bias;
  return e;
}
// BF16 math mode: one K-major BF16 plane per operand, BF16 products.  For results of more than half a tile's rows and more
// than 32 columns; smaller ones stay FP32-accurate.
static void gemm_half(GemmSide x, GemmSide y, long k, float alpha, float beta, float *c, long ldc, const float *row_bias) {
  using namespace mm;
  Problem<RawOperand<false, kBf16>, RawOperand<false, kBf16>, false, kBf16> p;
  p.epi = gemm_sides(x, y, alpha, beta, c, ldc, row_bias);
  const HalfMatrix hx = make_half_matrix(x.p, x.along_k ? x.ld : 1, x.along_k ? 1 : x.ld, x.rows, k);
  const HalfMatrix hy = make_half_matrix(y.p, y.along_k ? y.ld : 1, y.along_k ? 1 : y.ld, y.rows, k);
  p.M = x.rows; p.N = y.rows; p.K = hx.ld;
  launch_raw(p, [&](auto &q, int bn2) {
    attach_raw_map<kBf16>(q.a, hx.p, x.rows, hx.ld, hx.ld, TC_BM);
    attach_raw_map<kBf16>(q.b, hy.p, y.rows, hy.ld, hy.ld, bn2 / 2);
  });
}
static void gemm_raw(GemmSide x, GemmSide y, long k, float alpha, float beta, float *c, long ldc, const float *row_bias) {
  const mm::Epilogue epi = gemm_sides(x, y, alpha, beta, c, ldc, row_bias);
  if (!mm::raw_matrix_ok(x.p, x.ld) || !mm::raw_matrix_ok(y.p, y.ld)) {
    // a pitch or address that TMA cannot take: copy that matrix (a hundredth of the product's time at the sizes that come
    // here) instead of feeding the product through per-thread copies
    PackJob jobs[2] = {};
    GemmSide *sides[2] = {&x, &y};
    for (int i = 0; i < 2; i++) {
      GemmSide &s = *sides[i];
      if (mm::raw_matrix_ok(s.p, s.ld)) continue;
      PackJob &j = jobs[i];
      j = PackJob{s.p, nullptr, s.along_k ? s.rows : k, s.along_k ? k : s.rows, s.ld, ((s.along_k ? k : s.rows) + 3) / 4 * 4};
      j.dst = (float *)ws_alloc(sizeof(float) * j.lines * j.dst_ld);
      s.p = j.dst; s.ld = j.dst_ld;
    }
    const long pieces = std::max(jobs[0].lines * ((jobs[0].run + 1023) / 1024), jobs[1].lines * ((jobs[1].run + 1023) / 1024));
    pdl_launch(pack_matrix_kernel, dim3((unsigned)std::min<long>((pieces + 7) / 8, ctx().sm_count * 8l), 2), 256, 0, jobs[0], jobs[1]);
    check_launch("pack_matrix");
  }
  if (!x.along_k && y.along_k) gemm_raw_t<true, false>(x.p, x.ld, y.p, y.ld, x.rows, y.rows, k, epi);
  else if (x.along_k && y.along_k) gemm_raw_t<false, false>(x.p, x.ld, y.p, y.ld, x.rows, y.rows, k, epi);
  else if (!x.along_k) gemm_raw_t<true, true>(x.p, x.ld, y.p, y.ld, x.rows, y.rows, k, epi);
  else gemm_raw_t<false, true>(x.p, x.ld, y.p, y.ld, x.rows, y.rows, k, epi);
}
// The same over FP16 pairs: a pass measures both operands and one splits them, each as it lies in memory.
template <bool A_MN, bool B_MN>
static void gemm_pairs_t(const void *a, long lda, const void *b, long ldb, long m, long n, long k, const mm::Epilogue &epi,
                         const mm::Ranges &ranges) {
  using namespace mm;
  Problem<RawOperand<A_MN, kPairs>, RawOperand<B_MN, kPairs>, false, kPairs> p;
  p.epi = epi;
  p.M = m; p.N = n; p.K = k;
  p.range_a = ranges.rec[0]; p.range_b = ranges.rec[1]; p.ranges = ranges;
  launch_raw(p, [&](auto &q, int bn2) {
    attach_raw_map<kPairs>(q.a, a, m, k, lda, TC_BM);
    attach_raw_map<kPairs>(q.b, b, n, k, ldb, bn2 / 2);
  });
}
// False: there is no room for the pairs, and nothing has been done.
static bool gemm_pairs(GemmSide x, GemmSide y, long k, float alpha, float beta, float *c, long ldc, const float *row_bias) {
  using namespace mm;
  // the copies, with a little for the measures (under a hundredth of them) and the partial sums (blocks of 256 KB, up to
  // five rounds of clusters)
  double need = 96e6;
  for (const GemmSide &s : {x, y}) need += 4.1 * (double)(s.along_k ? s.rows : k) * (double)((s.along_k ? k : s.rows) + 64);
  if (!ws_reserve((size_t)need)) return false;
  const Epilogue epi = gemm_sides(x, y, alpha, beta, c, ldc, row_bias);
  const Measured m[2] = {new_measured(), new_measured()};
  RangeJob ranges[2];
  PairJob jobs[2];
  StraySide strays[2];
  const GemmSide *sides[2] = {&x, &y};
  long pieces = 0;
  for (int i = 0; i < 2; i++) {
    const GemmSide &s = *sides[i];
    const long lines = s.along_k ? s.rows : k, run = s.along_k ? k : s.rows, ldp = (run + 63) / 64 * 64;
    ranges[i] = range_job(s.p, lines, run, s.ld, m[i]);
    jobs[i] = PairJob{s.p, ws_alloc(sizeof(float) * lines * ldp), lines, run, s.ld, ldp, ((uintptr_t)s.p & 15) == 0 && s.ld % 4 == 0, {}};
    jobs[i].ranges.rec[0] = m[i].rec; jobs[i].ranges.rec[1] = m[1 - i].rec;
    strays[i] = StraySide{s.p, s.ld, run, s.along_k, m[i]};
    pieces = std::max(pieces, lines * ((ldp + 511) / 512));
  }
  launch_ranges(ranges[0], &ranges[1]);
  pdl_launch(split_matrix_kernel, dim3((unsigned)std::min<long>((pieces + 7) / 8, ctx().sm_count * 8l), 2), 256, 0, jobs[0], jobs[1]);
  check_launch("split_matrix");
  const Ranges &r = jobs[0].ranges;
  if (!x.along_k && y.along_k) gemm_pairs_t<true, false>(jobs[0].dst, jobs[0].ldp, jobs[1].dst, jobs[1].ldp, x.rows, y.rows, k, epi, r);
  else if (x.along_k && y.along_k) gemm_pairs_t<false, false>(jobs[0].dst, jobs[0].ldp, jobs[1].dst, jobs[1].ldp, x.rows, y.rows, k, epi, r);
  else if (!x.along_k) gemm_pairs_t<true, true>(jobs[0].dst, jobs[0].ldp, jobs[1].dst, jobs[1].ldp, x.rows, y.rows, k, epi, r);
  else gemm_pairs_t<false, true>(jobs[0].dst, jobs[0].ldp, jobs[1].dst, jobs[1].ldp, x.rows, y.rows, k, epi, r);
  pdl_launch(matrix_strays_kernel, dim3((unsigned)std::min(ceil_div(y.rows, 256), ctx().sm_count), 4), 256, 0, strays[0], strays[1], x.rows, y.rows, epi, r);
  check_launch("matrix_strays");
  return true;
}
// Whether pairs finish before TF32, the passes over the operands included.  Their copies are scratch that TF32 does without: bounded.
// Measured on both sides of the line (us, pairs / TF32): 2048^3 78.0 / 75.8, 2304^3 102.5 / 108.0, 2560^3 125 / 148, 1500 x 3001 x 2222 115 / 129, 4096 x 4096
// x 512 88 / 98, 1024 x 4096 x 4096 131 / 167.  Operands that have to stay in FP32 take up to two fifths longer than TF32 does
// (2304^3 142, 1024 x 4096 x 4096 217, 4096^3 731 / 621, 8192^3 5030 / 5004): the measuring pass, a copy, wider tiles.
static bool pairs_are_faster(long m, long n, long k) {
  if (4. * (double)k * (double)(m + n) > 16e9 || std::max(std::max(m, n), k) > 1l << 28) return false;
  const double passes = 14 + 4e-6 * (double)k * (double)(m + n) * (1 / 5.5 + 2 / 5.0);
  return mm::tc2_product_us(m, n, k, mm::kPairs, true) + passes < mm::tc2_product_us(m, n, k, mm::kTf32);
}
// Whether the warp-level engine (mm_small.cuh) finishes before the two-SM one.  The latter, as measured for the same sizes: 11 us to
// start, then the fill and fold of its long pipeline (0.026 per k up to 512) and 2.9 per GFLOP, or the operands' bytes
// at 3.3 TB/s; packing adds a launch and a pass over the operands.
static bool small_is_faster(long m, long n, long k, bool aligned) {
  const double gf = 2e-9 * (double)((m + 63) / 64 * 64) * (double)((n + 63) / 64 * 64) * (double)k, bytes = 4 * (double)k * (double)(m + n);
  double raw = 11 + std::max(0.026 * (double)std::min(k, 512l) + 2.9 * gf, bytes / 3.3e6);
  if (!aligned) raw += 5 + bytes / 2e6;
  return mm::small_product_us(m, n, k, aligned) < raw;
}

// Small and narrow products: operands as they lie, whatever their layout and alignment.
static void gemm_small(const GemmSide &x, const GemmSide &y, long k, float alpha, float beta, float *c, long ldc, const float *row_bias) {
  mm::SmallProblem p = {};
  p.a = mm::small_operand(x.p, x.ld); p.b = mm::small_operand(y.p, y.ld);
  p.M = (int)x.rows; p.N = (int)y.rows; p.K = (int)k;
  p.c = c; p.sm = 1; p.sn = ldc;
  p.alpha = alpha; p.beta = beta;
  p.bias = row_bias; p.bias_m = 1;
  mm::launch_small(p, x.along_k, y.along_k);
}

// FP32 FMA mode
static void gemm_simt(const GemmSide &x, const GemmSide &y, long k, float alpha, float beta, float *c, long ldc) {
  using namespace mm;
  Problem<Operand<LinearMap, LinearMap, 0>, Operand<LinearMap, LinearMap, 0>> p;
  auto side = [&](auto &op, const GemmSide &s) {
    op.base = s.p;
    op.rows = LinearMap{s.rows, s.along_k ? s.ld : 1};
    op.ks = LinearMap{k, s.along_k ? 1 : s.ld};
    op.H = op.W = 0; op.dH = op.dW = 1;
  };
  side(p.a, x); side(p.b, y);
  p.epi = Epilogue{c, nullptr, alpha, beta, LONG_MAX, 0, ldc};
  p.M = x.rows; p.N = y.rows; p.K = k;
  launch_simt(p);
}

void gemm(char transa, char transb, long m, long n, long k, float alpha, const float *a, long lda,
          const float *b, long ldb, float beta, float *c, long ldc, const float *row_bias) {
  const bool ta = transa == 't' || transa == 'T', tb = transb == 't' || transb == 'T';
  if (m <= 0 || n <= 0) return;
  constexpr long kPart = 1l << 30;   // the engines count rows and k in 32 bits
  if (m > kPart || n > kPart || k > kPart) {
    for (long l0 = 0; l0 < std::max(k, 1l); l0 += kPart)
      for (long j0 = 0; j0 < n; j0 += kPart)
        for (long i0 = 0; i0 < m; i0 += kPart)
          gemm(transa, transb, std::min(kPart, m - i0), std::min(kPart, n - j0), std::min(kPart, k - l0), alpha,
               a + (ta ? l0 + i0 * lda : i0 + l0 * lda), lda, b + (tb ? j0 + l0 * ldb : l0 + j0 * ldb), ldb, l0 ? 1.f : beta,
               c + i0 + j0 * ldc, ldc, l0 || !row_bias ? nullptr : row_bias + i0);
    return;
  }
  WsScope ws_scope;
  const int mode = ctx().math_mode;
  if (row_bias && (mode == 1 || k <= 0 || alpha == 0.f)) {   // engines without a bias input: D starts as the bias
    pdl_launch(broadcast_rows_kernel, ceil_div(m * n, 256), 256, 0, c, m, n, ldc, row_bias);
    check_launch("broadcast_rows");
    row_bias = nullptr;
    beta = 1.f;
  }
  if (k <= 0 || alpha == 0.f) {
    if (beta == 1.f) return;
    pdl_launch(scale_matrix_kernel, ceil_div(m * n, 256), 256, 0, c, m, n, ldc, beta);
    check_launch("scale_matrix");
    return;
  }
  // A(i,l): 'n' a[i + l*lda], 't' a[l + i*lda].  B(j,l): 'n' b[l + j*ldb], 't' b[j + l*ldb].
  const GemmSide x{a, lda, ta, m}, y{b, ldb, !tb, n};
  if (mode == 1) { gemm_simt(x, y, k, alpha, beta, c, ldc); return; }
  const bool aligned = mm::raw_matrix_ok(a, lda) && mm::raw_matrix_ok(b, ldb);
  if (mode == 2 && m > 128 && n > 32) gemm_half(x, y, k, alpha, beta, c, ldc, row_bias);
  else if (small_is_faster(m, n, k, aligned)) gemm_small(x, y, k, alpha, beta, c, ldc, row_bias);
  else if (!(mode == 0 && pairs_are_faster(m, n, k) && gemm_pairs(x, y, k, alpha, beta, c, ldc, row_bias)))
    gemm_raw(x, y, k, alpha, beta, c, ldc, row_bias);
}

// y = beta*y + alpha*op(A)*x.  'n': A is m x n column-major, y has m entries: threads own rows
// (coalesced across the column).  't': y has n entries, one warp per column of A.
// block = 32 rows x 32 column slices; the slices' partial sums are folded in slice order (deterministic)
static __global__ void __launch_bounds__(1024) gemv_n_kernel(long m, long n, float alpha, const float *__restrict__ a, long lda,
                                                             const float *__restrict__ x, long incx, float beta, float *y,
                                                             long incy) {
  pdl_begin();
  __shared__ float part[32][33];
  const long i = (long)blockIdx.x * 32 + threadIdx.x;
  float acc = 0.f;
  if (i < m) {
    // eight columns on the way at once, added in their order (gradBias of three layers over 256 rows 21 -> 15 us)
    for (long j0 = threadIdx.y; j0 < n; j0 += 8 * 32) {
      float v[8], w[8];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const long j = j0 + 32 * k;
        v[k] = j < n ? a[i + j * lda] : 0.f;
        w[k] = j < n ? x[j * incx] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (j0 + 32 * k < n) acc = fmaf(v[k], w[k], acc);
    }
  }
  part[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && i < m) {
    float sum = 0.f;
#pragma unroll
    for (int s = 0; s < 32; s++) sum += part[s][threadIdx.x];
    y[i * incy] = (beta == 0.f ? 0.f : beta * y[i * incy]) + alpha * sum;
  }
}
static __global__ void gemv_t_kernel(long m, long n, float alpha, const float *__restrict__ a, long lda,
                                     const float *__restrict__ x, long incx, float beta, float *y, long incy) {
  pdl_begin();
  const long j = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j >= n) return;
  const int lane = threadIdx.x & 31;
  float acc = 0.f;
  for (long i = lane; i < m; i += 32) acc = fmaf(a[i + j * lda], x[i * incx], acc);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) y[j * incy] = (beta == 0.f ? 0.f : beta * y[j * incy]) + alpha * acc;
}
static __global__ void axpy_kernel(long n, float a, const float *__restrict__ x, long incx, float *y, long incy) {
  pdl_begin();
  const long nthreads = (long)gridDim.x * blockDim.x;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nthreads)
    y[i * incy] = __fadd_rn(y[i * incy], __fmul_rn(a, x[i * incx]));
}
static __global__ void ger_kernel(long m, long n, float alpha, const float *__restrict__ x, long incx,
                                  const float *__restrict__ y, long incy, float *a, long lda) {
  pdl_begin();
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m * n) return;
  const long j = t / m, i = t - j * m;
  a[i + j * lda] += alpha * x[i * incx] * y[j * incy];
}

}  // namespace thc

using namespace thc;

THC_API void THGPUBlas_gemm(char transa, char transb, long m, long n, long k, float alpha, const float *a, long lda,
                            const float *b, long ldb, float beta, float *c, long ldc) {
  THC_BEGIN
  gemm(transa, transb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc);
  THC_END()
}

THC_API void THGPUBlas_gemv(char trans, long m, long n, float alpha, const float *a, long lda, const float *x,
                            long incx, float beta, float *y, long incy) {
  THC_BEGIN
  if (m <= 0 || n <= 0) return;
  if (trans == 't' || trans == 'T') {
    pdl_launch(gemv_t_kernel, ceil_div(n, 8), 256, 0, m, n, alpha, a, lda, x, incx, beta, y, incy);
    check_launch("gemv_t");
  } else {
    pdl_launch(gemv_n_kernel, ceil_div(m, 32), dim3(32, 32), 0, m, n, alpha, a, lda, x, incx, beta, y, incy);
    check_launch("gemv_n");
  }
  THC_END()
}

THC_API void THGPUBlas_axpy(long n, float a, const float *x, long incx, float *y, long incy) {
  THC_BEGIN
  if (n <= 0) return;
  int blocks = ceil_div(n, 256);
  const int cap = ctx().sm_count * 8;
  if (blocks > cap) blocks = cap;
  pdl_launch(axpy_kernel, blocks, 256, 0, n, a, x, incx, y, incy);
  check_launch("axpy");
  THC_END()
}

THC_API void THGPUBlas_ger(long m, long n, float alpha, const float *x, long incx, const float *y, long incy,
                           float *a, long lda) {
  THC_BEGIN
  if (m <= 0 || n <= 0) return;
  pdl_launch(ger_kernel, ceil_div(m * n, 256), 256, 0, m, n, alpha, x, incx, y, incy, a, lda);
  check_launch("ger");
  THC_END()
}

// ---- stall reporting of the tensor-core kernels ---------------------------------------------------------------
// One warp waits, with the engines' own bounded wait, on an mbarrier that nobody arrives on, and on expiry does
// what an engine CTA does: raises the stall flags and returns.  It faults nothing and waits no longer than
// `limit` SM cycles (plus one polling interval of a few tens of microseconds).
static __global__ void stall_probe_kernel(const mm::StallCtl ctl) {
  pdl_begin();
  __shared__ uint64_t bar;
  __shared__ mm::WaitCtl w;
  if (threadIdx.x == 0) {
    mm::mbar_init(mm::smem_u32(&bar), 1);
    mm::wait_ctl_init(&w, ctl);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (w.abort) return;   // a stall is already on record
  const bool ok = mm::mbar_wait(mm::smem_u32(&bar), 0, &w, mm::kWaitProbe);
  if (!ok && threadIdx.x == 0) mm::stall_raise(ctl, w.abort);
}

THC_API void THGPUSetWaitLimit(long cycles) {
  THC_BEGIN
  THC_CHECK(cycles >= 1024 && cycles <= (1l << 34), "wait limit must lie in [2^10, 2^34] SM cycles");
  ctx().stall_limit = cycles;
  THC_END()
}
THC_API long THGPUGetWaitLimit(void) { THC_BEGIN return (long)ctx().stall_limit; THC_END(-1) }

THC_API int THGPUStallProbe(long limit_cycles) {
  THC_BEGIN
  Context &c = ctx();
  if (limit_cycles < 0) {   // host only: what the host sees after a kernel has raised the flag
    *(volatile int *)c.stall_host = 1;
    return 0;
  }
  THC_CHECK(limit_cycles >= 1024 && limit_cycles <= (1l << 27), "probe limit must lie in [2^10, 2^27] SM cycles");
  mm::StallCtl ctl = stall_ctl();
  ctl.limit = limit_cycles;
  pdl_launch(stall_probe_kernel, 1, 32, 0, ctl);
  check_launch("stall_probe");
  return 0;
  THC_END(1)
}
