// BLAS front-ends on raw device pointers (column-major Fortran convention), the layer the
// reference implemented in gputorch/lib/THC/THCBlas.cpp: gemm dispatch :249-288 over four 16x16
// tile kernels :10-246 (three of which ignored the leading dimensions), gemv :291-467, axpy
// :470-483, ger :486-502.  Here gemm maps onto the shared matrix-multiply engines (tcgen05 3xTF32
// by default: the two-SM one, or a warp-level one for small and narrow products), all leading dimensions are honoured and C is not read when beta == 0.
#include "mm_launch.cuh"

namespace thc {

struct ScaleOp { float v; __device__ float operator()(const float *a) const { return a[0] * v; } };

static __global__ void scale_matrix_kernel(float *c, long m, long n, long ldc, float beta) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m * n) return;
  const long j = t / m, i = t - j * m;
  c[i + j * ldc] = beta == 0.f ? 0.f : beta * c[i + j * ldc];
}

// out[i + j * ldc] = bias[i]
static __global__ void broadcast_rows_kernel(float *c, long m, long n, long ldc, const float *__restrict__ bias) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m * n) return;
  const long j = t / m, i = t - j * m;
  c[i + j * ldc] = bias[i];
}
// Up to two matrices copied to pitches that TMA can address (blockIdx.y: which): lines of `run` floats.
struct PackJob { const float *src; float *dst; long lines, run, src_ld, dst_ld; };
static __global__ void __launch_bounds__(256) pack_matrix_kernel(const PackJob a, const PackJob b) {
  const PackJob &j = blockIdx.y ? b : a;
  const int lane = threadIdx.x & 31;
  const long warps = (long)gridDim.x * (blockDim.x >> 5);
  for (long l = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); l < j.lines; l += warps) {
    const float *s = j.src + l * j.src_ld;
    float *d = j.dst + l * j.dst_ld;
#pragma unroll 8
    for (long i = lane; i < j.run; i += 32) d[i] = s[i];
  }
}

// Tensor-core path over the matrices as they lie in memory (raw-operand engine): TMA reads either layout of
// either operand, so no pass over the operands precedes the product.
template <bool TA, bool TB>
static void gemm_raw_t(long m, long n, long k, float alpha, const float *a, long lda, const float *b, long ldb, float beta,
                       float *c, long ldc, const float *row_bias) {
  using namespace mm;
  // A(i,l): 'n' a[i + l*lda] runs along the rows (MN-major), 't' a[l + i*lda] along k.  B(j,l): 'n' b[l + j*ldb]
  // runs along k, 't' b[j + l*ldb] along the rows.
  typedef RawOperand<!TA> OpA;
  typedef RawOperand<TB> OpB;
  Problem<OpA, OpB> p;
  p.epi = Epilogue{c, nullptr, alpha, beta, LONG_MAX, 0, ldc};
  p.epi.row_bias = row_bias;
  p.M = m; p.N = n; p.K = k;
  launch_raw(p, [&](Problem<OpA, OpB> &q, int bn2) {
    attach_raw_map(q.a, a, m, k, lda, TC_BM);
    attach_raw_map(q.b, b, n, k, ldb, bn2 / 2);
  });
}
static void gemm_raw(bool ta, bool tb, long m, long n, long k, float alpha, const float *a, long lda, const float *b,
                     long ldb, float beta, float *c, long ldc, const float *row_bias) {
  if (!mm::raw_matrix_ok(a, lda) || !mm::raw_matrix_ok(b, ldb)) {
    // a pitch or address that TMA cannot take: copy that matrix (a hundredth of the product's time at the sizes that come
    // here) instead of feeding the product through per-thread copies
    PackJob ja = {}, jb = {};
    auto job = [](const float *src, long lines, long run, long ld, PackJob &j) {
      j = PackJob{src, nullptr, lines, run, ld, (run + 3) / 4 * 4};
      j.dst = (float *)ws_alloc(sizeof(float) * j.lines * j.dst_ld);
    };
    if (!mm::raw_matrix_ok(a, lda)) { job(a, ta ? m : k, ta ? k : m, lda, ja); a = ja.dst; lda = ja.dst_ld; }
    if (!mm::raw_matrix_ok(b, ldb)) { job(b, tb ? k : n, tb ? n : k, ldb, jb); b = jb.dst; ldb = jb.dst_ld; }
    const long lines = std::max(ja.lines, jb.lines);
    pack_matrix_kernel<<<dim3((unsigned)std::min<long>((lines + 7) / 8, ctx().sm_count * 8l), 2), 256, 0, stream()>>>(ja, jb);
    check_launch("pack_matrix");
  }
  if (!ta && !tb) gemm_raw_t<false, false>(m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, row_bias);
  else if (ta && !tb) gemm_raw_t<true, false>(m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, row_bias);
  else if (!ta && tb) gemm_raw_t<false, true>(m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, row_bias);
  else gemm_raw_t<true, true>(m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, row_bias);
}
// Whether the warp-level engine (mm_small.cuh) finishes before the two-SM one: both times in microseconds, as measured for
// m, n in 32 .. 2048 and k in 32 .. 2048.  Small: 5 to start, 22 per GFLOP (30 with 4-byte copies; n counts in tiles), about
// 1 us per MB of results.  Two-SM: 11 to start and 0.033 per k up to 512 (a tile's pipeline fill), 2.9 per GFLOP; tiles of
// 128 columns and less wait longer for each k tile; packing adds a launch and a pass over the operand.
static bool small_is_faster(long m, long n, long k, bool aligned) {
  if (!mm::tc2_tile_width(m, n)) return true;
  const double lo = (double)std::min(m, n), hi = (double)std::max(m, n), bn = lo <= 8 ? 8 : lo <= 16 ? 16 : lo <= 32 ? 32 : 64;
  const double gf = 2e-9 * (double)m * (double)n * (double)k, padded = gf * (std::ceil(lo / bn) * bn / lo) * (std::ceil(hi / 64) * 64 / hi);
  const double small = 5 + (aligned ? 22 : 30) * padded + 0.95e-6 * 4 * (double)m * (double)n;
  double raw = 11 + 0.033 * (double)std::min(k, 512l) + 2.9 * gf;
  if (n <= 128) raw += 0.0083 * (double)std::min(k, 2048l);
  if (!aligned) raw += 5 + 1e-6 * 4 * (double)k * (hi + lo);
  return small < raw;
}

// BF16 math mode: one BF16 plane per operand, the BF16 two-SM engine; products too small for it run FP32-accurate.
static void gemm_half(bool ta, bool tb, long m, long n, long k, float alpha, const float *a, long lda, const float *b,
                      long ldb, float beta, float *c, long ldc, const float *row_bias) {
  using namespace mm;
  HalfPlane pa = make_half_plane(a, ta ? lda : 1, ta ? 1 : lda, m, k);
  HalfPlane pb = make_half_plane(b, tb ? 1 : ldb, tb ? ldb : 1, n, k);
  Problem<SplitOperand, SplitOperand> p;
  p.a = half_operand(pa.p, m, pa.ld);
  p.b = half_operand(pb.p, n, pb.ld);
  p.epi = Epilogue{c, nullptr, alpha, beta, LONG_MAX, 0, ldc};
  p.epi.row_bias = row_bias;
  p.M = m; p.N = n; p.K = pa.ld / 2;
  launch_planes_half(p);
}

// Small and narrow products: operands as they lie, whatever their layout and alignment.
static void gemm_small(bool ta, bool tb, long m, long n, long k, float alpha, const float *a, long lda, const float *b,
                       long ldb, float beta, float *c, long ldc, const float *row_bias) {
  mm::SmallProblem p = {};
  p.a = mm::small_operand(a, lda); p.b = mm::small_operand(b, ldb);
  p.M = (int)m; p.N = (int)n; p.K = (int)k;
  p.c = c; p.sm = 1; p.sn = ldc;
  p.alpha = alpha; p.beta = beta;
  p.bias = row_bias; p.bias_m = 1;
  mm::launch_small(p, ta, !tb);
}

template <bool TA, bool TB>
static void gemm_t(long m, long n, long k, float alpha, const float *a, long lda, const float *b, long ldb,
                   float beta, float *c, long ldc) {
  using namespace mm;
  typedef Operand<LinearMap, LinearMap, 0, TA> OpA;     // 't': memory runs along k
  typedef Operand<LinearMap, LinearMap, 0, !TB> OpB;    // 'n': b[l + j*ldb] runs along k
  Problem<OpA, OpB> p;
  p.a.base = a;
  p.a.rows = LinearMap{m, TA ? lda : 1};
  p.a.ks = LinearMap{k, TA ? 1 : lda};
  p.b.base = b;
  p.b.rows = LinearMap{n, TB ? 1 : ldb};
  p.b.ks = LinearMap{k, TB ? ldb : 1};
  auto vec_ok = [](const float *base, long row_stride, long k_stride) {
    return (int)(((uintptr_t)base & 15) == 0 && row_stride % 4 == 0 && k_stride == 1);
  };
  p.a.vec4 = vec_ok(a, p.a.rows.stride, p.a.ks.stride);
  p.b.vec4 = vec_ok(b, p.b.rows.stride, p.b.ks.stride);
  p.a.H = p.a.W = p.b.H = p.b.W = 0;
  p.a.dH = p.a.dW = p.b.dH = p.b.dW = 1;
  p.epi = Epilogue{c, nullptr, alpha, beta, LONG_MAX, 0, ldc};
  p.M = m; p.N = n; p.K = k;
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
    broadcast_rows_kernel<<<ceil_div(m * n, 256), 256, 0, stream()>>>(c, m, n, ldc, row_bias);
    check_launch("broadcast_rows");
    row_bias = nullptr;
    beta = 1.f;
  }
  if (k <= 0 || alpha == 0.f) {
    if (beta == 1.f) return;
    scale_matrix_kernel<<<ceil_div(m * n, 256), 256, 0, stream()>>>(c, m, n, ldc, beta);
    check_launch("scale_matrix");
    return;
  }
  if (mode != 1) {
    const bool aligned = mm::raw_matrix_ok(a, lda) && mm::raw_matrix_ok(b, ldb);
    if (small_is_faster(m, n, k, aligned)) gemm_small(ta, tb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, row_bias);
    else if (mode == 2 && mm::tc2h_tile_width(m, n, false)) gemm_half(ta, tb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, row_bias);
    else gemm_raw(ta, tb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, row_bias);
    return;
  }
  if (!ta && !tb) gemm_t<false, false>(m, n, k, alpha, a, lda, b, ldb, beta, c, ldc);
  else if (ta && !tb) gemm_t<true, false>(m, n, k, alpha, a, lda, b, ldb, beta, c, ldc);
  else if (!ta && tb) gemm_t<false, true>(m, n, k, alpha, a, lda, b, ldb, beta, c, ldc);
  else gemm_t<true, true>(m, n, k, alpha, a, lda, b, ldb, beta, c, ldc);
}

// y = beta*y + alpha*op(A)*x.  'n': A is m x n column-major, y has m entries: threads own rows
// (coalesced across the column).  't': y has n entries, one warp per column of A.
// block = 32 rows x 32 column slices; the slices' partial sums are folded in slice order (deterministic)
static __global__ void __launch_bounds__(1024) gemv_n_kernel(long m, long n, float alpha, const float *__restrict__ a, long lda,
                                                             const float *__restrict__ x, long incx, float beta, float *y,
                                                             long incy) {
  __shared__ float part[32][33];
  const long i = (long)blockIdx.x * 32 + threadIdx.x;
  float acc = 0.f;
  if (i < m)
    for (long j = threadIdx.y; j < n; j += 32) acc = fmaf(a[i + j * lda], x[j * incx], acc);
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
  const long nthreads = (long)gridDim.x * blockDim.x;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nthreads)
    y[i * incy] = __fadd_rn(y[i * incy], __fmul_rn(a, x[i * incx]));
}
static __global__ void ger_kernel(long m, long n, float alpha, const float *__restrict__ x, long incx,
                                  const float *__restrict__ y, long incy, float *a, long lda) {
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
    gemv_t_kernel<<<ceil_div(n, 8), 256, 0, stream()>>>(m, n, alpha, a, lda, x, incx, beta, y, incy);
    check_launch("gemv_t");
  } else {
    gemv_n_kernel<<<ceil_div(m, 32), dim3(32, 32), 0, stream()>>>(m, n, alpha, a, lda, x, incx, beta, y, incy);
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
  axpy_kernel<<<blocks, 256, 0, stream()>>>(n, a, x, incx, y, incy);
  check_launch("axpy");
  THC_END()
}

THC_API void THGPUBlas_ger(long m, long n, float alpha, const float *x, long incx, const float *y, long incy,
                           float *a, long lda) {
  THC_BEGIN
  if (m <= 0 || n <= 0) return;
  ger_kernel<<<ceil_div(m * n, 256), 256, 0, stream()>>>(m, n, alpha, x, incx, y, incy, a, lda);
  check_launch("ger");
  THC_END()
}

// ---- stall reporting of the tensor-core kernels ---------------------------------------------------------------
// One warp waits, with the engines' own bounded wait, on an mbarrier that nobody arrives on, and on expiry does
// what an engine CTA does: raises the stall flags and returns.  It faults nothing and waits no longer than
// `limit` SM cycles (plus one polling interval of a few tens of microseconds).
static __global__ void stall_probe_kernel(const mm::StallCtl ctl) {
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
  stall_probe_kernel<<<1, 32, 0, stream()>>>(ctl);
  check_launch("stall_probe");
  return 0;
  THC_END(1)
}
