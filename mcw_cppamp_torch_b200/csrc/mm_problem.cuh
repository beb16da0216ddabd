// Operand / epilogue descriptions shared by the matrix-multiply engines.
//
// Every GEMM-shaped operation of the library (BLAS gemm behind addmm / Linear, and the three
// SpatialConvolutionMM passes) is stated once as
//
//     D(m, n) = sum_k  A(m, k) * B(n, k)          m < M, n < N, k < K
//
// which is the implicit-GEMM form of what the reference does by materialising a column matrix per image and calling a
// generic SGEMM on it (gputorch/lib/THC/gpunn-impl/SpatialConvolutionMM.cpp:10-92 im2col / col2im, :185-217 host loop;
// operand mapping in the table of the gemm call sites :194-216, :289-300, :404-417).  The tensor-core engine
// (mm_tc2r.cuh) reads its operands through TMA maps; the FP32 FMA engine (mm_simt.cuh) finds an element by adding a per-row
// and a per-k memory offset and passing a small box test that realises zero padding.
#ifndef THC_MM_PROBLEM_CUH
#define THC_MM_PROBLEM_CUH

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "thc_internal.h"

namespace thc {
namespace mm {

struct Info {
  long off;  // memory offset contribution (floats)
  int y, x;  // box-test coordinates contribution
};
constexpr int kInvalid = -(1 << 29);

// What the two-SM engine multiplies.  kTf32: FP32 values, split inside the SM.  kBf16: BF16 values (opt-in mode).  kPairs: FP32
// values that a pass over the operand has split into two FP16 halves (see RangeRec), FP32-accurate like kTf32.
enum : int { kTf32 = 0, kBf16 = 1, kPairs = 2 };

// ---- FP16 pairs --------------------------------------------------------------------------------------------------
// x * 2^e = hi + lo * 2^-11 with hi = fp16(x * 2^e), lo = fp16((x * 2^e - hi) * 2^11), where e puts the operand's largest value into
// [2^14, 2^15): 22 bits of every value whose hi is a normal FP16 number, that is down to 2^-28 of the largest, as the two TF32 parts hold
// (whose hi is truncated), at four bytes a value and twice the tensor pipe's TF32 rate.  FP16's exponents reach no further, and a
// result may rest on smaller values alone (a row of zeros but one), so a pass (range_kernel) measures each operand first.
//   A few smaller values (stray_allowance) are listed; the pairs hold zeros in their place, and what they add to the result is added
//   in FP32 (mm_strays.cuh).  Tensors of 10^8 values have a few: the density of a layer's outputs around zero leaves some
//   below 2^-28 of the largest.
//   More of them, an infinity or a NaN, or a largest value outside [2^-60, 2^60]: all operands of the product stay in FP32, in
//   the same buffers, and the same launch multiplies them as kTf32.
// How many: two hundred times what 10^8 normal values have.  Each may cost the launch that adds it 2 us (4096 x 4096 x 512 with 512 of them in
// a row: 1266 us, 88 over pairs without and about 120 in FP32), so that small operands are allowed few.
constexpr int kStrays = 512;
__host__ __device__ constexpr long stray_allowance(long values) { return values / (1 << 18) + 8; }   // (kStrays at most)
struct Stray { long at; float v; };   // element `at` of the operand, in the order it was measured in
struct RangeRec {
  unsigned max_bits;     // bits of the largest |x|; infinities and NaN rank above every number
  unsigned wide;         // the operand is in FP32 whatever the others say: too many strays, or another operand of its product asked for it
  unsigned ticket;
  unsigned strays;       // length of the list that goes with the record
  unsigned pad[4];
};
constexpr int kRangeWords = sizeof(RangeRec) / 4;
static_assert(kRangeWords == 8, "zeroed_words() keeps 32-byte boundaries");
// What stays of an operand's measures beside planes that outlive a call.
struct KeptRange { RangeRec rec; Stray strays[kStrays]; };
static_assert(sizeof(KeptRange) == kPlaneRecordBytes, "what plane_record() hands out");
__device__ __forceinline__ bool max_is_wide(unsigned max_bits) { return max_bits && (max_bits >> 23 < 127 - 60 || max_bits >> 23 > 127 + 60); }
__device__ __forceinline__ bool range_is_wide(const RangeRec &r) { return r.wide || max_is_wide(r.max_bits); }
// Non-zero magnitudes below these bits are strays (of an operand that is not wide).
__device__ __forceinline__ unsigned stray_limit(unsigned max_bits) { return max_bits ? ((max_bits >> 23) - 28u) << 23 : 0u; }
// 2^e of an operand that is not wide, and 2^-e
__device__ __forceinline__ float pair_scale(const RangeRec &r) { return r.max_bits ? __uint_as_float((127u + 14u + 127u - (r.max_bits >> 23)) << 23) : 1.f; }
__device__ __forceinline__ float pair_unscale(const RangeRec &r) { return r.max_bits ? __uint_as_float(((r.max_bits >> 23) - 14u) << 23) : 1.f; }
// The operands whose form is decided together.  [0]: the one at hand.
struct Ranges {
  const RangeRec *rec[3] = {nullptr, nullptr, nullptr};
  __device__ __forceinline__ bool wide() const {
    bool w = false;
#pragma unroll
    for (int i = 0; i < 3; i++) w = w || (rec[i] && range_is_wide(*rec[i]));
    return w;
  }
};
// An operand's record and list.  `kept`: of planes from an earlier call, which hold zeros for the strays also after they have been
// brought back to FP32; planes that this call wrote in FP32 hold everything.
struct Measured {
  RangeRec *rec = nullptr;
  Stray *list = nullptr;
  bool kept = false;
  __device__ __forceinline__ int strays(bool wide) const { return !rec || (wide && !kept) ? 0 : (int)rec->strays; }
};
// Division of a non-negative 31-bit integer by a runtime constant as multiply-high + shift.
struct FastDiv {
  unsigned d, mul, shr;
  __host__ static FastDiv make(long divisor) {
    FastDiv f;
    f.d = (unsigned)divisor;
    if (divisor <= 1) { f.mul = 0; f.shr = 0; return f; }
    int lg = 0;
    while ((1l << lg) < divisor) lg++;          // ceil(log2 d)
    const int p = 31 + lg;
    f.mul = (unsigned)(((1ull << p) + (unsigned long long)divisor - 1) / (unsigned long long)divisor);
    f.shr = (unsigned)(p - 32);
    return f;
  }
  __device__ __forceinline__ void divmod(unsigned n, unsigned &q, unsigned &r) const {
    q = d > 1 ? (__umulhi(n, mul) >> shr) : n;
    r = n - q * d;
  }
};

// idx -> idx * stride
struct LinearMap {
  long count, stride;
  __device__ __forceinline__ Info operator()(long idx) const {
    Info r;
    r.off = idx * stride;
    r.y = idx < count ? 0 : kInvalid;
    r.x = 0;
    return r;
  }
};

// idx = (img, y, x) over a [count/PP, PP/XW, XW] grid of pixels
struct PixelMap {
  long count;            // < 2^31 (checked by set())
  FastDiv PP, XW;
  long img_stride, y_stride, x_stride, off0;
  int sy, y0, sx, x0;
  void set(long count_, long pp, long xw) {
    THC_CHECK(count_ < (1l << 31) && pp > 0 && xw > 0, "problem too large for 32-bit pixel indices");
    count = count_; PP = FastDiv::make(pp); XW = FastDiv::make(xw);
  }
  __device__ __forceinline__ Info operator()(long idx) const {
    Info r;
    if (idx >= count) { r.off = 0; r.y = kInvalid; r.x = 0; return r; }
    unsigned img, p, y, x;
    PP.divmod((unsigned)idx, img, p);
    XW.divmod(p, y, x);
    r.off = (long)img * img_stride + (long)y * y_stride + (long)x * x_stride + off0;
    r.y = (int)y * sy + y0;
    r.x = (int)x * sx + x0;
    return r;
  }
};

// idx = (c, i, j) over [count/kHW, kHW/kW, kW] filter taps
struct TapMap {
  long count;            // < 2^31 (checked by set())
  FastDiv kHW, kW;
  long c_stride, i_stride, j_stride;
  int si, sj;
  void set(long count_, long khw, long kw) {
    THC_CHECK(count_ < (1l << 31) && khw > 0 && kw > 0, "problem too large for 32-bit tap indices");
    count = count_; kHW = FastDiv::make(khw); kW = FastDiv::make(kw);
  }
  __device__ __forceinline__ Info operator()(long idx) const {
    Info r;
    if (idx >= count) { r.off = 0; r.y = kInvalid; r.x = 0; return r; }
    unsigned c, t, i, j;
    kHW.divmod((unsigned)idx, c, t);
    kW.divmod(t, i, j);
    r.off = (long)c * c_stride + (long)i * i_stride + (long)j * j_stride;
    r.y = (int)i * si;
    r.x = (int)j * sj;
    return r;
  }
};

// BOX 0: valid rows/ks only.  BOX 1: additionally 0 <= y < H and 0 <= x < W (zero padding).
// BOX 2: the summed coordinates must be non-negative multiples of (dH, dW) and the quotients index
//        an H x W plane (gradInput of a strided convolution).
template <class RowMap_, class KMap_, int BOX_>
struct Operand {
  typedef RowMap_ RowMap;
  typedef KMap_ KMap;
  const float *base;
  RowMap rows;
  KMap ks;
  int H, W, dH, dW;
  __device__ __forceinline__ float fetch(const Info &r, const Info &k) const {
    const int ty = r.y + k.y, tx = r.x + k.x;
    if (BOX_ == 0) return ty >= 0 ? base[r.off + k.off] : 0.f;
    if (BOX_ == 1)
      return ((unsigned)ty < (unsigned)H && (unsigned)tx < (unsigned)W) ? base[r.off + k.off] : 0.f;
    if (ty < 0 || tx < 0) return 0.f;
    const int y = ty / dH, x = tx / dW;
    if (y * dH != ty || x * dW != tx || y >= H || x >= W) return 0.f;
    return base[r.off + k.off + (long)y * W + x];
  }
};

// ---------------------------------------------------------------------------------------------
// Operands of the two-SM engine, fetched by TMA (gathered windows: GatheredWindowOperand).  A tile row holds one swizzle span of 128 bytes: KV = 32 FP32 values
// (3xTF32 products) or 64 BF16 values.
//
// A plain matrix: K-major (memory runs along k) or MN-major (memory runs along the rows).  tmap: K-major {K, rows} with
// a {KV, tile rows} box and the 128-byte swizzle; MN-major {rows, K} with a {KV rows, KV k} box per KV-row block (FP32: the
// 32-byte-granule swizzle).  Elements beyond either extent read as zeros.
// kPairs: a row of memory is [hi values | lo values], each padded to whole spans (`lo`: distance of the two); `tmap` is over the
// FP16 values, `tmap_wide` over the FP32 values that the buffer holds instead when a range is too wide.
template <int PREC> struct TensorMaps {
  CUtensorMap tmap;
  __device__ __forceinline__ const CUtensorMap *map(bool) const { return &tmap; }
  __device__ __forceinline__ int half(bool) const { return 0; }
};
template <> struct TensorMaps<kPairs> {
  CUtensorMap tmap, tmap_wide;
  int lo;
  __device__ __forceinline__ const CUtensorMap *map(bool wide) const { return wide ? &tmap_wide : &tmap; }
  __device__ __forceinline__ int half(bool is_lo) const { return is_lo ? lo : 0; }
};
template <bool MN_, int PREC = kTf32>
struct RawOperand : TensorMaps<PREC> {
  static constexpr bool MN_MAJOR = MN_, GATHERED = false;
};

// Convolution windows over a channels-last plane [n_img][H][W][C] (C a multiple of KV), as rows (K-major): row = window (img,
// y, x) of the product's grid, k = (i, j, c).  tmap: im2col map {C, W, H, n_img}, KV channels of 128 consecutive windows at
// one filter tap per load, padding read as zeros.
template <int PREC = kTf32>
struct PlanesWindowOperand : TensorMaps<PREC> {
  static constexpr bool MN_MAJOR = false, GATHERED = false;
  int n_img;
  PixelMap rows;            // window -> coordinates of its corner
  FastDiv C, kW;
  // Corner (x, y) and image of row m, the start coordinates of an im2col load; rows past the end map beyond the last
  // image, where every read is out of bounds (zeros).
  __device__ __forceinline__ void tile_origin(long m, int &x, int &y, int &img) const {
    if (m >= rows.count) { x = rows.x0; y = rows.y0; img = n_img; return; }
    unsigned im, px, yy, xx;
    rows.PP.divmod((unsigned)m, im, px);
    rows.XW.divmod(px, yy, xx);
    x = (int)xx * rows.sx + rows.x0;
    y = (int)yy * rows.sy + rows.y0;
    img = (int)im;
  }
  // Tap (i, j) and channel of reduction index k.
  __device__ __forceinline__ void tile_tap(unsigned k, int &i, int &j, int &c) const {
    unsigned tap, cc, ii, jj;
    C.divmod(k, tap, cc);
    kW.divmod(tap, ii, jj);
    i = (int)ii; j = (int)jj; c = (int)cc;
  }
};

// Convolution windows of a layer of up to eight planes in BF16, as rows (K-major): k = (tap, plane), eight planes a tap.  Not by TMA: a tap of a
// window is 16 bytes of an image of eight-plane pixels (zeros around it where the layer pads), and the engine's warps copy a tile's
// taps, which lie side by side in the image as far as a filter row reaches, straight to their places in shared memory.
struct GatheredWindowOperand {
  static constexpr bool MN_MAJOR = false, GATHERED = true;
  const uint4 *image;
  int image_pixels, pitch;  // pixels of an image and of a row
  int taps, kW;
  PixelMap rows;            // window -> coordinates of its corner (count, PP, XW, sx, sy)
};

// The same windows as the MN-major operand of the weight-gradient product: rows = (tap, c), k = windows.  tmap: im2col
// map, KV channels of KV consecutive windows per load (one KV-row block of a k tile).
struct WindowStep { int x, y, img; };   // a number of windows as columns, rows and images
template <int PREC = kTf32>
struct WindowRowsOperand : TensorMaps<PREC> {
  static constexpr bool MN_MAJOR = true, GATHERED = false;
  int n_img, oH;
  WindowStep step[2];       // 32 and 64 windows
  PixelMap ks;              // window -> coordinates of its corner
  FastDiv C, kW;
  // Column, row and image of window k; past the last one, images that do not exist (every read is out of bounds: zeros).
  __device__ __forceinline__ void pixel(long k, int &x, int &y, int &img) const {
    if (k >= ks.count) { x = y = 0; img = n_img; return; }
    unsigned im, px, yy, xx;
    ks.PP.divmod((unsigned)k, im, px);
    ks.XW.divmod(px, yy, xx);
    x = (int)xx; y = (int)yy; img = (int)im;
  }
  __device__ __forceinline__ void row_tap(long r, int &i, int &j, int &c0) const {
    unsigned tap, c, ii, jj;
    C.divmod((unsigned)r, tap, c);
    kW.divmod(tap, ii, jj);
    i = (int)ii; j = (int)jj; c0 = (int)c;
  }
};

// out[(m / mdiv) * mouter + (m % mdiv) + n * nstride] = alpha*acc (+ bias[n]) (+ beta*old)
struct Epilogue {
  float *out;
  const float *bias;
  float alpha, beta;
  long mdiv, mouter, nstride;
  // Pixel-pair mode (pair_K > 0, beta == 0): a convolution with few output planes computes two horizontally
  // adjacent output pixels per row so that its tile is twice as wide.  Row m = (img, y, x2), column
  // n = (parity, plane): out[img * pair_img + plane * nstride + y * pair_oW + 2 * x2 + parity]; with an odd
  // output width the last pair of a row has no parity-1 pixel.
  long pair_K = 0, pair_oH = 1, pair_oW2 = 1, pair_oW = 0, pair_img = 0;
  const float *row_bias = nullptr;   // added per row (Linear: the output features are the rows); beta == 0, no `bias`
  __device__ __forceinline__ float rb(long m) const { return row_bias ? __ldg(row_bias + m) : 0.f; }
  static constexpr long kLastOdd = 1l << 62;
  // PAIR is a compile-time property of the problem: the common path carries none of the pair arithmetic
  // a / b, by the short division where it will do
  static __device__ __forceinline__ long quotient(long a, long b) { return ((a | b) >> 32) == 0 ? (long)((unsigned)a / (unsigned)b) : a / b; }
  template <bool PAIR = false>
  __device__ __forceinline__ long moff(long m) const {
    if (PAIR) {
      const long r = quotient(m, pair_oW2), x2 = m - r * pair_oW2, img = quotient(r, pair_oH), y = r - img * pair_oH;
      return (img * pair_img + y * pair_oW + 2 * x2) | (2 * x2 + 1 >= pair_oW ? kLastOdd : 0);
    }
    const long q = m < mdiv ? 0 : quotient(m, mdiv);
    return q * mouter + (m - q * mdiv);
  }
  // the same with the destination's previous value already in a register (never in pixel-pair mode)
  __device__ __forceinline__ void store_with(long mo, long n, float acc, float old) const {
    float v = alpha * acc;
    if (bias) v += bias[n];
    v += beta * old;
    out[mo + n * nstride] = v;
  }
  // beta == 0 with the bias fetched by the caller (several columns' bias values at once, ahead of the stores: a
  // load per column between the stores would serialise them, the compiler cannot move it across a store)
  template <bool PAIR = false>
  __device__ __forceinline__ float bias_of(long n) const {
    if (!bias) return 0.f;
    return __ldg(bias + (PAIR && n >= pair_K ? n - pair_K : n));
  }
  template <bool PAIR = false>
  __device__ __forceinline__ void store_biased(long mo, long n, float acc, float b) const {
    const float v = alpha * acc + b;
    if (PAIR) {
      const long par = n >= pair_K ? 1 : 0, plane = n - par * pair_K;
      if (par && (mo & kLastOdd)) return;
      out[(mo & ~kLastOdd) + plane * nstride + par] = v;
      return;
    }
    out[mo + n * nstride] = v;
  }
  template <bool PAIR = false>
  __device__ __forceinline__ void store(long mo, long n, float acc, float row_b = 0.f) const {
    if (PAIR) {
      const long par = n >= pair_K ? 1 : 0, plane = n - par * pair_K;
      if (par && (mo & kLastOdd)) return;
      float v = alpha * acc;
      if (bias) v += bias[plane];
      out[(mo & ~kLastOdd) + plane * nstride + par] = v;
      return;
    }
    const long o = mo + n * nstride;
    out[o] = value(n, acc, row_b, beta != 0.f ? out[o] : 0.f);
  }
  __device__ __forceinline__ float value(long n, float acc, float row_b, float old) const {
    float v = alpha * acc + row_b;
    if (bias) v += bias[n];
    if (beta != 0.f) v += beta * old;
    return v;
  }
};

template <class OpA_, class OpB_, bool PAIR_ = false, int PREC_ = kTf32>
struct Problem {
  typedef OpA_ OpA;
  typedef OpB_ OpB;
  static constexpr bool PAIR = PAIR_;   // pixel-pair epilogue (see Epilogue)
  static constexpr int PREC = PREC_;    // operands of the two-SM engine
  static constexpr int KV = PREC_ != kTf32 ? 64 : 32;   // k per tile of the two-SM engine
  // kPairs: the operands' records, and all that decide on the form
  const RangeRec *range_a = nullptr, *range_b = nullptr;
  Ranges ranges;
  OpA a;
  OpB b;
  Epilogue epi;
  long M, N, K;
  // split-K: gridDim.z slices of k_per_split (a multiple of the engine's k tile); partial sums go
  // to ws[z][n][m] and a second kernel folds them in slice order and applies the epilogue.
  long k_per_split;
  float *ws;
  // The persistent raw-operand engine splits only the tiles of its last, partly filled round: tiles (m fastest)
  // from tail_first on are cut into tail_splits slices of k_per_split, whose partial sums go to
  // ws[(tile - tail_first) * tail_splits + z][column of the tile][row of the tile] (256 rows); tail_finish_kernel
  // folds them.  Tiles before tail_first run over the whole reduction and store their results themselves.
  long tail_first = 0;
  int tail_splits = 1;
};

// Epilogue of one drain thread: its row m of the tile, NCOL columns from nb on.
template <class P, int NCOL>
__device__ __forceinline__ void tc2_store_rows(const P &p, const float (&acc)[NCOL], long m, long nb) {
  if constexpr (!P::PAIR) {
    // Plain accumulation into a destination whose ROWS are neighbours in memory (column-major gradWeight of a Linear
    // layer: out[m + n * nstride]): 16-byte reductions at the L2.  A thread holds one row and NCOL columns, a 16-byte
    // reduction wants four consecutive rows of one column, so the four lanes of a quad transpose each 4 x 4 block
    // through two rounds of shuffles (every lane of the warp takes part, also those whose row lies past M).  A
    // quarter of the memory-side operations of the per-element form below, which is what bounds a weight gradient
    // with a short reduction.
    if (p.epi.beta == 1.f && !p.epi.bias && p.epi.mdiv >= p.M && (p.epi.nstride & 3) == 0 &&
        nb + NCOL <= p.N && (reinterpret_cast<uintptr_t>(p.epi.out) & 15) == 0) {
      const unsigned full = 0xffffffffu;
      const int i = threadIdx.x & 3;
      const bool b0 = i & 1, b1 = i & 2;
      const long m0 = m - i;                       // first row of this quad; the warp's first row is a multiple of 32
      const bool whole = m0 + 3 < p.M;
      const float alpha = p.epi.alpha;
      const long st = p.epi.nstride;
      float *quad = p.epi.out + m0 + (nb + i) * st;   // (row m0, column nb + i); moff(m) = m since mdiv >= M
#pragma unroll
      for (int c0 = 0; c0 < NCOL; c0 += 4) {
        float a0 = alpha * acc[c0], a1 = alpha * acc[c0 + 1], a2 = alpha * acc[c0 + 2], a3 = alpha * acc[c0 + 3];
        float s0 = b0 ? a0 : a1, s1 = b0 ? a2 : a3;
        float r0 = __shfl_xor_sync(full, s0, 1), r1 = __shfl_xor_sync(full, s1, 1);
        if (b0) { a0 = r0; a2 = r1; } else { a1 = r0; a3 = r1; }
        s0 = b1 ? a0 : a2; s1 = b1 ? a1 : a3;
        r0 = __shfl_xor_sync(full, s0, 2); r1 = __shfl_xor_sync(full, s1, 2);
        if (b1) { a0 = r0; a1 = r1; } else { a2 = r0; a3 = r1; }
        // a_r = alpha * D(row m0 + r, column nb + c0 + i)
        float *dst = quad + (long)c0 * st;
        if (whole) {
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a0), "f"(a1), "f"(a2), "f"(a3) : "memory");
        } else {
          if (m0 < p.M) atomicAdd(dst, a0);
          if (m0 + 1 < p.M) atomicAdd(dst + 1, a1);
          if (m0 + 2 < p.M) atomicAdd(dst + 2, a2);
        }
      }
      return;
    }
  }
  if (m >= p.M) return;
  const long mo = p.epi.template moff<P::PAIR>(m);
  if (!P::PAIR && p.epi.nstride == 1 && nb + NCOL <= p.N &&
             ((reinterpret_cast<uintptr_t>(p.epi.out + mo + nb) & 15) == 0)) {
    // Row-major destination (the columns of a row are neighbours in memory) and this thread's NCOL columns start on
    // a 16-byte boundary: 16-byte loads and stores.  Neighbouring lanes are a whole row apart, so every access of a
    // warp touches 32 lines whatever its width; four columns per access instead of one cuts the number of those
    // accesses by four, which is what a product with a short reduction (an outer-product-like weight gradient)
    // spends its time on.
    float4 *o = reinterpret_cast<float4 *>(p.epi.out + mo + nb);
    const float alpha = p.epi.alpha, beta = p.epi.beta;
    const float *bias = p.epi.bias;
    const float row_b = p.epi.rb(m);
#pragma unroll
    for (int j0 = 0; j0 < NCOL; j0 += 16) {
      float4 old[4];
      float b[16];
      if (beta != 0.f) {
#pragma unroll
        for (int q = 0; q < 4; q++) old[q] = o[j0 / 4 + q];
      }
#pragma unroll
      for (int j = 0; j < 16; j++) b[j] = bias ? __ldg(bias + nb + j0 + j) : row_b;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        float4 v;
        v.x = alpha * acc[j0 + 4 * q + 0] + b[4 * q + 0];
        v.y = alpha * acc[j0 + 4 * q + 1] + b[4 * q + 1];
        v.z = alpha * acc[j0 + 4 * q + 2] + b[4 * q + 2];
        v.w = alpha * acc[j0 + 4 * q + 3] + b[4 * q + 3];
        if (beta != 0.f) {
          v.x += beta * old[q].x; v.y += beta * old[q].y; v.z += beta * old[q].z; v.w += beta * old[q].w;
        }
        o[j0 / 4 + q] = v;
      }
    }
  } else if (p.epi.beta == 0.f) {
    // Measured on the two-SM GEMM: this plain form (one pointer, a constant stride, bias values fetched ahead of
    // the stores) takes 4.7 k cycles for a 128 x 256 tile where a per-column call of Epilogue::store took 23 k.
    const float alpha = p.epi.alpha;
    if (!P::PAIR && nb + NCOL <= p.N) {
      float *o = p.epi.out + mo + nb * p.epi.nstride;
      const long st = p.epi.nstride;
      const float *bias = p.epi.bias;
      const float row_b = p.epi.rb(m);
#pragma unroll
      for (int j0 = 0; j0 < NCOL; j0 += 16) {
        float b[16];
#pragma unroll
        for (int j = 0; j < 16; j++) b[j] = bias ? __ldg(bias + nb + j0 + j) : row_b;
#pragma unroll
        for (int j = 0; j < 16; j++) o[(j0 + j) * st] = alpha * acc[j0 + j] + b[j];
      }
      return;
    }
    if constexpr (P::PAIR) {
      // Pixel-pair mode in 32-bit arithmetic (N = 2 * pair_K <= 128 columns): one base pointer per thread, a
      // 32 x 64-bit product per column.  The general form below spent about 280 cycles per column here.
      float *o0 = p.epi.out + (mo & ~Epilogue::kLastOdd);
      const bool has_odd = !(mo & Epilogue::kLastOdd);
      const int pk = (int)p.epi.pair_K, n_end = (int)p.N, n0 = (int)nb;
      const long st = p.epi.nstride;
      const float *bias = p.epi.bias;
#pragma unroll
      for (int j0 = 0; j0 < NCOL; j0 += 16) {
        float b[16];
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const int n = n0 + j0 + j, plane = n >= pk ? n - pk : n;
          b[j] = (bias && n < n_end) ? __ldg(bias + plane) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const int n = n0 + j0 + j, par = n >= pk ? 1 : 0, plane = n - par * pk;
          if (n < n_end && (has_odd || !par)) o0[(long)plane * st + par] = alpha * acc[j0 + j] + b[j];
        }
      }
      return;
    }
    const float row_b = P::PAIR ? 0.f : p.epi.rb(m);
#pragma unroll
    for (int j0 = 0; j0 < NCOL; j0 += 16) {
      float b[16];
#pragma unroll
      for (int j = 0; j < 16; j++) b[j] = row_b + (nb + j0 + j < p.N ? p.epi.template bias_of<P::PAIR>(nb + j0 + j) : 0.f);
#pragma unroll
      for (int j = 0; j < 16; j++)
        if (nb + j0 + j < p.N) p.epi.template store_biased<P::PAIR>(mo, nb + j0 + j, acc[j0 + j], b[j]);
    }
  } else if (p.epi.beta == 1.f && !p.epi.bias) {
    // Plain accumulation (gradWeight += ...): a reduction performed at the L2 cache per element, with no value
    // coming back, so the thread never waits for the old contents (a product with a short reduction is nothing
    // but this epilogue: fetching 16 old values at a time left it at a fifth of the HBM rate).  Every element is
    // touched once per launch, so the result does not depend on any order; it is the same FP32 add, except that
    // the memory-side adder flushes subnormal operands and results to zero.
    float *o = p.epi.out + mo + nb * p.epi.nstride;
    const long st = p.epi.nstride;
    const float alpha = p.epi.alpha;
#pragma unroll
    for (int j = 0; j < NCOL; j++)
      if (nb + j < p.N) atomicAdd(o + j * st, alpha * acc[j]);
  } else {
    // beta != 0: fetch the old values 16 at a time before any store, so that the loads overlap
#pragma unroll
    for (int j0 = 0; j0 < NCOL; j0 += 16) {
      float old[16];
#pragma unroll
      for (int j = 0; j < 16; j++) old[j] = nb + j0 + j < p.N ? p.epi.out[mo + (nb + j0 + j) * p.epi.nstride] : 0.f;
#pragma unroll
      for (int j = 0; j < 16; j++)
        if (nb + j0 + j < p.N) p.epi.store_with(mo, nb + j0 + j, acc[j0 + j], old[j]);
    }
  }
}


// Pixel-pair epilogue with whole-line stores (pair_K == 64 planes, 128-column tile, no split-K, beta == 0).  The warp
// owns 32 planes in BOTH parities: acc[j] = (parity 0, plane plane0 + j), acc[32 + j] = (parity 1, same plane).  A row
// of the product is a pair of horizontally adjacent output pixels, so a lane's two values of a plane are neighbours
// in memory while neighbouring lanes are two floats apart: stored as they lie, every store instruction would fill
// half of each sector.  Instead the warp transposes through shuffles: in pass k lane l stores parity l & 1 of the
// row that lane 16 k + l / 2 holds, so that the 32 lanes write 32 consecutive floats wherever their rows are
// consecutive pairs of one output row.  Every lane of the warp must call this (rows past M carry m >= p.M).
template <class P>
__device__ __forceinline__ void tc2_store_pair_rows(const P &p, const float (&acc)[64], long m, int plane0) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, par = lane & 1;
  const long long kNone = -1;
  const long long mo = m < p.M ? (long long)p.epi.template moff<true>(m) : kNone;
  const float alpha = p.epi.alpha;
  const long st = p.epi.nstride;
  const float *bias = p.epi.bias;
  float *base[2];
  bool live[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const long long smo = __shfl_sync(full, mo, 16 * k + (lane >> 1));
    live[k] = smo != kNone && !(par && (smo & Epilogue::kLastOdd));
    base[k] = p.epi.out + (smo & ~Epilogue::kLastOdd) + par + (long)plane0 * st;
  }
#pragma unroll
  for (int j0 = 0; j0 < 32; j0 += 8) {
    float b[8];
#pragma unroll
    for (int j = 0; j < 8; j++) b[j] = bias ? __ldg(bias + plane0 + j0 + j) : 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int src = 16 * k + (lane >> 1);
        const float v0 = __shfl_sync(full, acc[j0 + j], src), v1 = __shfl_sync(full, acc[32 + j0 + j], src);
        if (live[k]) base[k][(long)(j0 + j) * st] = alpha * (par ? v1 : v0) + b[j];
      }
    }
  }
}

}  // namespace mm
}  // namespace thc

#endif
