// Host-side dispatch of an mm::Problem onto an engine: picks the tile width, decides split-K,
// owns the split-K workspace, writes the TMA maps, launches, and folds the partials.
#ifndef THC_MM_LAUNCH_CUH
#define THC_MM_LAUNCH_CUH

#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "mm_planes.cuh"
#include "mm_simt.cuh"
#include "mm_small.cuh"
#include "mm_strays.cuh"
#include "mm_tc.cuh"
#include "per_device.h"

namespace thc {
namespace mm {

// How many k slices to cut a product into so that tiles * slices fills whole waves of `slots` concurrent tiles.
// Slicing costs a workspace round trip (slices * M * N floats written and read back), so it needs a clear
// gain: one slice unless the fill of the last wave rises by a quarter; every slice keeps at least 16 k tiles.
static long choose_splits(long tiles, long ktiles, int slots) {
  if (tiles >= 4l * slots || ktiles < 32) return 1;
  auto fill = [&](long s) {
    const long ctas = tiles * s, waves = (ctas + slots - 1) / slots;
    return (double)ctas / (double)(waves * slots);
  };
  long best = 1, max_s = ktiles / 16;
  if (max_s > 256) max_s = 256;
  const double base = fill(1);
  double best_fill = base;
  for (long s = 2; s <= max_s; s++) {
    const double f = fill(s);
    if (f > base * 1.25 && f > best_fill + 0.04) { best = s; best_fill = f; }
  }
  return best;
}

// The FP32 FMA engine.
template <class P>
static void launch_simt(P p) {
  if (p.M <= 0 || p.N <= 0) return;
  THC_CHECK(p.K > 0, "internal: matrix product with empty reduction");
  const long gm = (p.M + SIMT_BM - 1) / SIMT_BM, gn = (p.N + SIMT_BN - 1) / SIMT_BN;
  THC_CHECK(gn <= 65535, "matrix too wide for one launch");
  const long ktiles = (p.K + 31) / 32;
  long splits = choose_splits(gm * gn, ktiles, ctx().sm_count);
  p.ws = nullptr;
  p.k_per_split = p.K;
  if (splits > 1) {
    p.k_per_split = (ktiles + splits - 1) / splits * 32;
    splits = (p.K + p.k_per_split - 1) / p.k_per_split;
  }
  if (splits > 1) p.ws = (float *)ws_alloc(sizeof(float) * splits * p.M * p.N);
  pdl_launch(simt_kernel<P>, dim3((unsigned)gm, (unsigned)gn, (unsigned)splits), 256, 0, p);
  check_launch("simt_kernel");
  if (splits > 1) {
    pdl_launch(splitk_finish_kernel, dim3((unsigned)ceil_div(p.M, 256), (unsigned)(p.N < 32768 ? p.N : 32768)), 256, 0, p.ws, (int)splits, p.M, p.N, p.epi);
    check_launch("splitk_finish");
  }
}

// A driver function through the runtime (no link-time dependency on libcuda); null when the driver lacks it.  The callers keep it in
// a static of their own initialised by this call: a thread that comes while another looks it up waits for the result.
static void *driver_entry(const char *name) {
  void *ptr = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint(name, &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess) return ptr;
  cudaGetLastError();
  return nullptr;
}
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
  static const EncodeTiledFn fn = (EncodeTiledFn)driver_entry("cuTensorMapEncodeTiled");
  return fn;
}
typedef CUresult (*EncodeIm2colFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                   const int *, const int *, cuuint32_t, cuuint32_t, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeIm2colFn encode_im2col_fn() {
  static const EncodeIm2colFn fn = (EncodeIm2colFn)driver_entry("cuTensorMapEncodeIm2col");
  return fn;
}
// Slices for the `tail` tiles a persistent launch has left after its whole rounds over `slots` clusters.  A model in
// microseconds: a k tile step of a lone item takes `tile_us` (1.2; BF16 0.5); a partial-sum block (256 x BN2 floats) costs
// about 0.06 us of device-wide write + read-back, which the L2 holds; the folding kernel, queued as a programmatic
// dependent, 2 us.  Every slice keeps at least three k tiles, the pipeline fill of an item.  (With six tiles, 0.17 and 5 us,
// which fitted launches in ordinary order, products of few tiles left most clusters idle: the small convolution blocks
// 208 -> 202 and 91.7 -> 86.0 us; the VGG-A-style classifier over 13 images moved within its noise, 1.92 - 1.95 ms.)
static int choose_tail_splits(long tail, long ktiles, int slots, double tile_us) {
  int best = 1;
  double best_us = tile_us * (double)ktiles;
  const long max_s = std::min<long>(ktiles / 3, 4l * slots);
  for (long s = 2; s <= max_s; s++) {
    const long rounds = (tail * s + slots - 1) / slots, per = (ktiles + s - 1) / s;
    const double us = tile_us * (double)(rounds * per) + 0.06 * (double)(tail * s) + 2.0;
    if (us < best_us * 0.9) { best = (int)s; best_us = us; }
  }
  return best;
}

// Whether TMA can address a plain FP32 matrix (alignment, pitch).
static bool raw_matrix_ok(const float *base, long ld) {
  return encode_tiled_fn() && ((uintptr_t)base & 15) == 0 && ld % 4 == 0 && ld > 0;
}
// Element (r, k) of the matrix at base[r * ld + k], or base[k * ld + r] for MN; tile_rows: K-major rows per load.
static void encode_matrix(CUtensorMap *map, CUtensorMapDataType type, int size, const void *base, bool mn, long rows, long K, long ld, int tile_rows) {
  const cuuint32_t kv = 128 / (cuuint32_t)size;
  EncodeTiledFn enc = encode_tiled_fn();
  THC_CHECK(enc && ((uintptr_t)base & 15) == 0 && ld * size % 16 == 0, "internal: matrix not addressable by TMA");
  const cuuint64_t dims[2] = {(cuuint64_t)(mn ? rows : K), (cuuint64_t)(mn ? K : rows)};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * size};
  const cuuint32_t box[2] = {kv, mn ? kv : (cuuint32_t)tile_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(map, type, 2, (void *)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         mn && size == 4 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  THC_CHECK(r == CUDA_SUCCESS, "internal: cuTensorMapEncodeTiled failed");
}
// kPairs: `ld` is the padded length of a line's halves, whose FP32 form has that pitch.
template <int PREC, bool MN>
static void attach_raw_map(RawOperand<MN, PREC> &op, const void *base, long rows, long K, long ld, int tile_rows) {
  if constexpr (PREC == kPairs) {
    op.lo = (int)ld;
    encode_matrix(&op.tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, MN, MN ? 2 * ld : rows, MN ? K : 2 * ld, 2 * ld, tile_rows);
    encode_matrix(&op.tmap_wide, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, MN, rows, K, ld, tile_rows);
  } else if (PREC == kBf16) {
    encode_matrix(&op.tmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, MN, rows, K, ld, tile_rows);
  } else {
    encode_matrix(&op.tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, MN, rows, K, ld, tile_rows);
  }
}

// Windows of kH x kW taps on an [oH, oW] grid at strides (dH, dW) under padding (padH, padW), over a channels-last plane
// [N][H][W][C]: what the im2col maps describe.
struct Windows {
  long N, H, W, C, oH, oW;
  int kH, kW, dH, dW, padH, padW;
};
// Corners of the im2col bounding box; false when TMA cannot express them.
static bool window_corners(const Windows &v, int lower[2], int upper[2]) {
  const long up_w = -(long)v.padW + (v.oW - 1) * v.dW - (v.W - 1), up_h = -(long)v.padH + (v.oH - 1) * v.dH - (v.H - 1);
  if (v.padW > 128 || v.padH > 128 || v.padW < -127 || v.padH < -127 || up_w < -128 || up_w > 127 || up_h < -128 || up_h > 127 ||
      v.dW < 1 || v.dW > 8 || v.dH < 1 || v.dH > 8 || v.kH > 200 || v.kW > 200 || v.W >= (1l << 31) || v.H >= (1l << 31))
    return false;
  lower[0] = -v.padW; lower[1] = -v.padH; upper[0] = (int)up_w; upper[1] = (int)up_h;
  return true;
}
static bool windows_ok(const Windows &v) {
  int lo[2], up[2];
  return encode_im2col_fn() && encode_tiled_fn() && v.N < (1l << 30) && v.N * v.oH * v.oW < (1l << 31) && window_corners(v, lo, up);
}
static void set_window_pixels(PixelMap &m, const Windows &v) {
  m.set(v.N * v.oH * v.oW, v.oH * v.oW, v.oW);
  m.img_stride = m.y_stride = m.x_stride = m.off0 = 0;   // the TMA map knows the memory
  m.sy = v.dH; m.y0 = -v.padH; m.sx = v.dW; m.x0 = -v.padW;
}
static void encode_windows(CUtensorMap *map, CUtensorMapDataType type, int size, const void *base, const Windows &v, long C, int windows_per_load,
                           bool mn) {
  const int kv = 128 / size;
  EncodeIm2colFn enc = encode_im2col_fn();
  int lower[2], upper[2];
  THC_CHECK(enc && C % kv == 0 && ((uintptr_t)base & 15) == 0 && window_corners(v, lower, upper), "internal: windows not addressable by TMA");
  const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)v.W, (cuuint64_t)v.H, (cuuint64_t)v.N};
  const cuuint64_t strides[3] = {(cuuint64_t)C * size, (cuuint64_t)v.W * C * size, (cuuint64_t)v.H * v.W * C * size};
  const cuuint32_t estr[4] = {1, (cuuint32_t)v.dW, (cuuint32_t)v.dH, 1};
  const CUresult r = enc(map, type, 4, (void *)base, dims, strides, lower, upper, (cuuint32_t)kv, (cuuint32_t)windows_per_load, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, mn && size == 4 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  THC_CHECK(r == CUDA_SUCCESS, "internal: cuTensorMapEncodeIm2col failed");
}
// The maps of an operand of windows; per load `per` windows, or as many as a span has values (mn).
template <int PREC, class Op>
static void attach_windows(Op &op, const void *base, const Windows &v, int per, bool mn) {
  op.n_img = (int)v.N;
  if constexpr (PREC == kPairs) {
    op.lo = (int)v.C;
    encode_windows(&op.tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, v, 2 * v.C, mn ? 64 : per, mn);
    encode_windows(&op.tmap_wide, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, v, v.C, mn ? 32 : per, mn);
  } else if (PREC == kBf16) {
    encode_windows(&op.tmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, v, v.C, mn ? 64 : per, mn);
  } else {
    encode_windows(&op.tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, v, v.C, mn ? 32 : per, mn);
  }
}
template <int PREC>
static void attach_window_map(PlanesWindowOperand<PREC> &op, const void *base, const Windows &v) {
  set_window_pixels(op.rows, v);
  op.C = FastDiv::make(v.C); op.kW = FastDiv::make(v.kW);
  attach_windows<PREC>(op, base, v, TC_BM, false);
}
template <int PREC>
static void attach_window_rows_map(WindowRowsOperand<PREC> &op, const void *base, const Windows &v) {
  set_window_pixels(op.ks, v);
  op.C = FastDiv::make(v.C); op.kW = FastDiv::make(v.kW);
  op.oH = (int)v.oH;
  for (int i = 0; i < 2; i++) {
    const long n = 32l << i, P = v.oH * v.oW;
    op.step[i] = WindowStep{(int)(n % P % v.oW), (int)(n % P / v.oW), (int)(n / P)};
  }
  attach_windows<PREC>(op, base, v, 0, true);
}

// Width of the two-SM tile that pads N least (wider wins ties).  An MN-major 16-bit operand on the N side comes in blocks of
// 64 rows per CTA, which leaves 256 and 128.
static int tc2_tile_width(long N, bool half_mn = false) {
  int best = 0;
  long best_pad = 0;
  const int widths[4] = {256, 192, 128, 64};
  for (int w : widths) {
    if (half_mn && w % 128 != 0) continue;
    const long pad = (N + w - 1) / w * w;
    if (!best || pad < best_pad) { best = w; best_pad = pad; }
  }
  return best;
}
// Microseconds a cluster takes for one k tile of a tile of this width, as the convolution and addmm launches at full size showed it when one
// thread issued the MMAs.  Narrow tiles are faster since (pairs at 128 columns 0.6, see elect_one); the choices made by these values were within 2 % of the
// better form when forms were forced, and other values move the bounds of k slices and with them the last bits of results.
static double tc2_tile_us(int bn2, int prec) {
  if (prec == kBf16) return bn2 == 256 ? 0.55 : bn2 == 192 ? 0.47 : 0.4;
  if (prec == kPairs) return bn2 == 256 ? 1.3 : bn2 == 192 ? 1.1 : bn2 == 128 ? 0.9 : 0.8;
  return bn2 == 256 ? 1.25 : bn2 == 192 ? 1.0 : bn2 == 128 ? 0.79 : 0.7;
}
// Model of a product's time, for choices between ways of stating it.
static double tc2_product_us(long M, long N, long K, int prec, bool mn = false) {
  const int w = tc2_tile_width(N, prec != kTf32 && mn), kv = prec != kTf32 ? 64 : 32;
  const double tiles = (double)((M + 255) / 256) * (double)((N + w - 1) / w), ktiles = (double)((K + kv - 1) / kv);
  // a tile's epilogue and hand-over take about as long as two k tiles; a tile cut along k keeps at least six
  return std::max(tiles * (ktiles + 2) / (ctx().sm_count / 2), std::min(ktiles, 6.0) + 2) * tc2_tile_us(w, prec) + 8;
}

// The two-SM kernel (mm_tc2r.cuh) is compiled in files of its own, mm_tc2r_*.cu, which list the problems and tile widths there are.
// Clusters that the device runs at once (the kernel is persistent: a launch has no more), and a launch of `items` work items.
template <class P, int BN2> int tc2r_resident_clusters();
template <class P, int BN2> void launch_tc2r_kernel(const P &p, long items, bool early);

// Products over operands that TMA can fetch.  `attach(p, bn2)` writes the operands' tensor maps for the chosen tile width.
template <class P, class Attach>
static void launch_raw(P p, Attach attach) {
  if (p.M <= 0 || p.N <= 0) return;
  THC_CHECK(p.K > 0, "internal: matrix product with empty reduction");
  constexpr bool HALF_MN = P::PREC != kTf32 && P::OpB::MN_MAJOR;
  const int bn2 = tc2_tile_width(p.N, HALF_MN);
  attach(p, bn2);
  const long gm = (p.M + 255) / 256, gn = (p.N + bn2 - 1) / bn2, tiles = gm * gn;
  int slots = 0;
  // the widths a problem can come to: 16-bit MN-major 256 and 128, pixel pairs (at most 128 columns) 128 and 64, gathered windows 64
  auto with_width = [&](auto f) {
    if constexpr (!P::OpA::GATHERED)
      if (bn2 == 128) { f(std::integral_constant<int, 128>()); return; }
    if constexpr (!P::PAIR && !P::OpA::GATHERED) {
      if (bn2 == 256) { f(std::integral_constant<int, 256>()); return; }
      if constexpr (!HALF_MN)
        if (bn2 == 192) { f(std::integral_constant<int, 192>()); return; }
    }
    if constexpr (!HALF_MN)
      if (bn2 == 64) { f(std::integral_constant<int, 64>()); return; }
    fail("internal: tile width %d for a problem that has none", bn2);
  };
  with_width([&](auto w) { slots = tc2r_resident_clusters<P, decltype(w)::value>(); });
  const long ktiles = (p.K + P::KV - 1) / P::KV;
  // Every cluster first runs tiles / slots whole tiles; the remaining `tail` tiles (all of them when there are fewer
  // tiles than clusters) are cut along k so that they fill the clusters once more instead of leaving most idle.
  // BF16 products over K-major operands (whose results the next layer rounds to BF16 again) cut every tile alike, so that no
  // element's rounding depends on the tile it falls in.
  constexpr bool EVEN = P::PREC == kBf16 && !P::OpB::MN_MAJOR;
  const long tail = EVEN ? tiles : tiles % slots;
  const int splits = EVEN ? (int)choose_splits(tiles, ktiles, ctx().sm_count / 2) : tail ? choose_tail_splits(tail, ktiles, slots, P::PREC == kBf16 ? 0.5 : 1.2) : 1;
  p.ws = nullptr;
  p.k_per_split = p.K;
  p.tail_first = tiles;
  p.tail_splits = 1;
  if (splits > 1) {
    const long per = (ktiles + splits - 1) / splits;
    p.k_per_split = per * P::KV;
    p.tail_splits = (int)((p.K + p.k_per_split - 1) / p.k_per_split);
  }
  if (p.tail_splits > 1) {
    p.tail_first = tiles - tail;
    p.ws = (float *)ws_alloc(sizeof(float) * tail * p.tail_splits * bn2 * 256);
  }
  const long items = p.tail_first + (tiles - p.tail_first) * p.tail_splits;
  THC_CHECK(items < (1l << 31) - 4096, "matrix product with too many tiles for one launch");
  // a long launch gains nothing from starting early, and measured 1.5 % slower when it did (4096^3: 671 -> 682 us)
  const bool early = tc2_product_us(p.M, p.N, p.K, P::PREC, P::OpB::MN_MAJOR) < 100;
  with_width([&](auto w) { launch_tc2r_kernel<P, decltype(w)::value>(p, items, early); });
  ctx().products[P::PREC]++;
  if (p.ws) {
    // a few thousand blocks whatever the number of tail tiles: a lone tile cut into many slices gets a block per column
    const bool four = tail * (bn2 / 4) >= 2l * ctx().sm_count;
    const long blocks = ceil_div(8l * ctx().sm_count, tail), by = four ? std::min<long>(bn2 / 4, std::max<long>(16, blocks)) : std::min<long>(bn2, std::max<long>(32, blocks));
    pdl_launch(four ? tail_finish_kernel<4> : tail_finish_kernel<1>, dim3((unsigned)tail, (unsigned)by), 256, 0, p.ws, p.tail_splits, bn2, p.tail_first, gm, p.M, p.N,
               p.epi);
    check_launch("tail_finish");
  }
}

// ---- small and narrow products (mm_small.cuh) ----------------------------------------------------------------------
template <int BN, int WM, int WN, bool A_K, bool B_K>
static void launch_small_kernel(const SmallProblem &p) {
  constexpr int BM = 64, SMEM = SM_STAGES * (SmallTile<BM, A_K>::FLOATS + SmallTile<BN, B_K>::FLOATS) * 4;
  static thread_local int configured_for = -1;
  if (SMEM > 47 * 1024 && configured_for != ctx().device) {
    THC_CUDA(cudaFuncSetAttribute(small_kernel<BM, BN, WM, WN, A_K, B_K>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    configured_for = ctx().device;
  }
  const dim3 grid((unsigned)ceil_div(p.M, BM), (unsigned)ceil_div(p.N, BN), (unsigned)p.slices);
  pdl_launch(small_kernel<BM, BN, WM, WN, A_K, B_K>, grid, SM_THREADS, SMEM, p);
  check_launch("small_kernel");
}
template <int BN, int WM, int WN>
static void launch_small_layout(const SmallProblem &p, bool a_k, bool b_k) {
  if (a_k && b_k) launch_small_kernel<BN, WM, WN, true, true>(p);
  else if (a_k) launch_small_kernel<BN, WM, WN, true, false>(p);
  else if (b_k) launch_small_kernel<BN, WM, WN, false, true>(p);
  else launch_small_kernel<BN, WM, WN, false, false>(p);
}
inline SmallOperand small_operand(const float *base, long ld) {
  return SmallOperand{base, ld, ((uintptr_t)base & 15) == 0 && ld % 4 == 0 ? 1 : 0};
}
inline int small_tile_width(long n) { return n <= 8 ? 8 : n <= 16 ? 16 : n <= 32 ? 32 : 64; }
// k slices of a product of `tiles` 64 x bn tiles: until the tiles fill the device as deep as registers and shared memory
// allow, each at least two k tiles, and not so many that the block that folds them, one after the other, takes longer than
// a slice's own k tiles.
inline long small_slices(long tiles, long ktiles, int bn) {
  const long depth = bn == 64 ? 3 : bn == 8 ? 5 : 4;
  const long fold = (long)std::sqrt((double)ktiles * 64 / bn);
  return std::max(1l, std::min(std::min(depth * ctx().sm_count / tiles, ktiles / 2), std::min(fold, 32l)));
}
// Its time in microseconds, as measured for m, n, k in 1 .. 4096: a k tile takes a block longer the more blocks share its SM.
inline double small_product_us(long m, long n, long k, bool aligned) {
  const long lo = std::min(m, n), hi = std::max(m, n), ktiles = ceil_div(k, TC_BK);
  const int bn = small_tile_width(lo), depth = bn == 64 ? 3 : bn == 8 ? 5 : 4;
  const long tiles = (long)ceil_div(hi, 64) * ceil_div(lo, bn), slices = small_slices(tiles, ktiles, bn);
  const double blocks = (double)(tiles * slices) / ctx().sm_count, resident = std::min(blocks, (double)depth);
  const double step = bn == 64 ? 1.35 + 0.4 * resident : bn == 32 ? 1.3 + 0.15 * resident : bn == 16 ? 0.6 + 0.15 * resident : 0.45 + 0.15 * resident;
  const double waves = std::max(1.0, blocks / depth);
  return 5 + (aligned ? 1.0 : 1.3) * step * waves * (double)((ktiles + slices - 1) / slices) + (slices > 1 ? 0.25 * (double)slices : 0);
}
// few_rows_kernel, for both operands along k in whole 16-byte pieces: up to 4 rows on the short side, and up to 8 while the
// matrix stays in L2 many times over (a 4096 x 1000 one: 12.8 -> 9 us); beyond, the reads of the rows outweigh those
// of the matrix and the MMA tiles win (8 rows against 4096 x 9216: 43 us, here 53).
static bool launch_few_rows(const SmallProblem &p, bool a_k, bool b_k) {
  if (!(a_k && b_k && p.a.vec4 && p.b.vec4 && p.K % 4 == 0 && p.K <= 1 << 30 && p.N <= 8 && (p.N <= 4 || (long)p.M * p.K <= 1l << 23))) return false;
  const int ra = p.N == 1 || (p.N > 2 && p.N <= 4) ? 4 : 8;
  int groups = 8;   // sets of rows per block: as many as leave two blocks per SM, since they share the few rows
  while (groups > 1 && ceil_div(p.M, ra * groups) < 2 * ctx().sm_count) groups /= 2;
  const unsigned blocks = (unsigned)ceil_div(p.M, ra * groups);
  if (p.N == 1) pdl_launch(few_rows_kernel<1, 4, 2>, blocks, 256, 0, p, groups);
  else if (p.N == 2) pdl_launch(few_rows_kernel<2, 8, 2>, blocks, 256, 0, p, groups);
  else if (p.N <= 4) pdl_launch(few_rows_kernel<4, 4, 3>, blocks, 256, 0, p, groups);
  else pdl_launch(few_rows_kernel<8, 8, 1>, blocks, 256, 0, p, groups);
  check_launch("few_rows");
  return true;
}
// D = alpha * A * B^T + beta * D (+ bias) for A [M][K] and B [N][K]; a_k / b_k: the operand's memory runs along k.
static void launch_small(SmallProblem p, bool a_k, bool b_k) {
  if (p.N > p.M) {   // the longer side takes the 64-row tiles
    std::swap(p.a, p.b); std::swap(a_k, b_k); std::swap(p.M, p.N); std::swap(p.sm, p.sn); std::swap(p.bias_m, p.bias_n);
  }
  p.stalled = stall_ctl().dev_flag;
  if (launch_few_rows(p, a_k, b_k)) return;
  const int bn = small_tile_width(p.N);
  const long tiles = (long)ceil_div(p.M, 64) * ceil_div(p.N, bn), ktiles = ceil_div(p.K, TC_BK), slices = small_slices(tiles, ktiles, bn);
  p.tiles_per_slice = ceil_div(ktiles, slices);
  p.slices = ceil_div(ktiles, p.tiles_per_slice);
  if (p.slices > 1) {
    p.ws = (float *)ws_alloc(sizeof(float) * tiles * p.slices * 64 * bn);
    p.tickets = zero_words();
  }
  if (bn == 8) launch_small_layout<8, 4, 1>(p, a_k, b_k);
  else if (bn == 16) launch_small_layout<16, 4, 1>(p, a_k, b_k);
  else if (bn == 32) launch_small_layout<32, 4, 1>(p, a_k, b_k);
  else launch_small_layout<64, 2, 2>(p, a_k, b_k);
}

template <class Main, class First = NoPass, class Second = NoPass>
static void launch_passes(const Main &main, size_t smem, const char *what, const First &first = {}, const Second &second = {}) {
  const unsigned blocks = main.blocks + first.blocks + second.blocks;
  if (!blocks) return;
  pdl_launch(passes_kernel<Main, First, Second>, blocks, 256, smem, main, first, second);
  check_launch(what);
}
// Channels-last planes of an NCHW activation tensor (or its cells), FP32 or BF16.
struct ActPlanes {
  void *p = nullptr;
  long N = 0, H = 0, W = 0, Cp = 0;
  // per-channel sums of the transposed tensor, when asked for: [chan_blocks][C] partials (see PlanesPass)
  float *chan_partial = nullptr;
  int chan_blocks = 0;
};
static long padded_channels(long C, int prec) { return prec != kTf32 ? (C + 63) / 64 * 64 : (C + 31) / 32 * 32; }
static size_t planes_bytes(long N, long HW, long Cp, int prec) { return (size_t)N * HW * Cp * (prec == kBf16 ? 2 : 4); }
// Tiles of 128 pixels.  (BF16 with sums: 64, whose sums are as they always were.)
template <int PREC, bool SUMS>
static bool wide_tile(long HW) {
  return PREC == kTf32 || ((PREC == kPairs || !SUMS) && (HW + 127) / 128 * 128 * 10 <= (HW + 63) / 64 * 64 * 11);
}
// Channels whose sums fit next to the tile in 48 KB: 4096 is a width that layers have, and their sums are a pass over gradOutput otherwise
// (weight gradient of 4096 x 512 x 1 x 1 over 64 images of 13 x 13: 192 -> 165 us in BF16, 309 -> 281 FP32-accurate; of 3968 planes 162 and 277).
template <int PREC>
static long most_sums(long HW) { return PREC != kTf32 && wide_tile<PREC, true>(HW) ? 3968 : 4096; }
// `dst`: room for planes_bytes(), or null for workspace.  `form`: kPairs.  `first`, `second`: passes that share the launch.
template <int PREC, bool SUMS, class First, class Second>
static ActPlanes make_act_planes(const float *src, long N, long C, long H, long W, void *dst, const PairForm &form, const First &first, const Second &second) {
  ActPlanes ap;
  const long HW = H * W;
  ap.N = N; ap.H = H; ap.W = W; ap.Cp = padded_channels(C, PREC);
  ap.p = dst ? dst : ws_alloc(planes_bytes(N, HW, ap.Cp, PREC));
  const bool wide = wide_tile<PREC, SUMS>(HW);
  const long cap = ctx().sm_count * 16l, needed = N * ((HW + (wide ? 127 : 63)) / (wide ? 128 : 64)) * (ap.Cp / (PREC != kTf32 ? 64 : 32));
  long blocks = std::min(needed, cap);
  size_t smem = 0;
  if (SUMS) {
    // every block leaves a row of per-channel sums to fold, which on a small tensor (a few tiles per block) costs as much as the
    // transposition: a quarter of the blocks keeps it short; a large one wants all its blocks (at 1024 images the same cut cost it 3 %)
    if (needed <= 4 * cap && blocks > cap / 4) blocks = cap / 4;
    ap.chan_blocks = (int)blocks;
    ap.chan_partial = (float *)ws_alloc(sizeof(float) * blocks * C);
    smem = sizeof(float) * C;
  }
  auto go = [&](auto pt) {
    launch_passes(PlanesPass<PREC, decltype(pt)::value, SUMS>{(unsigned)blocks, src, N, (int)C, (int)HW, (int)ap.Cp, ap.p, ap.chan_partial, form}, smem, "nchw_to_planes", first,
                  second);
  };
  if constexpr (PREC == kTf32) go(std::integral_constant<int, 128>());
  else if (wide) go(std::integral_constant<int, 128>());
  else go(std::integral_constant<int, 64>());
  return ap;
}

// ---- FP16 pairs -------------------------------------------------------------------------------------------------------
// A zeroed record for range_kernel, and room for its list.
static Measured new_measured() { return Measured{(RangeRec *)zeroed_words(kRangeWords), (Stray *)ws_alloc(sizeof(Stray) * kStrays)}; }
// Neighbours in memory are neighbours along a line wherever lines are long or lie apart.
static RangeJob range_job(const float *p, long lines, long run, long ld, const Measured &m) {
  const bool flat = (ld == run || lines == 1) && (lines < 4 || run < 64);
  return RangeJob{p, lines, run, ld, flat, ((uintptr_t)p & 15) == 0 && (flat || ld % 4 == 0), m.rec, m.list, 0, nullptr, nullptr};
}
static RangeJob range_job_flat(const float *p, long n, const Measured &m) { return range_job(p, 1, n, n, m); }
static void launch_ranges(RangeJob a, RangeJob *b) {
  auto sets = [](const RangeJob &j) { return j.flat ? (j.lines * j.run + 511) / 512 : (j.run + 127) / 128 * ((j.lines + 3) / 4); };
  dim3 grid(1, b ? 2 : 1);
  for (RangeJob *j : {&a, b})
    if (j) {
      j->blocks = (unsigned)std::max(1l, std::min((sets(*j) + 7) / 8, std::min(ctx().sm_count * 5l, (long)kRangeBlocks)));
      j->block_range = (uint2 *)ws_alloc(sizeof(uint2) * j->blocks + sizeof(unsigned) * sets(*j));
      j->set_low = (unsigned *)(j->block_range + j->blocks);
      grid.x = std::max(grid.x, j->blocks);
    }
  pdl_launch(range_kernel, grid, 256, 0, a, b ? *b : a);
  check_launch("range");
}

// One BF16 plane of a strided matrix, rows padded to 64 values.
struct HalfMatrix {
  __nv_bfloat16 *p = nullptr;
  long ld = 0;
};
static HalfMatrix make_half_matrix(const float *src, long rs, long ks, long rows, long K) {
  HalfMatrix hm;
  hm.ld = (K + 63) / 64 * 64;
  hm.p = (__nv_bfloat16 *)ws_alloc(sizeof(__nv_bfloat16) * rows * hm.ld);
  const long blocks = std::min(((rows + 63) / 64) * (hm.ld / 64), (long)ctx().sm_count * 16);
  pdl_launch(bf16_rows_kernel, (unsigned)blocks, 256, 0, src, rs, ks, rows, K, hm.p, hm.ld);
  check_launch("bf16_rows");
  return hm;
}

}  // namespace mm
}  // namespace thc

#endif
