// nn.SpatialConvolutionMM on torch.GPUTensor: forward, gradInput, gradParameters.
//
// The reference (gputorch/lib/THC/gpunn-impl/SpatialConvolutionMM.cpp: updateOutput :110-225,
// updateGradInput :227-311, accGradParameters :313-429) loops over the images of a batch on the
// host and, per image, launches im2col / col2im and a 16x16-tile SGEMM.  Here each pass is one
// implicit-GEMM product over the whole batch: the activations are brought into channels-last form once per
// call, from which the tensor-core engine's TMA loads fetch the windows (the FP32 FMA engine gathers them
// from the NCHW tensor element by element).  Results follow the CPU nn semantics
// (mcw_nn/generic/SpatialConvolutionMM.c) and also cover dW/dH > 1, which the CPU MM path rejects
// (:148-149) and the reference GPU path supports.
#include "mm_launch.cuh"

#include <unordered_map>
#include <utility>
#include <vector>

namespace thc {

struct ConvGeom {
  long N, C, H, W, K, oH, oW, P, R;
  int kH, kW, dH, dW, pad;
  bool batch;
};

static ConvGeom conv_geom(const THGPUTensor *input, const THGPUTensor *weight, int kW, int kH, int dW, int dH, int padding) {
  THC_ARG(input->nDimension == 3 || input->nDimension == 4, 2, "3D or 4D (batch mode) tensor is expected");
  THC_ARG(kW > 0 && kH > 0 && dW > 0 && dH > 0 && padding >= 0, 1, "invalid kernel / stride / padding");
  THC_ARG(weight->nDimension == 2, 1, "weight must be 2D (nOutputPlane x nInputPlane*kH*kW)");
  ConvGeom g;
  g.batch = input->nDimension == 4;
  const int o = g.batch ? 1 : 0;
  g.N = g.batch ? input->size[0] : 1;
  g.C = input->size[o];
  g.H = input->size[o + 1];
  g.W = input->size[o + 2];
  g.K = weight->size[0];
  g.kH = kH; g.kW = kW; g.dH = dH; g.dW = dW; g.pad = padding;
  g.R = g.C * kH * kW;
  THC_ARG(weight->size[1] == g.R, 2, "input channels and nInputPlane dont match");
  THC_ARG(g.H + 2 * padding >= kH && g.W + 2 * padding >= kW, 2, "input image smaller than kernel size");
  g.oH = (g.H + 2 * padding - kH) / dH + 1;
  g.oW = (g.W + 2 * padding - kW) / dW + 1;
  g.P = g.oH * g.oW;
  THC_CHECK(g.C * g.H * g.W < (1l << 31) && g.K * g.P < (1l << 31), "image too large");
  return g;
}

// What the planes kept in a module's `finput` were made from.  accGradParameters reuses them only when it is
// handed the very input (same device memory, same layer and precision) that the forward pass transposed; every forward pass
// begins by forgetting the entry, so that planes of an earlier pass are never taken for those of one that does not write `finput`,
// or that fails: what the input's memory holds may have changed since.
// Keyed by the address of finput's data; one table per host thread, as the rest of the library's state.
namespace {
// Pairs have a record (mm::KeptRange), `record` of the context's (plane_record); the slots belong to the entries of this table.
struct PlaneStamp { const float *input; int prec; long N, C, H, W, K; int kH, kW, dH, dW, pad; int record; long epoch; };
thread_local std::unordered_map<const float *, PlaneStamp> g_plane_stamps;
thread_local std::vector<int> g_free_records;   // of the slots below g_records
thread_local int g_records = 0;
void stamp_planes(const THGPUTensor *finput, const float *input, const ConvGeom &g, int prec) {
  if (!finput || !finput->storage) return;
  int record = -1;
  if (g_plane_stamps.size() >= kPlaneRecords) { g_plane_stamps.clear(); g_free_records.clear(); g_records = 0; }
  if (prec == mm::kPairs) {
    if (g_free_records.empty()) record = g_records++;
    else { record = g_free_records.back(); g_free_records.pop_back(); }
    plane_record(record);   // there before the entry is
  }
  g_plane_stamps[data_ptr(finput)] = PlaneStamp{input, prec, g.N, g.C, g.H, g.W, g.K, g.kH, g.kW, g.dH, g.dW, g.pad, record, ctx().plane_epoch};
}
void forget_planes(const THGPUTensor *finput) {
  if (!finput || !finput->storage) return;
  auto it = g_plane_stamps.find(data_ptr(finput));
  if (it == g_plane_stamps.end()) return;
  if (it->second.record >= 0) g_free_records.push_back(it->second.record);
  g_plane_stamps.erase(it);
}
// Planes that are marked as made ahead of the launch that makes them: not any more, should that launch not come about.
struct UnmadePlanes {
  const THGPUTensor *finput;
  ~UnmadePlanes() { forget_planes(finput); }
};
// The record of planes that are known to be fresh.
mm::KeptRange *planes_record(const void *planes) { return (mm::KeptRange *)plane_record(g_plane_stamps.at((const float *)planes).record); }
}  // namespace

// ------------------------------------------------------------------------------------------------
// Tensor-core passes.  The activations are brought into channels-last form once per call (planes, or cells: see mm::Cells),
// channel counts padded to whole swizzle spans, after which every operand tile of the three products is one TMA load.

static mm::Cells cells_of(const ConvGeom &g, bool unfoldH, bool unfoldW, int prec) {
  mm::Cells u;
  u.C = (int)g.C; u.kH = g.kH; u.kW = g.kW; u.dH = g.dH; u.dW = g.dW; u.pad = g.pad; u.H = (int)g.H; u.W = (int)g.W;
  u.eH = unfoldH ? g.kH : std::min(g.dH, g.kH); u.eW = unfoldW ? g.kW : std::min(g.dW, g.kW);
  u.kHs = unfoldH ? 1 : (g.kH + g.dH - 1) / g.dH; u.kWs = unfoldW ? 1 : (g.kW + g.dW - 1) / g.dW;
  u.stepH = g.dH; u.stepW = g.dW;
  const int e = u.eH * u.eW, q4 = (u.C + 3) / 4 * 4;
  u.Cq = mm::padded_channels(e * q4, prec) == mm::padded_channels(e * u.C, prec) ? q4 : u.C;
  u.Cr = e * u.Cq; u.Cs = (int)mm::padded_channels(u.Cr, prec);
  u.Hs = (int)g.oH + u.kHs - 1; u.Ws = (int)g.oW + u.kWs - 1;
  u.direct = false;
  return u;
}
static mm::Cells direct_cells(const ConvGeom &g, int prec) {
  mm::Cells u = cells_of(g, false, false, prec);
  u.eH = u.eW = 1; u.kHs = g.kH; u.kWs = g.kW; u.stepH = u.stepW = 1;
  u.Cq = u.Cr = u.C; u.Cs = (int)mm::padded_channels(u.C, prec);
  u.Hs = (int)g.H; u.Ws = (int)g.W;
  u.direct = true;
  return u;
}
// The layer's windows over its restated input.
static mm::Windows forward_windows(const ConvGeom &g, const mm::Cells &u) {
  return mm::Windows{g.N, u.Hs, u.Ws, u.Cs, g.oH, g.oW, u.kHs, u.kWs, u.direct ? g.dH : 1, u.direct ? g.dW : 1, u.direct ? g.pad : 0,
                     u.direct ? g.pad : 0};
}

// A tcgen05.mma occupies the tensor pipe about 80 cycles however narrow it is, so with up to 64 output planes two horizontally
// adjacent output pixels share a row of the product (pixel-pair mode): half the rows, twice the columns, a window one
// stride wider.  Worth it when the wider window costs less than the rows save; not for windows of one column.
// FP32 only: BF16 products are bound by their operands' bytes, which the wider window adds to.
static bool pair_windows(const mm::Windows &v, long Kout, int prec, mm::Windows &p) {
  if (prec == mm::kBf16) return false;
  p = v;
  p.oW = (v.oW + 1) / 2; p.dW = 2 * v.dW; p.kW = v.kW + v.dW;
  return Kout <= 64 && Kout > 16 && v.oW >= 2 && 4 * p.kW <= 7 * v.kW && v.N * v.oH * p.oW > 128 && mm::windows_ok(p);
}
static double windows_us(const mm::Windows &v, long Kout, int prec) {
  mm::Windows p;
  if (pair_windows(v, Kout, prec, p)) return mm::tc2_product_us(p.N * p.oH * p.oW, 2 * Kout, (long)p.kH * p.kW * p.C, prec);
  return mm::tc2_product_us(v.N * v.oH * v.oW, Kout, (long)v.kH * v.kW * v.C, prec);
}

// Scratch of a pass.  A layer over one plane is restated over 32 channels, so a batch of a few GB may come to planes of a hundred:
// such batches are taken in groups of images, shared out evenly, whose planes are used and given up one after the other.  A
// group of kGroupScratch bytes is still some hundred tiles, many more than there are clusters, so that nothing is lost on
// whole rounds and no BF16 tile is cut where it was not before.
constexpr double kGroupScratch = 2e9, kImageScratch = 64e9;
// Images per group of a batch whose planes take `bytes` an image, when the whole may have `allowed`.
static long images_per_group(long N, double bytes, double allowed) {
  if (bytes * (double)N <= allowed) return N;
  const long fit = std::max(1l, (long)(kGroupScratch / bytes)), groups = (N + fit - 1) / fit;
  return (N + groups - 1) / groups;
}
// What planes may take in one piece: twice the tensors they restate, which is no blow-up, or a tenth of the device.
static double whole_scratch(double floats) { return std::max(16e9, 2 * 4 * floats); }

// How a layer is restated for its forward and weight-gradient products: the form that costs least by the model of the product's
// time plus one pass that writes it and one that reads it back for the weight gradient (5 TB/s).  Channel counts that
// are multiples of a swizzle span stay direct; few planes become cells, in the extreme (3 planes, 3 x 3) columns, because
// padding 3 planes to 32 would multiply the products tenfold.  False: no form that TMA can express.
static bool restate(const ConvGeom &g, int prec, mm::Cells &best) {
  if (g.K * g.R >= (1l << 31) || g.N * g.P >= (1l << 31)) return false;
  double best_us = 0;
  bool found = false;
  if (prec == mm::kBf16 && g.C <= 8 && (long)g.kH * g.kW * 8 <= 6144) {
    // Few planes in BF16: the column matrix with eight planes per tap, k = (tap, plane).  The reduction keeps that order
    // because a step in this mode rounds every layer's result to BF16 again, which turns a different order's last bit into
    // other masks and maxima further up.
    best = cells_of(g, true, true, mm::kBf16);
    best.Cq = 8;
    best.Cr = best.eH * best.eW * 8; best.Cs = (int)mm::padded_channels(best.Cr, mm::kBf16);
    if (mm::windows_ok(forward_windows(g, best)) && (double)mm::planes_bytes(1, g.P, best.Cs, mm::kBf16) < kImageScratch) return true;
  }
  // Forms of more channels than the table of CellsPass holds only where there is no other: strides beyond the eight
  // that a window map takes, over many planes, and windows beyond 128 taps (as columns).  64 planes under 16 x 16 / 16, 16 images:
  // 300 us forward and 155 for the weight gradient, 1911 and 1870 on the FMA engine; 131 x 131 taps over 16 planes: 6.6 and
  // 2.2 ms, 13.6 and 11.9 there.
  for (const long most : {(long)mm::kCellTable, 1l << 28}) {
    for (int o = 0; o < 5; o++) {
      if (o > 0 && g.N * g.oH >= (1l << 31)) continue;
      if ((o == 1 && g.dH == 1 && g.dW == 1) || (o == 2 && g.kW == 1) || (o == 3 && g.kH == 1)) continue;   // the same as another
      if (o && g.dH * (long)g.kH * g.dW * g.kW * g.C > (1l << 28)) continue;
      const mm::Cells u = o == 0 ? direct_cells(g, prec) : cells_of(g, o >= 3, o == 2 || o == 4, prec);
      if (o > 0 && (u.Cs > most || (long)u.Ws * u.Cs >= (1l << 31))) continue;
      const mm::Windows v = forward_windows(g, u);
      const double bytes = (double)mm::planes_bytes(g.N, (long)u.Hs * u.Ws, u.Cs, prec);
      if (!mm::windows_ok(v) || bytes > (double)g.N * kImageScratch) continue;
      const double us = windows_us(v, g.K, prec) + 2 * bytes / 5e6;
      if (!found || us < best_us) { best = u; best_us = us; found = true; }
      if (o == 0 && u.Cs == u.C) break;   // nothing is padded
    }
    if (found) break;
  }
  return found;
}

// Whether the gradInput product can be stated: over gradOutput's planes, stride 1 as it is, strided layers through the folded
// cells (their gradient, brought back by unfold_grad_input_kernel).
static mm::Windows grad_input_windows(const ConvGeom &g, const mm::Cells &u, int prec) {
  const int padH = u.direct ? g.kH - 1 - g.pad : u.kHs - 1, padW = u.direct ? g.kW - 1 - g.pad : u.kWs - 1;
  return mm::Windows{g.N, g.oH, g.oW, mm::padded_channels(g.K, prec), u.direct ? g.H : u.Hs, u.direct ? g.W : u.Ws, u.kHs, u.kWs, 1, 1, padH, padW};
}
static mm::Cells grad_input_cells(const ConvGeom &g, int prec) {
  return g.dH == 1 && g.dW == 1 ? direct_cells(g, prec) : cells_of(g, false, false, prec);
}

// kPairs: the measures of the tensors that a call's products read, whose form is decided together (mm::RangeRec).
struct Records {
  mm::Measured act, weight, gout;
  // `own` first, then the others
  mm::Ranges joint(const mm::Measured &own) const {
    mm::Ranges r;
    int n = 0;
    r.rec[n++] = own.rec;
    for (const mm::RangeRec *x : {act.rec, weight.rec, gout.rec})
      if (x != own.rec) r.rec[n++] = x;
    return r;
  }
};
static mm::LayerShape layer_shape(const ConvGeom &g) {
  return mm::LayerShape{g.N, (int)g.C, (int)g.H, (int)g.W, (int)g.K, (int)g.oH, (int)g.oW, g.kH, g.kW, g.dH, g.dW, g.pad};
}
// What the strays of a forward product's (GRAD_INPUT: a gradInput product's) operands add to its result.
template <bool GRAD_INPUT>
static void add_strays(const ConvGeom &g, const float *src, const float *w, float *out, const Records &rec) {
  const long planes = GRAD_INPUT ? g.C : g.K;
  const dim3 grid((unsigned)std::min(g.N, 37l), (unsigned)std::min(planes, 8l));
  pdl_launch(mm::window_strays_kernel<GRAD_INPUT>, grid, 256, 0, src, w, out, layer_shape(g), GRAD_INPUT ? rec.gout : rec.act, rec.weight,
             rec.joint(rec.weight));
  check_launch("window_strays");
}

// Weights beyond which a pass over them is worth a launch of its own: next to another pass an SM holds half its blocks, by the other's registers or tile.
constexpr long kManyWeights = 3l << 20;
// Repacked weights of a product of windows, rows r < rows: the buffer, and the pass that fills it, which shares a launch with the one that makes
// the windows' planes or has one of its own ahead of the product.  (us, together / apart, turned filters: 103 M weights in BF16 593 / 431 + 4, 9.4 M 50 / 45 + 4; 4.1 M of
// 1 x 1 forward 65 / 62 with their product; 2.4 M 15 / 13 + 7.)
template <int PREC, bool FLIP>
struct FilterForm {
  mm::Windows full, v;   // the layer's windows, and those of the product (pixel pairs)
  bool pair = false;
  long rows = 0, wrows = 0, Kd = 0;
  unsigned alone = 0;    // the pass's blocks where it has a launch of its own
  mm::RepackPass<PREC, FLIP> pass;
};
template <int PREC, bool FLIP>
static FilterForm<PREC, FLIP> filter_form(const mm::Windows &full, const float *w, const mm::Cells &u, long K, long rows, const Records &rec) {
  FilterForm<PREC, FLIP> f;
  f.full = f.v = full;
  mm::Windows p;
  if (pair_windows(full, rows, PREC, p)) { f.pair = true; f.v = p; }
  f.rows = rows; f.wrows = (f.pair ? 2 : 1) * rows; f.Kd = (long)f.v.kH * f.v.kW * f.v.C;
  THC_CHECK(f.wrows * f.Kd < (1l << 31), "filter too large");
  void *wp = ws_alloc((size_t)f.wrows * f.Kd * (PREC == mm::kBf16 ? 2 : 4));
  const long blocks = std::min<long>((f.wrows * (f.Kd / 4) + 255) / 256, ctx().sm_count * 8l);
  f.pass = mm::RepackPass<PREC, FLIP>{(unsigned)blocks, w, u, (int)K, (int)rows, (int)f.v.C, f.pair ? full.dW : 0, wp, rec.joint(rec.weight)};
  if (f.wrows * f.Kd > kManyWeights) std::swap(f.alone, f.pass.blocks);
  return f;
}
// out[n, r, y, x] = bias[r] + the product of the windows over `act` with the repacked weights
template <int PREC, bool PAIR, bool FLIP>
static void window_product_t(const void *act, const FilterForm<PREC, FLIP> &f, const float *bias, float *out, const Records &rec) {
  using namespace mm;
  const Windows &full = f.full, &v = f.v;
  const long rows = f.rows;
  if (f.alone) {
    const auto &w = f.pass;
    pdl_launch(repack_weight_kernel<PREC, FLIP>, f.alone, 256, 0, w.w, w.u, w.K, w.rows, w.chans, w.pair_shift, w.out, w.ranges);
    check_launch("repack_weight");
  }
  Problem<PlanesWindowOperand<PREC>, RawOperand<false, PREC>, PAIR, PREC> p;
  p.range_a = rec.act.rec; p.range_b = rec.weight.rec; p.ranges = rec.joint(rec.act);
  attach_window_map<PREC>(p.a, act, v);
  const long P = full.oH * full.oW;
  p.epi = Epilogue{out, bias, 1.f, 0.f, P, rows * P, P};
  if (PAIR) {
    p.epi.pair_K = rows; p.epi.pair_oH = full.oH; p.epi.pair_oW2 = v.oW; p.epi.pair_oW = full.oW; p.epi.pair_img = rows * P;
  }
  p.M = v.N * v.oH * v.oW; p.N = f.wrows; p.K = f.Kd;
  launch_raw(p, [&](auto &q, int bn2) { attach_raw_map<PREC>(q.b, f.pass.out, f.wrows, f.Kd, f.Kd, bn2 / 2); });
}
template <int PREC, bool FLIP>
static void window_product(const void *act, const FilterForm<PREC, FLIP> &f, const float *bias, float *out, const Records &rec) {
  if constexpr (PREC != mm::kBf16)
    if (f.pair) { window_product_t<PREC, true>(act, f, bias, out, rec); return; }
  window_product_t<PREC, false>(act, f, bias, out, rec);
}

// The restated input in `dst`, and the weights of `repack`.
template <int PREC>
static void restate_input(const ConvGeom &g, const mm::Cells &u, const float *in, void *dst, const mm::PairForm &form,
                          const mm::RepackPass<PREC, false> &repack) {
  if (u.direct) { mm::make_act_planes<PREC, false>(in, g.N, g.C, g.H, g.W, dst, form, repack, mm::NoPass{}); return; }
  if constexpr (PREC == mm::kBf16) {
    const size_t smem = sizeof(uint4) * g.kH * (g.W + 2 * g.pad);
    if (u.Cq == 8 && u.kHs == 1 && u.kWs == 1 && g.C <= 8 && smem <= 200 * 1024) {
      static thread_local int configured_for = -1;
      if (configured_for != ctx().device) {
        THC_CUDA(cudaFuncSetAttribute(mm::passes_kernel<mm::Columns8Pass, mm::RepackPass<PREC, false>, mm::NoPass>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        configured_for = ctx().device;
      }
      mm::launch_passes(mm::Columns8Pass{(unsigned)(g.N * u.Hs), in, (uint4 *)dst, u}, smem, "columns8", repack);
      return;
    }
  }
  // a block per row of cells; a row is shared by several blocks where the rows of few images leave SMs idle (one
  // 224 x 224 image: 8.4 us with one block each)
  const long rows = g.N * u.Hs, chunks = (long)u.Ws * u.Cs / (PREC != mm::kTf32 ? 8 : 4);
  const unsigned parts = (unsigned)std::max(1l, std::min((chunks + 255) / 256, 4l * ctx().sm_count / rows));
  if constexpr (PREC != mm::kBf16) {
    const int q = u.Cs / (PREC == mm::kPairs ? 8 : 4);
    const long Wp = (long)(u.Ws - 1) * u.dW + u.eW, ld = (Wp + 15) / 32 * 32 + 16, smem = 4l * u.C * u.eH * ld;
    // Rows long enough to hide a block's barriers, of few input lines.  By units of 16 bytes a row, forward pass of the layer staged and
    // not (us): 3 x 3 over 224 wide (1792 units) 451 / 510, 13 images 101 / 112, 7 x 7 / 2 (1840) 241 / 271, 500 wide
    // (8000) 8239 / 8954, 128 wide 4 planes (1040) 224 / 228; 912 units 384 / 409 over 14592 rows, 132.5 / 132.6 over 3648, 48.4 / 47.7 over
    // 912; 832 units 168.6 / 170.4 over 6400 rows, 768 183 / 194 over 12288; below, it loses: 608 112.3 / 109.5, 536 76.6 / 73.0, 464
    // 44.1 / 38.2, 256 59.6 / 51.7 and 206 / 187.  45 lines of 85 columns (1360): 211.5 / 205.3, 21 lines gain.
    const long units = chunks * (PREC == mm::kPairs ? 2 : 1);
    if (256 % q == 0 && smem <= 40 * 1024 && rows >= 2l * ctx().sm_count && u.C * u.eH <= 24 &&
        (units >= 1024 || (units >= 768 && rows >= 32l * ctx().sm_count))) {
      mm::launch_passes(mm::StagedCellsPass<PREC>{(unsigned)std::min(rows, 16l * ctx().sm_count), in, dst, g.N, u, (int)Wp, (int)ld, form}, smem, "cells_staged", repack);
      return;
    }
  }
  const unsigned blocks = (unsigned)rows * parts;
  if (u.Cs <= mm::kCellTable) mm::launch_passes(mm::CellsPass<PREC, true>{blocks, (unsigned)rows, in, dst, u, form}, sizeof(int2) * u.Cs, "cells_input", repack);
  else mm::launch_passes(mm::CellsPass<PREC, false>{blocks, (unsigned)rows, in, dst, u, form}, 0, "cells_input", repack);
}

// Room for the restated input in `finput` (the counterpart of the column matrix the reference keeps there): a
// [1, N, Hs, Ws, floats per pixel] tensor that accGradParameters reads back instead of making it again.  Null: no room that a
// TMA map can address.
static void *planes_in(THGPUTensor *finput, const ConvGeom &g, const mm::Cells &u, const float *in, int prec) {
  const long s[5] = {1, g.N, u.Hs, u.Ws, prec == mm::kBf16 ? u.Cs / 2 : u.Cs};
  resize_nd(finput, 5, s, nullptr);
  forget_planes(finput);
  if (!is_contiguous(finput) || ((uintptr_t)data_ptr(finput) & 15) != 0) return nullptr;
  stamp_planes(finput, in, g, prec);
  return data_ptr(finput);
}

// The planes the forward pass of this very layer over this very input left in `finput`, or null.  A `finput` that has been given
// another shape since has been used for something else.
static const void *planes_made_from(const THGPUTensor *finput, const float *input, const ConvGeom &g, const mm::Cells &u, int prec) {
  if (!finput || !finput->storage || finput->nDimension != 5 || !is_contiguous(finput)) return nullptr;
  const long shape[5] = {1, g.N, u.Hs, u.Ws, prec == mm::kBf16 ? u.Cs / 2 : u.Cs};
  if (!std::equal(shape, shape + 5, finput->size)) return nullptr;
  auto it = g_plane_stamps.find(data_ptr(finput));
  if (it == g_plane_stamps.end()) return nullptr;
  const PlaneStamp &s = it->second;
  const bool same = s.input == input && s.prec == prec && s.N == g.N && s.C == g.C && s.H == g.H && s.W == g.W && s.K == g.K &&
                    s.kH == g.kH && s.kW == g.kW && s.dH == g.dH && s.dW == g.dW && s.pad == g.pad && s.epoch == ctx().plane_epoch;
  return same ? data_ptr(finput) : nullptr;
}

// BF16: the forward product of a layer of up to eight planes over windows that the engine gathers from an image of eight-plane pixels, in the
// k order, the tiles and the k slices of the product over the column matrix, whose bits it gives.  Where nobody keeps that matrix (a weight
// gradient of the same precision reads it) and its tiles are 64 wide, the widest that K <= 64 comes to.  False: another form.
static bool gathered_forward(const ConvGeom &g, const mm::Cells &u, const float *in, const float *w, const float *bias, float *out) {
  using namespace mm;
  const long rows = (g.oH - 1) * g.dH + g.kH, pitch = (g.oW - 1) * g.dW + g.kW;
  if (u.direct || u.Cq != 8 || u.kHs != 1 || u.kWs != 1 || g.C > 8 || g.K > 64 || rows * pitch >= 1l << 27 || 16. * (double)(g.N * rows * pitch) > kGroupScratch ||
      (double)planes_bytes(g.N, g.P, u.Cs, kBf16) > kGroupScratch || !encode_tiled_fn())
    return false;
  const auto filter = filter_form<kBf16, false>(forward_windows(g, u), w, u, g.K, g.K, Records{});
  uint4 *image = (uint4 *)ws_alloc(sizeof(uint4) * g.N * rows * pitch);
  const long pieces = g.N * rows * ((pitch + 127) / 128);
  launch_passes(Pixels8Pass{(unsigned)std::min((pieces + 7) / 8, 16l * ctx().sm_count), in, image, g.N, (int)g.C, (int)g.H, (int)g.W, g.pad, (int)rows, (int)pitch}, 0,
                "pixels8", filter.pass);
  Problem<GatheredWindowOperand, RawOperand<false, kBf16>, false, kBf16> p;
  p.a.image = image; p.a.image_pixels = (int)(rows * pitch); p.a.pitch = (int)pitch; p.a.taps = g.kH * g.kW; p.a.kW = g.kW;
  p.a.rows.set(g.N * g.P, g.P, g.oW);
  p.a.rows.sy = g.dH; p.a.rows.sx = g.dW;
  p.epi = Epilogue{out, bias, 1.f, 0.f, g.P, g.K * g.P, g.P};
  p.M = g.N * g.P; p.N = g.K; p.K = filter.Kd;
  launch_raw(p, [&](auto &q, int bn2) { attach_raw_map<kBf16>(q.b, filter.pass.out, filter.wrows, filter.Kd, filter.Kd, bn2 / 2); });
  return true;
}

template <int PREC>
static void conv_forward_tc(const ConvGeom &g, const mm::Cells &u, const float *in, const float *w, const float *bias, float *out,
                            THGPUTensor *finput) {
  const double bytes = (double)mm::planes_bytes(1, (long)u.Hs * u.Ws, u.Cs, PREC), floats = (double)g.N * g.C * g.H * g.W;
  if (finput && bytes * (double)g.N > whole_scratch(floats)) finput = nullptr;
  const long per = finput ? g.N : images_per_group(g.N, bytes, kGroupScratch);
  for (long n0 = 0; n0 < g.N; n0 += per) {
    WsScope ws_scope;
    ConvGeom s = g;
    s.N = std::min(per, g.N - n0);
    const float *x = in + n0 * g.C * g.H * g.W;
    if (PREC == mm::kBf16 && !finput && gathered_forward(s, u, x, w, bias, out + n0 * g.K * g.P)) continue;
    Records rec;
    if constexpr (PREC == mm::kPairs) {   // (for each group: records last for some thousand words, see zeroed_words)
      rec.act = mm::new_measured(); rec.weight = mm::new_measured();
      mm::RangeJob jw = mm::range_job_flat(w, g.K * g.R, rec.weight);
      mm::launch_ranges(mm::range_job_flat(x, s.N * g.C * g.H * g.W, rec.act), &jw);
    }
    mm::PairForm form;
    form.ranges = rec.joint(rec.act);
    const auto filter = filter_form<PREC, false>(forward_windows(s, u), w, u, g.K, g.K, rec);
    void *act = finput ? planes_in(finput, s, u, x, PREC) : nullptr;
    UnmadePlanes unmade{act ? finput : nullptr};
    if (act && PREC == mm::kPairs) { form.keep = planes_record(act); form.list = rec.act.list; }
    if (!act) act = ws_alloc(mm::planes_bytes(s.N, (long)u.Hs * u.Ws, u.Cs, PREC));
    restate_input<PREC>(s, u, x, act, form, filter.pass);
    unmade.finput = nullptr;
    window_product(act, filter, bias, out + n0 * g.K * g.P, rec);
    if (PREC == mm::kPairs) add_strays<false>(s, x, w, out + n0 * g.K * g.P, rec);
  }
}

// Wt[c][(ko, i, j)] = W[ko][(c, i, j)]: the weight matrix as the gathered gradInput product reads it; `turned`: with the filter rotated
// by 180 degrees, the weights of gradInput as a layer over gradOutput.
static __global__ void __launch_bounds__(256) transpose_weight_kernel(const float *__restrict__ w, float *__restrict__ wt,
                                                                      long K, long C, long kHW, bool turned) {
  pdl_begin();
  const long total = K * C * kHW;
  const long nthreads = (long)gridDim.x * blockDim.x;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += nthreads) {
    const long tap = t % kHW, q = t / kHW, ko = q % K, c = q / K;
    wt[t] = w[(ko * C + c) * kHW + (turned ? kHW - 1 - tap : tap)];
  }
}
static const float *transposed_weight(const ConvGeom &g, const float *w, bool turned) {
  const long kHW = (long)g.kH * g.kW, total = g.C * g.K * kHW;
  float *wt = (float *)ws_alloc(sizeof(float) * total);
  pdl_launch(transpose_weight_kernel, (unsigned)std::min<long>((total + 255) / 256, ctx().sm_count * 8l), 256, 0, w, wt, g.K, g.C, kHW, turned);
  check_launch("transpose_weight");
  return wt;
}

// gradInput of a layer with few output planes stated as a layer of its own, whose input is gradOutput: padding two planes to a span of
// channels multiplies the product by 16, which restate() knows to avoid (13 x 13 taps, 271 <- 2 planes of 110 x 118, four images in
// BF16: 915 us over padded planes, 177 so; 9 x 9, 32 <- 2, 46 of 87 x 88: 516 and 121).  False: the padded planes cost less.
static bool grad_input_layer(const ConvGeom &g, int prec, ConvGeom &t, mm::Cells &u) {
  if (g.dH != 1 || g.dW != 1 || g.kH != g.kW || g.pad >= g.kH || 2 * g.K > mm::padded_channels(g.K, prec)) return false;
  t = g;
  t.C = g.K; t.K = g.C; t.H = g.oH; t.W = g.oW; t.oH = g.H; t.oW = g.W; t.P = g.H * g.W;
  t.pad = g.kH - 1 - g.pad; t.R = g.K * g.kH * g.kW;
  if (!restate(t, prec, u) || u.direct) return false;
  const double bytes = (double)mm::planes_bytes(g.N, (long)u.Hs * u.Ws, u.Cs, prec);
  const double own = windows_us(forward_windows(t, u), t.K, prec) + 2 * bytes / 5e6 + 10;   // and two launches more
  return own < windows_us(grad_input_windows(g, grad_input_cells(g, prec), prec), g.C, prec);
}

// gradInput = forward pass of gradOutput's planes under the filter rotated by 180 degrees with its plane roles swapped.
static Records grad_input_records(const Records &records) {
  Records rec = records;
  std::swap(rec.act, rec.gout);   // the windows run over gradOutput here
  return rec;
}
template <int PREC>
static FilterForm<PREC, true> grad_input_filter(const ConvGeom &g, const float *w, const Records &records) {
  const mm::Cells u = grad_input_cells(g, PREC);
  return filter_form<PREC, true>(grad_input_windows(g, u, PREC), w, u, g.K, u.direct ? g.C : u.Cr, grad_input_records(records));
}
template <int PREC>
static void conv_grad_input_tc(const ConvGeom &g, const mm::ActPlanes &pgo, const FilterForm<PREC, true> &filter, float *gin, const Records &records) {
  const Records rec = grad_input_records(records);
  const mm::Cells &u = filter.pass.u;
  if (u.direct) { window_product(pgo.p, filter, nullptr, gin, rec); return; }
  float *gS = (float *)ws_alloc(sizeof(float) * g.N * u.Cr * (long)(u.Hs * u.Ws));
  window_product(pgo.p, filter, nullptr, gS, rec);
  const long planes = g.N * g.C, HW = g.H * g.W, group = std::max(1l, 1024 / HW);
  const unsigned by = (unsigned)std::min((planes + group - 1) / group, ctx().sm_count * 32l);
  const unsigned bx = (unsigned)std::min((group * HW + 1023) / 1024, std::max(1l, ctx().sm_count * 32l / by));
  pdl_launch(mm::unfold_grad_input_kernel, dim3(bx, by), 256, 0, gS, gin, u,
             mm::UnfoldGeom{planes, (int)group, mm::FastDiv::make(HW), mm::FastDiv::make(g.C), mm::FastDiv::make(g.W), mm::FastDiv::make(u.dH), mm::FastDiv::make(u.dW)});
  check_launch("unfold_grad_input");
}

// gw += scale * T, and the fold of gradBias.  (us, together / apart: 9.4 M weights 49 / 33 + 4 from FP16 pairs or BF16, 2.4 M 23 / 23 + 6.)
template <bool PAIRS>
static void unpack_grad_weight(const ConvGeom &g, const mm::Cells &u, const float *T, float *gw, const mm::WgradPlace &pl, float scale, const mm::WgradStrays &strays,
                               const mm::ChanFinishPass &bias) {
  using namespace mm;
  const long blocks = std::min((g.K * g.R + 255) / 256, ctx().sm_count * 32l);
  auto pass = [&](auto alone) { return UnpackGradPass<PAIRS, decltype(alone)::value>{(unsigned)blocks, T, gw, u, (int)g.K, WgradDivs::of(u), pl, scale, strays}; };
  if (g.K * g.R <= kManyWeights) {
    launch_passes(pass(std::false_type()), 0, "unpack_grad_weight", bias);
  } else {
    launch_passes(bias, 0, "conv_grad_bias_finish");
    launch_passes(pass(std::true_type()), 0, "unpack_grad_weight");
  }
}

// gradW[ko][(c,i,j)] += scale * sum over windows of gradOut[ko] * S[tap, ch]: the reduction runs over pixels, along which
// neither tensor is contiguous in channels-last form, so both enter as MN-major operands.  Three ways round, by cost:
//   0  rows = output planes, columns = (tap, ch)
//   1  rows = (tap, ch), columns = output planes
//   2  rows = (bi, ch), columns = (bj, output plane): with the reduction running over the full restated width,
//        T[(bi, ch)][(j', ko)] = sum_{n, y, x'} S[n][y + bi][x'][ch] * gradOut[n][y][x' - (kWs - 1 - j')][ko]
//      is the gradient of tap (bi, bj = kWs - 1 - j'): the column shift is a zero-padded window of the gradOutput
//      plane, which TMA's im2col mode reads like any other.  For layers with few output planes and columns, whose
//      64-wide tiles would run at half the tensor-pipe rate.
// and, for the column form (one tap), whose two operands are plain matrices of a few columns:
//   3  f pixels side by side, rows = (pixel mod f, ko), columns = (pixel mod f, ch) of the same memory read as wider
//      matrices: the f diagonal blocks of the result are the gradient's partial sums.  The other blocks are computed in
//      vain, but a k tile costs the same however little of its 256 x 64 tile is used, and there are f times fewer.
template <int PREC>
static void conv_acc_grad_tc(const ConvGeom &g, const mm::Cells &u, const void *act, const mm::ActPlanes &pgo, const float *gout, long n0, float *gw,
                             float scale, const Records &rec, const mm::ChanFinishPass &bias) {
  using namespace mm;
  const WgradStrays strays{rec.act, rec.gout, rec.joint(rec.act), n0, act, gout, layer_shape(g)};
  const Windows v = forward_windows(g, u);
  const long Kp = pgo.Cp, Cs = u.Cs, Rp = (long)u.kHs * u.kWs * Cs, pixels = g.N * g.P;
  const long M2 = (long)u.kHs * Cs, N2 = (long)u.kWs * Kp;
  const Windows va{g.N, u.Hs, u.Ws, Cs, g.oH, u.Ws, u.kHs, 1, 1, 1, 0, 0};
  const Windows vb{g.N, g.oH, g.oW, Kp, g.oH, u.Ws, 1, u.kWs, 1, 1, 0, u.kWs - 1};
  double us[3] = {tc2_product_us(g.K, Rp, pixels, PREC, true), tc2_product_us(Rp, g.K, pixels, PREC, true),
                  !u.direct && u.kWs > 1 && windows_ok(va) && windows_ok(vb) ? tc2_product_us(M2, N2, g.N * g.oH * u.Ws, PREC, true) : 1e30};
  int way = us[2] < us[0] && us[2] < us[1] ? 2 : us[1] < us[0] ? 1 : 0;
  long f = 1;
  if (PREC != kPairs && u.kHs == 1 && u.kWs == 1 && !u.direct)   // (a pair's halves lie side by side, not a pixel's neighbours)
    while (2 * f * Kp <= 256 && 2 * f * Cs <= 256 && pixels % (2 * f) == 0) f *= 2;
  if (f > 1 && tc2_product_us(f * Kp, f * Cs, pixels / f, PREC, true) < us[way]) {
    const long Mf = f * Kp, Nf = f * Cs;
    float *T = (float *)ws_alloc(sizeof(float) * Mf * Nf);
    Problem<RawOperand<true, PREC>, RawOperand<true, PREC>, false, PREC> p;
    p.range_a = rec.gout.rec; p.range_b = rec.act.rec; p.ranges = rec.joint(rec.act);
    p.epi = Epilogue{T, nullptr, 1.f, 0.f, 1, Nf, 1};                 // T[m * Nf + n]
    p.M = Mf; p.N = Nf; p.K = pixels / f;
    launch_raw(p, [&](auto &q, int bn2) {
      attach_raw_map<PREC>(q.a, pgo.p, Mf, pixels / f, Mf, TC_BM);
      attach_raw_map<PREC>(q.b, act, Nf, pixels / f, Nf, bn2 / 2);
    });
    const WgradPlace pl{Nf, 1, 0, 0, 0, (int)f, Kp * Nf + Cs};
    unpack_grad_weight<PREC == kPairs>(g, u, T, gw, pl, scale, strays, bias);
    return;
  }
  const long cols = way == 2 ? N2 : way == 1 ? g.K : Rp, rows = way == 2 ? M2 : way == 1 ? Rp : g.K;
  float *T = (float *)ws_alloc(sizeof(float) * rows * cols);
  WgradPlace pl;
  if (way == 0) {
    Problem<RawOperand<true, PREC>, WindowRowsOperand<PREC>, false, PREC> p;
    p.range_a = rec.gout.rec; p.range_b = rec.act.rec; p.ranges = rec.joint(rec.act);
    attach_window_rows_map<PREC>(p.b, act, v);
    p.epi = Epilogue{T, nullptr, 1.f, 0.f, 1, Rp, 1};                 // T[m * Rp + n]
    p.M = g.K; p.N = Rp; p.K = pixels;
    launch_raw(p, [&](auto &q, int) { attach_raw_map<PREC>(q.a, pgo.p, Kp, pixels, Kp, TC_BM); });
    pl = WgradPlace{Rp, 1, u.kWs * Cs, Cs, 0, 1, 0};
  } else if (way == 1) {
    Problem<WindowRowsOperand<PREC>, RawOperand<true, PREC>, false, PREC> p;
    p.range_a = rec.act.rec; p.range_b = rec.gout.rec; p.ranges = rec.joint(rec.act);
    attach_window_rows_map<PREC>(p.a, act, v);
    p.epi = Epilogue{T, nullptr, 1.f, 0.f, LONG_MAX, 0, Rp};          // T[n * Rp + m]
    p.M = Rp; p.N = g.K; p.K = pixels;
    launch_raw(p, [&](auto &q, int bn2) { attach_raw_map<PREC>(q.b, pgo.p, Kp, pixels, Kp, bn2 / 2); });
    pl = WgradPlace{Rp, 1, u.kWs * Cs, Cs, 0, 1, 0};
  } else {
    Problem<WindowRowsOperand<PREC>, WindowRowsOperand<PREC>, false, PREC> p;
    p.range_a = rec.act.rec; p.range_b = rec.gout.rec; p.ranges = rec.joint(rec.act);
    attach_window_rows_map<PREC>(p.a, act, va);
    attach_window_rows_map<PREC>(p.b, pgo.p, vb);
    p.epi = Epilogue{T, nullptr, 1.f, 0.f, 1, N2, 1};                 // T[m * N2 + n]
    p.M = M2; p.N = N2; p.K = g.N * g.oH * u.Ws;
    launch_raw(p, [](auto &, int) {});
    pl = WgradPlace{1, N2, Cs * N2, -Kp, (u.kWs - 1) * Kp, 1, 0};
  }
  unpack_grad_weight<PREC == kPairs>(g, u, T, gw, pl, scale, strays, bias);
}

// ------------------------------------------------------------------------------------------------
// Element gathers straight from NCHW on the FP32 FMA engine: the "simt" math mode, and windows beyond what TMA can express.

static mm::PixelMap input_windows(const ConvGeom &g) {  // (img, y, x) -> top-left corner of its window
  mm::PixelMap m;
  m.set(g.N * g.P, g.P, g.oW);
  m.img_stride = g.C * g.H * g.W; m.y_stride = g.dH * g.W; m.x_stride = g.dW;
  m.off0 = -(long)g.pad * g.W - g.pad;
  m.sy = g.dH; m.y0 = -g.pad; m.sx = g.dW; m.x0 = -g.pad;
  return m;
}
static mm::TapMap input_taps(const ConvGeom &g) {  // (c, i, j) -> offset inside the window
  mm::TapMap m;
  m.set(g.R, g.kH * g.kW, g.kW);
  m.c_stride = g.H * g.W; m.i_stride = g.W; m.j_stride = 1;
  m.si = 1; m.sj = 1;
  return m;
}

static void conv_forward_simt(const ConvGeom &g, const float *in, const float *w, const float *bias, float *out) {
  using namespace mm;
  Problem<Operand<PixelMap, TapMap, 1>, Operand<LinearMap, LinearMap, 0>> p;   // im2col rows; weight [K, R]
  p.a.base = in; p.a.rows = input_windows(g); p.a.ks = input_taps(g);
  p.a.H = (int)g.H; p.a.W = (int)g.W; p.a.dH = p.a.dW = 1;
  p.b.base = w; p.b.rows = LinearMap{g.K, g.R}; p.b.ks = LinearMap{g.R, 1};
  p.b.H = p.b.W = 0; p.b.dH = p.b.dW = 1;
  p.epi = Epilogue{out, bias, 1.f, 0.f, g.P, g.K * g.P, g.P};
  p.M = g.N * g.P; p.N = g.K; p.K = g.R;
  launch_simt(p);
}

static void conv_grad_input_simt(const ConvGeom &g, const float *gout, const float *w, float *gin) {
  using namespace mm;
  const long kHW = (long)g.kH * g.kW, Kd = g.K * kHW;
  const float *wt = transposed_weight(g, w, false);
  // rows = input pixels, k = (ko, i, j); only taps with (h + pad - i) % dH == 0 contribute
  Problem<Operand<PixelMap, TapMap, 2>, Operand<LinearMap, LinearMap, 0>> p;
  PixelMap rows;
  rows.set(g.N * g.H * g.W, g.H * g.W, g.W);
  rows.img_stride = g.K * g.P; rows.y_stride = 0; rows.x_stride = 0; rows.off0 = 0;
  rows.sy = 1; rows.y0 = g.pad; rows.sx = 1; rows.x0 = g.pad;
  TapMap ks;
  ks.set(Kd, kHW, g.kW);
  ks.c_stride = g.P; ks.i_stride = 0; ks.j_stride = 0; ks.si = -1; ks.sj = -1;
  p.a.base = gout; p.a.rows = rows; p.a.ks = ks; p.a.H = (int)g.oH; p.a.W = (int)g.oW; p.a.dH = g.dH; p.a.dW = g.dW;
  p.b.base = wt; p.b.rows = LinearMap{g.C, Kd}; p.b.ks = LinearMap{Kd, 1};
  p.b.H = p.b.W = 0; p.b.dH = p.b.dW = 1;
  p.epi = Epilogue{gin, nullptr, 1.f, 0.f, g.H * g.W, g.C * g.H * g.W, g.H * g.W};
  p.M = rows.count; p.N = g.C; p.K = Kd;
  launch_simt(p);
}

static void conv_acc_grad_simt(const ConvGeom &g, const float *in, const float *gout, float *gw, float scale) {
  using namespace mm;
  Problem<Operand<TapMap, PixelMap, 1>, Operand<LinearMap, PixelMap, 0>> p;   // input under tap r of window (img, y, x); gradOut[img, ko, p]
  p.a.base = in; p.a.rows = input_taps(g); p.a.ks = input_windows(g);
  p.a.H = (int)g.H; p.a.W = (int)g.W; p.a.dH = p.a.dW = 1;
  p.b.base = gout; p.b.rows = LinearMap{g.K, g.P};
  p.b.ks.set(g.N * g.P, g.P, g.P);
  p.b.ks.img_stride = g.K * g.P; p.b.ks.y_stride = 0; p.b.ks.x_stride = 1; p.b.ks.off0 = 0;
  p.b.ks.sy = 0; p.b.ks.y0 = 0; p.b.ks.sx = 0; p.b.ks.x0 = 0;
  p.b.H = p.b.W = 0; p.b.dH = p.b.dW = 1;
  p.epi = Epilogue{gw, nullptr, scale, 1.f, LONG_MAX, 0, g.R};
  p.M = g.R; p.N = g.K; p.K = g.N * g.P;
  launch_simt(p);
}

// gradBias[k] += scale * sum_{img, p} gradOut[img, k, p].  Pass 1: block (k, s) sums the images
// s, s+S, ... of plane k into partial[k][s]; pass 2 folds the S partials in order (deterministic).
static __global__ void __launch_bounds__(256) conv_grad_bias_partial_kernel(const float *__restrict__ gout,
                                                                            float *__restrict__ partial, long N, long K,
                                                                            long P) {
  pdl_begin();
  __shared__ float sm[8];
  const long k = blockIdx.x;
  // One image per warp at a time (eight images in flight per block), four independent partial sums per lane:
  // with one dependent load chain per thread, or one image per block, small planes (13 x 13) left the kernel
  // waiting on memory latency.
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
  for (long img = blockIdx.y + (long)warp * gridDim.y; img < N; img += 8l * gridDim.y) {
    const float *g = gout + (img * K + k) * P;
    long p = lane;
    for (; p + 96 < P; p += 128) { a0 += g[p]; a1 += g[p + 32]; a2 += g[p + 64]; a3 += g[p + 96]; }
    for (; p < P; p += 32) a0 += g[p];
  }
  float acc = (a0 + a1) + (a2 + a3);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    acc = threadIdx.x < 8 ? sm[threadIdx.x] : 0.f;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (threadIdx.x == 0) partial[k * gridDim.y + blockIdx.y] = acc;
  }
}
static __global__ void conv_grad_bias_finish_kernel(const float *__restrict__ partial, float *gbias, long K, int S,
                                                    float scale) {
  pdl_begin();
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  float acc = 0.f;
  for (int s = 0; s < S; s++) acc += partial[k * S + s];
  gbias[k] += scale * acc;
}

static void grad_bias(const ConvGeom &g, const float *gout, float *gb, float scale) {
  long S = (long)ctx().sm_count * 8 / g.K;
  if (S > g.N) S = g.N;
  if (S < 1) S = 1;
  float *partial = (float *)ws_alloc(sizeof(float) * g.K * S);
  pdl_launch(conv_grad_bias_partial_kernel, dim3((unsigned)g.K, (unsigned)S), 256, 0, gout, partial, g.N, g.K, g.P);
  check_launch("conv_grad_bias_partial");
  pdl_launch(conv_grad_bias_finish_kernel, ceil_div(g.K, 128), 128, 0, partial, gb, g.K, (int)S, scale);
  check_launch("conv_grad_bias_finish");
}

// Which products the BF16 math mode runs in BF16: those whose output has more than a tile's worth of rows and enough columns to
// be bound by arithmetic.  The others, the weight gradient of a first layer among them, stay FP32-accurate: their sums over
// all pixels are what the rest of the step's precision rests on, and they gain least.
static bool half_forward(const ConvGeom &g) { return ctx().math_mode == 2 && g.N * g.P > 128 && g.K > 32; }
static bool half_grad_input(const ConvGeom &g) {
  return ctx().math_mode == 2 && g.dH == 1 && g.dW == 1 && g.pad < g.kH && g.pad < g.kW && g.N * g.H * g.W > 128 && g.C > 32;
}
static bool half_acc_grad(const ConvGeom &g) {
  const long Kp = (g.K + 7) / 8 * 8, Rp = (long)g.kH * g.kW * ((g.C + 7) / 8 * 8);
  return ctx().math_mode == 2 && ((Kp > 128 && Rp > 64) || (Rp > 128 && Kp > 64));
}

// FP16 pairs or TF32 for the FP32-accurate products of a layer, all of which share its planes: by the forward product's time and
// the pass that measures the input, with 10 us for the launches that measure and check.  Forward and backward near the line (us, pairs /
// TF32): 64 planes under 11 x 11 / 4 over 32 images 259 / 255, over 64 398 / 508; 64 -> 128 of 112 x 112, 4 images, 210 / 211; 64 -> 192 under 5 x 5, 27 x
// 27, 16 images, 175 / 247; 512 -> 512 of 14 x 14, 13 images, 223 / 244; 64 -> 64 of 56 x 56, 32 images, 259 / 267.  Where an operand has to stay
// in FP32 a layer takes longer than in TF32, by the measuring passes, spans of 64 channels and tiles of 128 or 256: 1024 images
// 64 -> 192 8.13 ms / 7.16, 384 -> 256 4.45 / 4.31; 13 images 256 -> 256 of 56 x 56 778 us / 705, 512 -> 512 of 14 x 14 290 / 244; 96 -> 96 (128 for 96
// channels), 64 images, 1250 / 1000.  The column form stays in TF32, whose weight gradient stacks pixels.
static bool restate_accurate(const ConvGeom &g, bool pairs, mm::Cells &u, int &prec) {
  prec = mm::kTf32;
  const bool ok = restate(g, mm::kTf32, u);
  mm::Cells up;
  if (!ok || !pairs || g.R > 1l << 28 || g.K * g.kH * g.kW > 1l << 28 ||   // (a row of weights and its second half: 31 bits)
      windows_us(forward_windows(g, u), g.K, prec) < 30 || !restate(g, mm::kPairs, up) || up.Cs > mm::UnpairPass<6>::kMost ||
      (up.kHs == 1 && up.kWs == 1 && !up.direct))
    return ok;
  // (filter_form counts the repacked weights in 31 bits; channels in spans of 64 may make more of them than spans of 32)
  const mm::Cells gi = grad_input_cells(g, mm::kPairs);
  if (2. * g.K * up.kHs * up.kWs * up.Cs >= 0x1p31 || 2. * (gi.direct ? gi.C : gi.Cr) * gi.kHs * gi.kWs * mm::padded_channels(g.K, mm::kPairs) >= 0x1p31) return ok;
  auto us = [&](const mm::Cells &c, int pr) {
    return windows_us(forward_windows(g, c), g.K, pr) + 2 * (double)mm::planes_bytes(g.N, (long)c.Hs * c.Ws, c.Cs, pr) / 5e6;
  };
  if (us(up, mm::kPairs) + 10 + 4e-6 / 5.5 * (double)(g.N * g.C * g.H * g.W) < us(u, mm::kTf32)) { u = up; prec = mm::kPairs; }
  return ok;
}

static void conv_forward(const ConvGeom &g, const float *in, const float *w, const float *bias, float *out, THGPUTensor *finput) {
  mm::Cells u;
  const bool half = half_forward(g);
  int prec = mm::kBf16;
  if (ctx().math_mode != 1 && (half ? restate(g, prec, u) : restate_accurate(g, ctx().math_mode == 0, u, prec))) {
    // kept for a weight gradient of the same precision only, no other reads them back: the BF16 column matrix of the 11 x 11 / 4
    // layer over 3 planes is 6.2 MB an image, and its weight gradient FP32-accurate
    THGPUTensor *keep = half == half_acc_grad(g) ? finput : nullptr;
    if (keep && ctx().math_mode == 2 && !half) {   // an FP32-accurate layer of that mode: its weight gradient may run over pairs (conv_backward)
      mm::Cells uw;
      int pw;
      restate_accurate(g, true, uw, pw);
      if (pw != prec) keep = nullptr;
    }
    if (prec == mm::kPairs) {
      try {
        conv_forward_tc<mm::kPairs>(g, u, in, w, bias, out, keep);
        return;
      } catch (const OutOfMemory &) {   // FP32 planes may take half of it (channels in spans of 32, not 64)
        restate(g, mm::kTf32, u);
      }
    }
    if (prec == mm::kBf16) conv_forward_tc<mm::kBf16>(g, u, in, w, bias, out, keep);
    else conv_forward_tc<mm::kTf32>(g, u, in, w, bias, out, keep);
    return;
  }
  conv_forward_simt(g, in, w, bias, out);
}

// gradInput (when gin is given) and gradWeight / gradBias (when gw is) of one precision, sharing one transposition of gradOutput.
// `act`: the input's planes, or null (n0: the image of their record that they start with); w_ok / in_ok: whether the weight gradient / gradInput runs over planes.
template <int PREC>
static void conv_backward_group(const ConvGeom &g, const mm::Cells &u, bool in_ok, bool w_ok, const float *in, const void *act, const float *gout,
                                const float *w, float *gin, float *gw, float *gb, float scale, const Records &rec, long n0, const mm::UnpairPass<3> &unpair) {
  WsScope ws_scope;
  mm::ActPlanes pgo;
  mm::PairForm form;
  form.ranges = rec.joint(rec.gout);
  FilterForm<PREC, true> filter;
  if (in_ok) filter = grad_input_filter<PREC>(g, w, rec);
  auto make = [&](const auto &second) {
    return gw && g.K <= mm::most_sums<PREC>(g.oH * g.oW) ? mm::make_act_planes<PREC, true>(gout, g.N, g.K, g.oH, g.oW, nullptr, form, filter.pass, second)
                                                         : mm::make_act_planes<PREC, false>(gout, g.N, g.K, g.oH, g.oW, nullptr, form, filter.pass, second);
  };
  if (in_ok || w_ok) {
    if constexpr (PREC == mm::kPairs) pgo = make(unpair);
    else pgo = make(mm::NoPass{});
  }
  if (in_ok) {
    conv_grad_input_tc<PREC>(g, pgo, filter, gin, rec);
    if (PREC == mm::kPairs) add_strays<true>(g, gout, w, gin, rec);
  } else if (gin) {
    conv_grad_input_simt(g, gout, w, gin);
  }
  if (!gw) return;
  mm::ChanFinishPass bias;   // gradBias comes along with the transposition of gradOutput
  if (pgo.chan_partial) bias = mm::ChanFinishPass{(unsigned)((g.K + 7) / 8), pgo.chan_partial, pgo.chan_blocks, g.K, gb, scale};
  if (w_ok) {
    if (!act) {
      void *made = ws_alloc(mm::planes_bytes(g.N, (long)u.Hs * u.Ws, u.Cs, PREC));
      form.ranges = rec.joint(rec.act);
      restate_input<PREC>(g, u, in, made, form, {});
      act = made;
    }
    conv_acc_grad_tc<PREC>(g, u, act, pgo, gout, n0, gw, scale, rec, bias);
  } else {
    conv_acc_grad_simt(g, in, gout, gw, scale);
    mm::launch_passes(bias, 0, "conv_grad_bias_finish");
  }
  if (!bias.blocks) grad_bias(g, gout, gb, scale);
}
// False: there is no room for planes of this precision (kPairs), and nothing has been done.
template <int PREC>
static bool conv_backward_tc(const ConvGeom &g, const mm::Cells &u, bool restated, const float *in, const float *gout, const float *w, float *gin,
                             float *gw, float *gb, float scale, const THGPUTensor *finput) {
  const mm::Cells ui = grad_input_cells(g, PREC);
  const bool in_ok = gin && mm::windows_ok(grad_input_windows(g, ui, PREC)), w_ok = gw && restated;
  // the input's planes: those the forward pass left in finput (as the CPU nn path reuses its finput,
  // mcw_nn/generic/SpatialConvolutionMM.c:284-346), else made group by group
  const char *act = w_ok ? (const char *)planes_made_from(finput, in, g, u, PREC) : nullptr;
  const size_t act_image = w_ok ? mm::planes_bytes(1, (long)u.Hs * u.Ws, u.Cs, PREC) : 0;
  double bytes = 0;
  if (in_ok || w_ok) bytes += (double)mm::planes_bytes(1, g.P, mm::padded_channels(g.K, PREC), PREC);
  if (in_ok && !ui.direct) bytes += 4. * ui.Cr * ui.Hs * ui.Ws;
  if (w_ok && !act) bytes += (double)act_image;
  const long image = g.C * g.H * g.W, per = images_per_group(g.N, bytes, whole_scratch((double)g.N * (image + g.K * g.P)));
  // with the weights' forms, the measures (under a hundredth of the planes) and the partial sums (see gemm_pairs)
  if (PREC == mm::kPairs &&
      !ws_reserve((size_t)(1.01 * bytes * (double)per + 16. * (double)(g.K + 64) * std::max(u.kHs * u.kWs * (double)u.Cs, (double)g.R) + 96e6)))
    return false;
  for (long n0 = 0; n0 < g.N; n0 += per) {
    ConvGeom s = g;
    s.N = std::min(per, g.N - n0);
    const float *x = in ? in + n0 * image : nullptr, *go = gout + n0 * g.K * g.P;
    float *gi = gin ? gin + n0 * image : nullptr;
    ConvGeom t;
    mm::Cells ut;
    const bool layer = gin && grad_input_layer(s, PREC, t, ut), own = gin && !layer, own_ok = own && in_ok;
    if (own || gw) {
      WsScope ws_scope;
      Records rec;
      mm::UnpairPass<3> unpair;
      if constexpr (PREC == mm::kPairs) {   // (for each group: records last for some thousand words, see zeroed_words)
        rec.gout = mm::new_measured();
        if (own_ok) rec.weight = mm::new_measured();
        mm::RangeJob jw = mm::range_job_flat(w, g.K * g.R, rec.weight);
        mm::launch_ranges(mm::range_job_flat(go, s.N * g.K * g.P, rec.gout), own_ok ? &jw : nullptr);
        if (act) {
          mm::KeptRange *kept = planes_record(act);
          rec.act = mm::Measured{&kept->rec, kept->strays, true};
          const long pixels = g.N * u.Hs * u.Ws, most = 4l * ctx().sm_count;
          if (u.Cs <= mm::UnpairPass<3>::kMost) unpair = mm::UnpairPass<3>::of((void *)act, pixels, u.Cs, rec.joint(rec.act), &kept->rec, most);
          else mm::launch_passes(mm::UnpairPass<6>::of((void *)act, pixels, u.Cs, rec.joint(rec.act), &kept->rec, most), 0, "unpair");
        } else if (w_ok) {
          rec.act = mm::new_measured();
          mm::launch_ranges(mm::range_job_flat(x, s.N * image, rec.act), nullptr);
        }
      }
      conv_backward_group<PREC>(s, u, own_ok, w_ok, x, act ? act + n0 * act_image : nullptr, go, w, own ? gi : nullptr, gw, gb, scale, rec, act ? n0 : 0, unpair);
    }
    if (layer) {   // last: its own groups use up words
      WsScope ws_scope;
      conv_forward_tc<PREC>(t, ut, go, transposed_weight(s, w, true), nullptr, gi, nullptr);
    }
  }
  return true;
}
static void conv_backward(const ConvGeom &g, const float *in, const float *gout, const float *w, float *gin, float *gw, float *gb, float scale,
                          const THGPUTensor *finput) {
  if (ctx().math_mode == 1) {
    if (gin) conv_grad_input_simt(g, gout, w, gin);
    if (gw) {
      conv_acc_grad_simt(g, in, gout, gw, scale);
      grad_bias(g, gout, gb, scale);
    }
    return;
  }
  const bool hin = gin && half_grad_input(g), hw = gw && half_acc_grad(g);
  mm::Cells u;
  if (hin || hw) {
    const bool ok = restate(g, mm::kBf16, u);
    conv_backward_tc<mm::kBf16>(g, u, ok, in, gout, w, hin ? gin : nullptr, hw ? gw : nullptr, gb, scale, finput);
  }
  if ((gin && !hin) || (gw && !hw)) {
    int prec;
    // in the BF16 mode only for weight gradients: another last bit of a layer's result or gradInput would turn into others where the
    // next layer rounds it (the first layer's over 256 images: 385 -> 225 us)
    const bool ok = restate_accurate(g, ctx().math_mode == 0 || !gin || hin, u, prec);
    if (prec == mm::kPairs) {
      if (conv_backward_tc<mm::kPairs>(g, u, ok, in, gout, w, hin ? nullptr : gin, hw ? nullptr : gw, gb, scale, finput)) return;
      restate(g, mm::kTf32, u);
    }
    conv_backward_tc<mm::kTf32>(g, u, ok, in, gout, w, hin ? nullptr : gin, hw ? nullptr : gw, gb, scale, finput);
  }
}

static void check_grad_output(const ConvGeom &g, const THGPUTensor *gradOutput) {
  const int o = g.batch ? 1 : 0;
  THC_ARG(gradOutput->nDimension == (g.batch ? 4 : 3), 3, "gradOutput must have the rank of the output");
  THC_ARG(gradOutput->size[o] == g.K, 1, "Number of output features is not equal to nOutputPlane");
  THC_ARG(gradOutput->size[o + 1] == g.oH && gradOutput->size[o + 2] == g.oW && (!g.batch || gradOutput->size[0] == g.N), 3,
          "gradOutput has the wrong size");
}

}  // namespace thc

using namespace thc;

THC_API int THGPUNN_SpatialConvolutionMM_updateOutput(THGPUTensor *input, THGPUTensor *output, THGPUTensor *weight,
    THGPUTensor *bias, THGPUTensor *finput, THGPUTensor *fgradInput, int kW, int kH, int dW, int dH, int padding) {
  (void)fgradInput;
  THC_BEGIN
  forget_planes(finput);
  WsScope ws_scope;
  const ConvGeom g = conv_geom(input, weight, kW, kH, dW, dH, padding);
  THC_ARG(bias->nDimension == 1 && bias->size[0] == g.K, 1, "bias must have nOutputPlane entries");
  TensorRef in(tensor_new_contiguous(input)); TensorRef w(tensor_new_contiguous(weight)); TensorRef b(tensor_new_contiguous(bias));
  if (g.batch) { const long s[4] = {g.N, g.K, g.oH, g.oW}; resize_nd(output, 4, s, nullptr); }
  else { const long s[3] = {g.K, g.oH, g.oW}; resize_nd(output, 3, s, nullptr); }
  THC_CHECK(is_contiguous(output), "output must be contiguous");
  conv_forward(g, data_ptr(in), data_ptr(w), data_ptr(b), data_ptr(output), finput);
  return 0;
  THC_END(1)
}

THC_API int THGPUNN_SpatialConvolutionMM_updateGradInput(THGPUTensor *input, THGPUTensor *gradOutput, THGPUTensor *gradInput,
    THGPUTensor *weight, THGPUTensor *finput, THGPUTensor *fgradInput, int kW, int kH, int dW, int dH, int padding) {
  (void)finput; (void)fgradInput;
  THC_BEGIN
  WsScope ws_scope;
  const ConvGeom g = conv_geom(input, weight, kW, kH, dW, dH, padding);
  check_grad_output(g, gradOutput);
  TensorRef go(tensor_new_contiguous(gradOutput)); TensorRef w(tensor_new_contiguous(weight));
  tensor_resize_as(gradInput, input);
  THC_CHECK(is_contiguous(gradInput), "gradInput must be contiguous");
  conv_backward(g, nullptr, data_ptr(go), data_ptr(w), data_ptr(gradInput), nullptr, nullptr, 0.f, nullptr);
  return 0;
  THC_END(1)
}

THC_API int THGPUNN_SpatialConvolutionMM_accGradParameters(THGPUTensor *input, THGPUTensor *gradOutput, THGPUTensor *gradWeight,
    THGPUTensor *gradBias, THGPUTensor *finput, THGPUTensor *fgradInput, int kW, int kH, int dW, int dH, int padding, float scale) {
  (void)fgradInput;
  THC_BEGIN
  WsScope ws_scope;
  const ConvGeom g = conv_geom(input, gradWeight, kW, kH, dW, dH, padding);
  check_grad_output(g, gradOutput);
  THC_ARG(gradBias->nDimension == 1 && gradBias->size[0] == g.K, 1, "gradBias must have nOutputPlane entries");
  THC_CHECK(is_contiguous(gradWeight) && is_contiguous(gradBias), "gradWeight / gradBias must be contiguous");
  TensorRef in(tensor_new_contiguous(input)); TensorRef go(tensor_new_contiguous(gradOutput));
  conv_backward(g, data_ptr(in), data_ptr(go), nullptr, nullptr, data_ptr(gradWeight), data_ptr(gradBias), scale, finput);
  return 0;
  THC_END(1)
}

// updateGradInput (skipped when gradInput is null) followed by accGradParameters, sharing one transposition of
// gradOutput.  The reference has no such entry: nn.Module:backward calls the two methods one after the other
// (mcw_nn/Module.lua), and a GPU module may override backward with this.
THC_API int THGPUNN_SpatialConvolutionMM_backward(THGPUTensor *input, THGPUTensor *gradOutput, THGPUTensor *gradInput,
    THGPUTensor *weight, THGPUTensor *gradWeight, THGPUTensor *gradBias, THGPUTensor *finput, THGPUTensor *fgradInput,
    int kW, int kH, int dW, int dH, int padding, float scale) {
  (void)fgradInput;
  THC_BEGIN
  WsScope ws_scope;
  const ConvGeom g = conv_geom(input, weight, kW, kH, dW, dH, padding);
  check_grad_output(g, gradOutput);
  THC_ARG(gradWeight->nDimension == 2 && gradWeight->size[0] == g.K && gradWeight->size[1] == g.R, 1,
          "gradWeight must have the shape of weight");
  THC_ARG(gradBias->nDimension == 1 && gradBias->size[0] == g.K, 1, "gradBias must have nOutputPlane entries");
  THC_CHECK(is_contiguous(gradWeight) && is_contiguous(gradBias), "gradWeight / gradBias must be contiguous");
  TensorRef in(tensor_new_contiguous(input)); TensorRef go(tensor_new_contiguous(gradOutput)); TensorRef w(tensor_new_contiguous(weight));
  if (gradInput) {
    tensor_resize_as(gradInput, input);
    THC_CHECK(is_contiguous(gradInput), "gradInput must be contiguous");
  }
  conv_backward(g, data_ptr(in), data_ptr(go), data_ptr(w), gradInput ? data_ptr(gradInput) : nullptr, data_ptr(gradWeight), data_ptr(gradBias),
                scale, finput);
  return 0;
  THC_END(1)
}
