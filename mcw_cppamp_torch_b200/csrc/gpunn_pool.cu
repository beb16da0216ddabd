// nn.SpatialMaxPooling on torch.GPUTensor.
//
// Forward follows gputorch/lib/THC/gpunn-impl/SpatialMaxPooling.cpp:9-81,205-281 and the CPU
// kernel mcw_nn/generic/SpatialMaxPooling.c:5-56: window scanned rows-then-columns with a strict
// '>' so the first maximum wins; `indices` is a float tensor [2, (N,) C, oH, oW] holding the 1-based
// window-local row (plane 0) and column (plane 1) of the maximum.
// Backward: the reference GPU code only handled non-overlapping windows (:293-294) with a scatter;
// here every INPUT pixel gathers from the (at most ceil(kH/dH)*ceil(kW/dW)) windows that cover it,
// visiting them in ascending (y, x) order, which is the order in which the CPU loop
// (mcw_nn/generic/SpatialMaxPooling.c:147-176) adds them: no atomics, deterministic, and bit-equal
// to the CPU result for overlapping windows too.
#include <algorithm>
#include <cfloat>
#include <initializer_list>

#include "thc_internal.h"

namespace thc {

// 31-bit division by a runtime constant (multiply-high + shift): the kernels below decompose flat
// indices on every element, which 64-bit hardware division made the dominant cost.
struct Div32 {
  unsigned d, mul, shr;
  static Div32 make(long divisor) {
    Div32 f;
    f.d = (unsigned)divisor;
    if (divisor <= 1) { f.mul = 0; f.shr = 0; return f; }
    int lg = 0;
    while ((1l << lg) < divisor) lg++;
    const int p = 31 + lg;
    f.mul = (unsigned)(((1ull << p) + (unsigned long long)divisor - 1) / (unsigned long long)divisor);
    f.shr = (unsigned)(p - 32);
    return f;
  }
  __device__ __forceinline__ unsigned div(unsigned n) const { return d > 1 ? (__umulhi(n, mul) >> shr) : n; }
};

// Any window and stride: grid.y strides over planes, grid.x * block over the plane's outputs (no division by the plane size).
static __global__ void __launch_bounds__(256) maxpool_forward_kernel(const float *__restrict__ in, float *__restrict__ out,
                                                                     float *__restrict__ indy, float *__restrict__ indx,
                                                                     long planes, int H, int W, int oH, int oW, Div32 doW,
                                                                     int kH, int kW, int dH, int dW) {
  pdl_begin();
  const unsigned P = (unsigned)(oH * oW);
  for (long plane = blockIdx.y; plane < planes; plane += gridDim.y) {
    const float *ip0 = in + plane * H * W;
    const long ob = plane * P;
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < P; t += gridDim.x * blockDim.x) {
      const unsigned y = doW.div(t), x = t - y * oW;
      const float *ip = ip0 + (y * dH) * W + x * dW;
      float best = -INFINITY;  // the CPU starts from (float)(-DBL_MAX) = -inf
      int bi = -1, cnt = 0;
      for (int i = 0; i < kH; i++)
        for (int j = 0; j < kW; j++) {
          const float v = ip[i * W + j];
          if (v > best) { best = v; bi = cnt; }
          cnt++;
        }
      out[ob + t] = best;
      // bi == -1 (all NaN / -inf) reproduces the CPU's (int)(-1 / kW) + 1 and (-1 % kW) + 1
      indy[ob + t] = (float)(bi / kW + 1);
      indx[ob + t] = (float)(bi % kW + 1);
    }
  }
}

// One work item = G consecutive planes (small planes) or one band of input rows of one plane (large planes).
// Phase 1 turns every window that can reach the item's pixels into (flat position of its maximum, gradOutput
// value) in shared memory, reading indices and gradOutput exactly once and coalesced; phase 2 lets every input
// pixel scan the windows covering it.  Global traffic is the algorithmic minimum.
static __global__ void __launch_bounds__(256) maxpool_backward_kernel(const float *__restrict__ gout,
                                                                      const float *__restrict__ indy,
                                                                      const float *__restrict__ indx, float *__restrict__ gin,
                                                                      long planes, int H, int W, Div32 dW_in, int oH, int oW,
                                                                      Div32 doW, int kH, int kW, int dH, int dW, Div32 ddH,
                                                                      Div32 ddW, int G, int band_rows, int bands) {
  pdl_begin();
  extern __shared__ int pool_sm[];
  auto div_dH = [&](unsigned v) { return (int)ddH.div(v); };
  auto div_dW = [&](unsigned v) { return (int)ddW.div(v); };
  const int HW = H * W, oHW = oH * oW;
  const long groups = (planes + G - 1) / G;
  const long items = groups * bands;
  for (long item = blockIdx.x; item < items; item += gridDim.x) {
    const long grp = item / bands;
    const int band = (int)(item - grp * bands);
    const long p0 = grp * G;
    const int np = (int)(planes - p0 < G ? planes - p0 : G);
    const int h0 = band * band_rows, h1 = h0 + band_rows < H ? h0 + band_rows : H;
    // window rows that can cover input rows [h0, h1)
    int ylo = h0 - kH + 1;
    ylo = ylo <= 0 ? 0 : div_dH((unsigned)(ylo + dH - 1));
    int yhi = div_dH((unsigned)(h1 - 1));
    if (yhi > oH - 1) yhi = oH - 1;
    const int nwy = yhi >= ylo ? yhi - ylo + 1 : 0;
    const int nwin = nwy * oW;                 // per plane
    int *tgt = pool_sm;
    float *val = reinterpret_cast<float *>(pool_sm + np * nwin);
    for (int t = threadIdx.x; t < np * nwin; t += blockDim.x) {
      int pl = 0, r = t;
      if (np > 1) { pl = t / nwin; r = t - pl * nwin; }
      const int yy = (int)doW.div((unsigned)r), x = r - yy * oW, y = ylo + yy;
      const long o = (p0 + pl) * oHW + (long)y * oW + x;
      tgt[t] = ((int)indy[o] - 1 + y * dH) * W + ((int)indx[o] - 1 + x * dW);
      val[t] = gout[o];
    }
    __syncthreads();
    const int npix = (h1 - h0) * W;            // per plane
    for (int t = threadIdx.x; t < np * npix; t += blockDim.x) {
      int pl = 0, r = t;
      if (np > 1) { pl = t / npix; r = t - pl * npix; }
      const int hh = (int)dW_in.div((unsigned)r), w = r - hh * W, h = h0 + hh;
      // windows y with y*dH <= h <= y*dH + kH - 1, clipped to the output
      int y0 = h - kH + 1;
      y0 = y0 <= 0 ? 0 : div_dH((unsigned)(y0 + dH - 1));
      int y1 = div_dH((unsigned)h);
      if (y1 > oH - 1) y1 = oH - 1;
      int x0 = w - kW + 1;
      x0 = x0 <= 0 ? 0 : div_dW((unsigned)(x0 + dW - 1));
      int x1 = div_dW((unsigned)w);
      if (x1 > oW - 1) x1 = oW - 1;
      const int me = h * W + w;
      const int *tp = tgt + pl * nwin;
      const float *vp = val + pl * nwin;
      float acc = 0.f;
      for (int y = y0; y <= y1; y++)
        for (int x = x0; x <= x1; x++) {
          const int i = (y - ylo) * oW + x;
          if (tp[i] == me) acc += vp[i];
        }
      gin[(p0 + pl) * HW + (long)h0 * W + r] = acc;
    }
    __syncthreads();
  }
}

// The 2 x 2 and 3 x 3 windows at stride 2.  A group of LP lanes takes a band of kBand rows of one plane (planes of more than LP
// columns in tiles): all loads of the band are issued before the first is used, which is what keeps enough of them in flight
// (a walk with two rows' prefetch reached 60 % of the HBM rate), and no index arithmetic is left per element.
constexpr int kBand = 4;
struct PoolGeom {
  long planes;
  int H, W, oH, oW, xtiles, bands;   // bands of output rows (forward) or cell rows (backward, and forward with a threshold)
};
// nn.Threshold and the pooling behind it in one pass (template parameter TH of the kernels below): the thresholded plane, which is the
// pooling's input, is written while the pooling reads it, and on the way back the pooling's gradInput while the threshold reads it,
// instead of being written by one kernel and read again by the next.  Every pixel belongs to one band and one lane there, so the
// tiles cover whole planes and not only the windows.  Bound by HBM: of three passes over the plane forward and four backward one is
// gone (64 images of 64 x 224 x 224, 2 x 2 windows: 267 + 216 -> 363 us forward, 233 + 365 -> 507 backward).
struct ThresholdPass {
  const float *in = nullptr;   // backward: what the threshold was applied to
  float *out = nullptr;        // forward: the thresholded plane; backward: the threshold's gradInput
  float th = 0.f, val = 0.f;
};
// Rows of pixel pairs, columns 2b and 2b + 1 of each lane, leave as 8-byte accesses: on odd addresses as the pairs one column to the left.
// Every lane of the group takes part.  `first`: no lane of this tile stores the column to the left; `last`: nor the one to the right.
template <int LP>
struct PairStore {
  float *dst;
  bool odd;
  __device__ __forceinline__ explicit PairStore(float *d) : dst(d), odd((reinterpret_cast<uintptr_t>(d) & 4) != 0) {}
  __device__ __forceinline__ void row(float p0, float p1, bool c0, bool c1, bool first, bool last, int W) {
    const float left = __shfl_up_sync(0xffffffffu, p1, 1, LP);
    if (!odd) {
      if (c1) *reinterpret_cast<float2 *>(dst) = make_float2(p0, p1);
      else if (c0) dst[0] = p0;
    } else {
      if (c0) {
        if (!first) *reinterpret_cast<float2 *>(dst - 1) = make_float2(left, p0);
        else dst[0] = p0;
      }
      if (c1 && last) dst[1] = p1;
    }
    dst += W;
    odd ^= (W & 1) != 0;
  }
};

// Forward.  Lane `sub` owns window column x and reads input columns 2x and 2x + 1 of each row once (column 2x + 2 is the right-hand
// lane's first); a row's maximum over the window's columns serves both windows it belongs to: 4.5 loads an output where a
// thread per output issues 9.
template <int K, int LP, bool TH>
static __global__ void __launch_bounds__(256) maxpool_forward_band_kernel(const float *__restrict__ in, float *__restrict__ out,
                                                                          float *__restrict__ indy, float *__restrict__ indx, const PoolGeom p,
                                                                          const ThresholdPass t) {
  pdl_begin();
  constexpr int PPW = 32 / LP, ROWS = 2 * kBand + K - 2;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, sub = lane % LP, seg = lane / LP;
  const long warps = ((long)gridDim.x * blockDim.x) >> 5, warp0 = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned per_plane = (unsigned)(p.xtiles * p.bands);
  const long items = (p.planes + PPW - 1) / PPW * per_plane;
  for (long item = warp0; item < items; item += warps) {
    const long grp = item / per_plane;
    const unsigned r = (unsigned)(item - grp * per_plane), band = r / (unsigned)p.xtiles, xt = r - band * p.xtiles;
    const long plane = grp * PPW + seg;
    const int x = (int)xt * LP + sub, y0 = (int)band * kBand, h0 = 2 * y0;
    const bool live = plane < p.planes, l0 = live && 2 * x < p.W, l1 = live && 2 * x + 1 < p.W;
    const bool edge = K == 3 && sub == LP - 1 && live && 2 * x + 2 < p.W;   // the next lane's first column is in the next tile
    const float *src = in + (plane * p.H + h0) * (long)p.W + 2 * x;
    const float none = -INFINITY;   // the CPU starts from (float)(-DBL_MAX) = -inf
    float a[ROWS], b[ROWS], c[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; k++) {
      const bool ok = h0 + k < p.H;
      a[k] = ok && l0 ? src[k * p.W] : none;
      b[k] = ok && l1 ? src[k * p.W + 1] : none;
    }
    if (K == 3) {
#pragma unroll
      for (int k = 0; k < ROWS; k++) c[k] = edge && h0 + k < p.H ? src[k * p.W + 2] : none;
    }
    if constexpr (TH) {
      auto pass = [&](bool there, float v) { return !there || v > t.th ? v : t.val; };
#pragma unroll
      for (int k = 0; k < ROWS; k++) {
        const bool ok = h0 + k < p.H;
        a[k] = pass(ok && l0, a[k]); b[k] = pass(ok && l1, b[k]);
        if (K == 3) c[k] = pass(edge && ok, c[k]);
      }
      PairStore<LP> store(t.out + (plane * p.H + h0) * (long)p.W + 2 * x);
#pragma unroll
      for (int k = 0; k < 2 * kBand; k++)
        if (h0 + k < p.H) store.row(a[k], b[k], l0, l1, sub == 0, sub == LP - 1 || 2 * x + 2 >= p.W, p.W);
    }
    // maximum and its column of every row of the band (first one wins, NaN never does)
    float m[ROWS];
    int j[ROWS];
#pragma unroll
    for (int k = 0; k < ROWS; k++) {
      m[k] = none; j[k] = -1;
      if (a[k] > m[k]) { m[k] = a[k]; j[k] = 0; }
      if (b[k] > m[k]) { m[k] = b[k]; j[k] = 1; }
      if (K == 3) {
        const float n = __shfl_down_sync(full, a[k], 1, LP), cc = sub < LP - 1 ? n : c[k];
        if (cc > m[k]) { m[k] = cc; j[k] = 2; }
      }
    }
    if (live && x < p.oW) {
      const long o = (plane * p.oH + y0) * (long)p.oW + x;
#pragma unroll
      for (int y = 0; y < kBand; y++) {
        if (y0 + y >= p.oH) break;
        float best = m[2 * y];
        int bi = 0, bj = j[2 * y];
#pragma unroll
        for (int k = 1; k < K; k++)
          if (m[2 * y + k] > best) { best = m[2 * y + k]; bi = k; bj = j[2 * y + k]; }
        // nothing found (all NaN / -inf): row 1, column 0, the CPU's (int)(-1 / kW) + 1 and (-1 % kW) + 1
        out[o + y * p.oW] = best;
        indy[o + y * p.oW] = (float)(bi + 1);
        indx[o + y * p.oW] = (float)(bj + 1);
      }
    }
  }
}

// Backward for 3 x 3 windows.  Lane `sub` holds the windows (y, b) of its column and owns the four pixels of each cell (y, b), rows
// 2y and 2y + 1, columns 2b and 2b + 1.  Those are reached by windows (y-1, b-1), (y-1, b), (y, b-1), (y, b) only, whose
// target codes and values sit in this lane's and the left lane's registers: each pixel adds those that aim at it in that order,
// the CPU's order of additions (ascending window row, then column), so the result is bit-equal to it.  A row of the result
// leaves as 8-byte pairs, on odd addresses as the pairs one column to the left.
// Planes of more than 32 cells: tiles of 31 cells whose first lane holds the window left of the tile.
template <int LP, bool TH>
static __global__ void __launch_bounds__(256) maxpool3_backward_kernel(const float *__restrict__ gout, const float *__restrict__ indy,
                                                                       const float *__restrict__ indx, float *__restrict__ gin, const PoolGeom p,
                                                                       const ThresholdPass th) {
  pdl_begin();
  constexpr int PPW = 32 / LP;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, sub = lane % LP, seg = lane / LP;
  const long warps = ((long)gridDim.x * blockDim.x) >> 5, warp0 = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned per_plane = (unsigned)(p.xtiles * p.bands);
  const long items = (p.planes + PPW - 1) / PPW * per_plane;
  const bool halo = p.xtiles > 1;
  for (long item = warp0; item < items; item += warps) {
    const long grp = item / per_plane;
    const unsigned r = (unsigned)(item - grp * per_plane), band = r / (unsigned)p.xtiles, xt = r - band * p.xtiles;
    const long plane = grp * PPW + seg;
    const bool live = plane < p.planes;
    const int b = halo ? (int)xt * (LP - 1) + sub - 1 : sub, y0 = (int)band * kBand;
    const bool mine = live && b >= 0 && b < p.oW;
    const bool keep = live && !(halo && sub == 0), c0 = keep && 2 * b < p.W, c1 = keep && 2 * b + 1 < p.W;
    const long w0 = (plane * p.oH + y0) * (long)p.oW + b;
    // windows y0 - 1 .. y0 + kBand - 1: 3 * row + column of the target, counted from 1 (4 .. 12; 0: no window), and value
    float iy[kBand + 1], ix[kBand + 1], v[kBand + 1];
#pragma unroll
    for (int d = 0; d <= kBand; d++) {
      const bool ok = mine && (unsigned)(y0 + d - 1) < (unsigned)p.oH;
      const long o = w0 + (d - 1) * p.oW;
      iy[d] = ok ? indy[o] : 0.f; ix[d] = ok ? indx[o] : 0.f; v[d] = ok ? gout[o] : 0.f;
    }
    const long at = (plane * p.H + 2 * y0) * (long)p.W + 2 * b;
    float i0[2 * kBand], i1[2 * kBand];   // TH: what the threshold was applied to
    if constexpr (TH) {
#pragma unroll
      for (int k = 0; k < 2 * kBand; k++) {
        const bool ok = 2 * y0 + k < p.H;
        i0[k] = ok && c0 ? th.in[at + k * p.W] : 0.f;
        i1[k] = ok && c1 ? th.in[at + k * p.W + 1] : 0.f;
      }
    }
    PairStore<LP> store(gin + at), store_th(th.out + at);
    const bool first = sub <= (halo ? 1 : 0), last = sub == LP - 1 || 2 * b + 2 >= p.W;
    auto put = [&](int k, float p0, float p1) {
      store.row(p0, p1, c0, c1, first, last, p.W);
      if constexpr (TH) store_th.row(i0[k] > th.th ? p0 : 0.f, i1[k] > th.th ? p1 : 0.f, c0, c1, first, last, p.W);
    };
    auto add = [](float acc, bool hit, float x) { return hit ? acc + x : acc; };
    float pt = fmaf(3.f, iy[0], ix[0]), pv = v[0];
    float plt = __shfl_up_sync(full, pt, 1, LP), plv = __shfl_up_sync(full, pv, 1, LP);
    if (sub == 0) plt = 0.f;
#pragma unroll
    for (int d = 1; d <= kBand; d++) {
      if (2 * (y0 + d - 1) >= p.H) break;
      const float t = fmaf(3.f, iy[d], ix[d]), x = v[d];
      float lt = __shfl_up_sync(full, t, 1, LP);
      const float lx = __shfl_up_sync(full, x, 1, LP);
      if (sub == 0) lt = 0.f;
      const float p00 = add(add(add(add(0.f, plt == 12.f, plv), pt == 10.f, pv), lt == 6.f, lx), t == 4.f, x);
      const float p01 = add(add(0.f, pt == 11.f, pv), t == 5.f, x);
      const float p10 = add(add(0.f, lt == 9.f, lx), t == 7.f, x);
      const float p11 = add(0.f, t == 8.f, x);
      put(2 * d - 2, p00, p01);
      if (2 * (y0 + d - 1) + 1 < p.H) put(2 * d - 1, p10, p11);
      pt = t; pv = x; plt = lt; plv = lx;
    }
  }
}

// Backward for windows of 2 x 2 at stride 2: every pixel belongs to one window.  A thread owns V neighbouring windows and writes
// their 2 x 2V pixels (V = 2 where 16-byte stores are possible); rows and columns below and right of the last window are zero.
template <int V, bool TH>
static __global__ void __launch_bounds__(256) maxpool2_backward_kernel(const float *__restrict__ gout, const float *__restrict__ indy,
                                                                       const float *__restrict__ indx, float *__restrict__ gin, long rows,
                                                                       int H, int W, int oH, int oW, int cells_h, int cells_w, Div32 dcw,
                                                                       const ThresholdPass th) {
  pdl_begin();
  // rows = planes * cells_h; a cell row has cells_w / V items
  const int per = cells_w / V;
  for (long row0 = blockIdx.y; row0 * 64 < rows; row0 += gridDim.y) {
    const unsigned n = (unsigned)(min(64l, rows - row0 * 64) * per);
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
      const unsigned q = dcw.div(t);
      const int x = (int)(t - q * per) * V;
      const long row = row0 * 64 + q, plane = row / cells_h;
      const int y = (int)(row - plane * cells_h);
      const long at = (plane * H + 2 * y) * (long)W + 2 * x;
      const bool second = V == 2 || 2 * x + 1 < W, below = 2 * y + 1 < H;
      float top[2 * V], low[2 * V], in_top[2 * V], in_low[2 * V];   // in_*, TH: what the threshold was applied to
      auto load = [&](const float *s, float (&v)[2 * V]) {
        if constexpr (V == 2) {
          const float4 f = *reinterpret_cast<const float4 *>(s);
          v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else {
          v[0] = s[0];
          v[1] = second ? s[1] : 0.f;
        }
      };
      auto store = [&](float *d, const float (&v)[2 * V]) {
        if constexpr (V == 2) {
          *reinterpret_cast<float4 *>(d) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
          d[0] = v[0];
          if (second) d[1] = v[1];
        }
      };
      if constexpr (TH) {
        load(th.in + at, in_top);
        if (below) load(th.in + at + W, in_low);
      }
#pragma unroll
      for (int k = 0; k < V; k++) {
        float iy = 0.f, ix = 0.f, v = 0.f;
        if (y < oH && x + k < oW) {
          const long o = (plane * oH + y) * oW + x + k;
          iy = indy[o]; ix = indx[o]; v = gout[o];
        }
        v = __fadd_rn(v, 0.f);   // what the CPU's addition to a zeroed pixel leaves: -0 becomes +0
        top[2 * k] = iy == 1.f && ix == 1.f ? v : 0.f; top[2 * k + 1] = iy == 1.f && ix == 2.f ? v : 0.f;
        low[2 * k] = iy == 2.f && ix == 1.f ? v : 0.f; low[2 * k + 1] = iy == 2.f && ix == 2.f ? v : 0.f;
      }
      store(gin + at, top);
      if (below) store(gin + at + W, low);
      if constexpr (TH) {
#pragma unroll
        for (int k = 0; k < 2 * V; k++) { top[k] = in_top[k] > th.th ? top[k] : 0.f; low[k] = below && in_low[k] > th.th ? low[k] : 0.f; }
        store(th.out + at, top);
        if (below) store(th.out + at + W, low);
      }
    }
  }
}

// ---- the same windows over small planes -----------------------------------------------------------------------------------
// A block takes G whole planes, one stretch of memory, through shared memory: whatever the width, global memory is read and written in
// 16-byte pieces of that stretch.  Bound by HBM and by the barriers between a block's passes, of which other blocks of the SM make use.  The
// kernels by rows touch parts of sectors and lines at both ends of a row, which costs most on short rows and, once the tensors have
// left L2, in DRAM.  Threshold and 3 x 3 pooling in one pass, by rows -> by planes (us; the bytes at the copy rate): 65536 planes of
// 55 x 55 forward 462 -> 335 (330), backward 584 -> 476 (452); 196608 of 27 x 27 440 -> 235 (236), 600 -> 371 (324); 262144 of 13 x 13
// 150 -> 74 (72), 194 -> 125 (99).  Forward, five blocks an SM with six pieces of a thread on the way each: four pieces 340, 239, 77; eight without
// a bound on registers (119 of them, two blocks) 415, 296, 93.  Without a threshold, where five blocks spill 48 bytes a thread, four (8 bytes): 315, 227, 78 -> 279, 202, 68.
struct PlaneGeom {
  long planes;
  int G, H, W, HW, oH, oW, P;
  Div32 dP, doW;                    // outputs of a plane, of a row
  int cells, cw, ring;              // backward: 2 x 2 cells of a plane and of a row; windows of a plane with a ring of empty ones around
  Div32 dcells, dcw, dring, dS;
};
constexpr int kPlanePieces = 4;   // 16-byte pieces of a thread in the backward kernel: at most 4096 pixels a group
// f(i, n): global elements i .. i + n of [start, end), n = 4 on 16-byte boundaries, 1 at the ends; `U` pieces of a thread at once
// (load, then use).
template <int U, class Load, class Use>
__device__ __forceinline__ void stretch(long start, long end, Load load, Use use) {
  const long first = (start + 3) & ~3l, last = end & ~3l;
  for (long i0 = first + 4l * threadIdx.x; i0 < last; i0 += 4l * U * blockDim.x) {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i0 + 4l * u * blockDim.x < last) v[u] = load(i0 + 4l * u * blockDim.x);
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i0 + 4l * u * blockDim.x < last) use(i0 + 4l * u * blockDim.x, v[u]);
  }
}
// the up to three elements on either side of the 16-byte pieces
template <class One>
__device__ __forceinline__ void stretch_ends(long start, long end, One one) {
  const long first = min((start + 3) & ~3l, end), last = max(end & ~3l, first);
  const int t = threadIdx.x;
  if (t < first - start) one(start + t);
  if (t >= 32 && t - 32 < end - last) one(last + t - 32);
}

template <int K, bool TH>
static __global__ void __launch_bounds__(256, TH ? 5 : 4) maxpool_forward_planes_kernel(const float *__restrict__ in, float *__restrict__ out,
                                                                            float *__restrict__ indy, float *__restrict__ indx, const PlaneGeom q,
                                                                            const ThresholdPass t) {
  pdl_begin();
  extern __shared__ float4 planes_sm[];
  float *sm = reinterpret_cast<float *>(planes_sm);
  const long groups = (q.planes + q.G - 1) / q.G;
  auto pass = [&](float v) { return !TH || v > t.th ? v : t.val; };
  for (long g = blockIdx.x; g < groups; g += gridDim.x) {
    const long p0 = g * q.G, start = p0 * q.HW;
    const int np = (int)min((long)q.G, q.planes - p0);
    const long end = start + (long)np * q.HW, base = start & ~3l;
    stretch<6>(start, end, [&](long i) { return __ldg(reinterpret_cast<const float4 *>(in + i)); }, [&](long i, float4 v) {
      v = make_float4(pass(v.x), pass(v.y), pass(v.z), pass(v.w));
      if (TH) *reinterpret_cast<float4 *>(t.out + i) = v;
      *reinterpret_cast<float4 *>(sm + (i - base)) = v;
    });
    stretch_ends(start, end, [&](long i) {
      const float v = pass(in[i]);
      if (TH) t.out[i] = v;
      sm[i - base] = v;
    });
    __syncthreads();
    const float *src = sm + (start - base);
    for (unsigned o = threadIdx.x; o < (unsigned)(np * q.P); o += blockDim.x) {
      const unsigned pl = q.dP.div(o), r = o - pl * q.P, y = q.doW.div(r), x = r - y * q.oW;
      const float *w = src + pl * q.HW + 2 * y * q.W + 2 * x;
      float best = -INFINITY;   // as in the kernels above, nothing found included
      int bi = 0, bj = -1;
#pragma unroll
      for (int i = 0; i < K; i++)
#pragma unroll
        for (int j = 0; j < K; j++) {
          const float v = w[i * q.W + j];
          if (v > best) { best = v; bi = i; bj = j; }
        }
      const long at = p0 * q.P + o;
      out[at] = best;
      indy[at] = (float)(bi + 1);
      indx[at] = (float)(bj + 1);
    }
    __syncthreads();
  }
}
// The windows' targets and values go to shared memory first, in a ring of empty windows; a thread then makes the four pixels of a cell from
// the four windows that reach it (see maxpool3_backward_kernel; 2 x 2 windows: from the one), and the pixels leave as one stretch.
template <int K, bool TH>
static __global__ void __launch_bounds__(256) maxpool_backward_planes_kernel(const float *__restrict__ gout, const float *__restrict__ indy,
                                                                             const float *__restrict__ indx, float *__restrict__ gin, const PlaneGeom q,
                                                                             const ThresholdPass th) {
  pdl_begin();
  extern __shared__ float4 planes_sm[];
  float *px = reinterpret_cast<float *>(planes_sm);
  float2 *win = reinterpret_cast<float2 *>(px + (q.G * q.HW + 7) / 4 * 4);
  const long groups = (q.planes + q.G - 1) / q.G;
  const int S = q.oW + 2;
  for (long g = blockIdx.x; g < groups; g += gridDim.x) {
    const long p0 = g * q.G, start = p0 * q.HW;
    const int np = (int)min((long)q.G, q.planes - p0);
    const long end = start + (long)np * q.HW, base = start & ~3l;
    // every load of the group is under way before the first is waited for
    const long first = (start + 3) & ~3l, last = end & ~3l;
    float4 x[kPlanePieces];
    if constexpr (TH) {
#pragma unroll
      for (int u = 0; u < kPlanePieces; u++) {
        const long i = first + 4l * (threadIdx.x + 256 * u);
        if (i < last) x[u] = __ldg(reinterpret_cast<const float4 *>(th.in + i));
      }
    }
    const unsigned rings = (unsigned)(np * q.ring);
    for (unsigned c0 = threadIdx.x; c0 < rings; c0 += 256 * kPlanePieces) {
      float iy[kPlanePieces], ix[kPlanePieces], v[kPlanePieces];
#pragma unroll
      for (int u = 0; u < kPlanePieces; u++) {
        const unsigned c = c0 + 256 * u, pl = q.dring.div(c), r = c - pl * q.ring, yy = q.dS.div(r), xx = r - yy * S;
        const bool there = c < rings && yy - 1 < (unsigned)q.oH && xx - 1 < (unsigned)q.oW;
        const long o = (p0 + pl) * q.P + (int)(yy - 1) * q.oW + (int)(xx - 1);
        iy[u] = there ? indy[o] : 0.f; ix[u] = there ? indx[o] : 0.f; v[u] = there ? gout[o] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kPlanePieces; u++)   // 3 * row + column of the target, counted from 1 (4 .. 12; 0: no window), and value
        if (c0 + 256 * u < rings) win[c0 + 256 * u] = make_float2(fmaf(3.f, iy[u], ix[u]), v[u]);
    }
    __syncthreads();
    auto add = [](float acc, bool hit, float x) { return hit ? acc + x : acc; };
    for (unsigned c = threadIdx.x; c < (unsigned)(np * q.cells); c += blockDim.x) {
      const unsigned pl = q.dcells.div(c), r = c - pl * q.cells, cy = q.dcw.div(r), cx = r - cy * q.cw;
      const float2 *b = win + pl * q.ring + (cy + 1) * S + cx + 1;
      const float2 w = b[0];
      float p00, p01, p10, p11;
      if (K == 3) {
        const float2 l = b[-1], u = b[-S], ul = b[-S - 1];
        p00 = add(add(add(add(0.f, ul.x == 12.f, ul.y), u.x == 10.f, u.y), l.x == 6.f, l.y), w.x == 4.f, w.y);
        p01 = add(add(0.f, u.x == 11.f, u.y), w.x == 5.f, w.y);
        p10 = add(add(0.f, l.x == 9.f, l.y), w.x == 7.f, w.y);
        p11 = add(0.f, w.x == 8.f, w.y);
      } else {
        p00 = add(0.f, w.x == 4.f, w.y); p01 = add(0.f, w.x == 5.f, w.y);
        p10 = add(0.f, w.x == 7.f, w.y); p11 = add(0.f, w.x == 8.f, w.y);
      }
      float *d = px + (start - base) + pl * q.HW + 2 * cy * q.W + 2 * cx;
      const bool right = 2 * cx + 1 < (unsigned)q.W, below = 2 * cy + 1 < (unsigned)q.H;
      d[0] = p00;
      if (right) d[1] = p01;
      if (below) d[q.W] = p10;
      if (below && right) d[q.W + 1] = p11;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPlanePieces; u++) {
      const long i = first + 4l * (threadIdx.x + 256 * u);
      if (i >= last) break;
      float4 v = *reinterpret_cast<const float4 *>(px + (i - base));
      *reinterpret_cast<float4 *>(gin + i) = v;
      if constexpr (TH) {
        v = make_float4(x[u].x > th.th ? v.x : 0.f, x[u].y > th.th ? v.y : 0.f, x[u].z > th.th ? v.z : 0.f, x[u].w > th.th ? v.w : 0.f);
        *reinterpret_cast<float4 *>(th.out + i) = v;
      }
    }
    stretch_ends(start, end, [&](long i) {
      const float v = px[i - base];
      gin[i] = v;
      if (TH) th.out[i] = th.in[i] > th.th ? v : 0.f;
    });
    __syncthreads();
  }
}
// By rows: lanes of a plane, and the share of lanes and band rows with work, in percent.
static long rows_lanes(long cw) { return cw <= 8 ? 8 : cw <= 16 ? 16 : 32; }
static long rows_fill(long w, long lanes, long h) { return 100 * w * h / (lanes * ((h + kBand - 1) / kBand * kBand)); }
// Planes per block, or G = 0 where the kernels by rows do better (us, by rows / by planes, threshold included; without one see rows_alone).
//   Few pixels: 174 planes of 43 x 35 (0.3 M) forward 4.7 / 6.3, backward 5.2 / 7.0; 400 of 31 x 100 (1.2 M) 6.5 / 5.5, 6.6 / 5.9; 8192 of 13 x 13 (1.4 M) 8.2 /
//     6.4, 11.3 / 7.5; 1024 of 55 x 55 (3.1 M) 10.3 / 8.5, 11.0 / 10.0.
//   Forward: 54 114 / 80, 56 116 / 99 (its columns meet in the same banks), 100 216 / 175; 2 x 2 54 94 / 81, 60 109 / 102, but 100 164 / 169.
//   Backward: 3 x 3 by planes wherever a group fits; 28 82 / 71, 56 144 / 120.  2 x 2 by rows, which leave in whole sectors for
//     widths of whole 16-byte pieces and meet in L2 otherwise, as long as the tensors stay there: 28 63 / 78, 14 17.7 / 22, 24576 of 27 x 27 (18 M pixels)
//     48 / 53, 196608 (143 M) 418 / 354, 65536 of 55 x 55 570 / 468, 262144 of 13 x 13 122 / 129, 16384 of 54 x 54 (48 M) 130 / 119.
//   Below 2^20 pixels, behind a threshold, where rows leave half their lanes idle (from 2^18 on three fifths; the two modules by themselves / rows / planes): 0.6 M of
//     11 x 5, 3 x 3 forward 6.9 / 8.5 / 4.4, backward 8.0 / 10.3 / 5.8, 2 x 2 forward 6.4 / 7.7 / 4.2; 0.3 M of 9 x 9 4.3 / 5.4 / 3.8, 5.9 / 6.2 / 5.0; 0.9 M of 17 x 17 6.6 / 8.3 / 5.0, 8.7 / 10.6 / 6.2.
static PlaneGeom plane_geom(long planes, long H, long W, long oH, long oW, int k, bool backward, bool threshold, size_t &smem) {
  PlaneGeom q = {};
  q.planes = planes; q.H = (int)H; q.W = (int)W; q.HW = (int)std::min(H * W, 1l << 30); q.oH = (int)oH; q.oW = (int)oW; q.P = (int)(oH * oW);
  const long ch = (H + 1) / 2, cw = (W + 1) / 2, ring = (oH + 2) * (oW + 2), bytes = 4 * H * W + (backward ? 8 * ring : 0), pixels = planes * H * W;
  if (bytes > 47 * 1024 || pixels < 1l << 18) return q;
  if (pixels < 1l << 20 && (!threshold || rows_fill(cw, (cw + rows_lanes(cw) - 1) / rows_lanes(cw) * rows_lanes(cw), ch) >= (pixels < 1l << 19 ? 40 : 50))) return q;
  if (!backward && k == 2 && W > 64 && W % 2 == 0) return q;
  if (backward && H * W > 1024 * kPlanePieces) return q;
  if (backward && k == 2 && (W % 4 == 0 || W <= 16 || pixels < 40l << 20)) return q;
  q.G = (int)std::max(1l, std::min(backward ? std::min(1024 * kPlanePieces / (H * W), 47 * 1024 / bytes) : 24 * 1024 / bytes, planes / (4l * ctx().sm_count)));
  q.cells = (int)(ch * cw); q.cw = (int)cw; q.ring = (int)ring;
  q.dP = Div32::make(q.P); q.doW = Div32::make(oW); q.dcells = Div32::make(q.cells); q.dcw = Div32::make(cw); q.dring = Div32::make(ring); q.dS = Div32::make(oW + 2);
  smem = (size_t)(4 * ((q.G * q.HW + 7) / 4 * 4) + (backward ? 8l * q.G * ring : 0));
  return q;
}
// Pooling by itself moves a third to a half less, and rows do better wherever they keep their lanes busy (fill: rows_fill).
// us, by rows / by planes, 24 M pixels (6 times as many: the same within a tenth, unless noted).
//   Forward, 3 x 3: 9 columns (fill 50) 49 / 41, 13 (56) 47 / 41, 16 (77) 37 / 45, 19 (42) 59 / 43, 23 (63) 45 / 45, 25 (75) 41 / 46, 31 (88) 39 / 44,
//     33 (50) 55 / 45, 42 (62) 45 / 45, 46 (63) 45 / 47, 55 (81) 39 / 45, 64 (94) 35 / 47, 72 (53) 47 / 40, 97 (75) 41 / 47.
//     2 x 2: 14 (77) 39 / 37, six times as many 204 / 155; 16 (100) 35 / 38, 22 (63) 37 / 37 and 210 / 178, 27 (66) 39 / 37, 28 (77) 37 / 39, 39 (56) 37 / 37, 56 (88) 35 / 45.
//   Backward, 3 x 3: even widths, whose rows leave in whole pairs, 12 (56) 1 / 0.94, 14 (77) 1 / 1.14, 22 (63) 1 / 0.92, 24 (75) 1 / 1.0, 28 (77) 43 / 45, 32 (100) 37 / 45, 36 (51) 53 / 43,
//     44 (63) 45 / 43; odd ones 13 (77) 61 / 49, 15 (100) 45 / 51, 23 (75) 61 / 49, 29 (88) 53 / 43, 31 (100) 45 / 47, 45 (69) 47 / 45.  One plane a group, 46 to 64: 43 / 53 to 35 / 42.
//     2 x 2: groups that fill little of a block, 46 and 47, 143 M pixels: 221 / 246, 213 / 240; 50 and more 1 / 0.84 to 1.
static bool rows_alone(const PlaneGeom &q, int k, bool backward) {
  const long ch = (q.H + 1) / 2, LP = rows_lanes(q.cw);
  if (!backward) return rows_fill(q.oW, (q.oW + LP - 1) / LP * LP, q.oH) >= (LP == 32 ? 63 : k == 2 && LP == 8 ? 80 : 70);
  if (k == 2) return 10l * q.G * q.HW < 6l * 1024 * kPlanePieces;
  return q.G == 1 || rows_fill(q.cw, q.cw <= 32 ? LP : (q.cw + 30) / 31 * 32, ch) >= (q.W % 2 ? 90 : 70);
}
static unsigned plane_blocks(const PlaneGeom &q) { return (unsigned)std::min((q.planes + q.G - 1) / q.G, (long)ctx().sm_count * 64); }

static unsigned band_blocks(const PoolGeom &p, int planes_per_warp) {
  const long items = (p.planes + planes_per_warp - 1) / planes_per_warp * p.xtiles * p.bands;
  return (unsigned)std::min((items + 7) / 8, (long)ctx().sm_count * 64);
}
// The 2 x 2 and 3 x 3 windows at stride 2, behind a threshold (TH) or by themselves.
template <bool TH>
static void forward_bands(const float *src, float *o, float *iy, float *ix, long planes, long H, long W, long oH, long oW, int k, const ThresholdPass &t) {
  size_t smem = 0;
  const PlaneGeom q = plane_geom(planes, H, W, oH, oW, k, false, TH, smem);
  if (q.G && (TH || !rows_alone(q, k, false)) && (((uintptr_t)src | (uintptr_t)t.out) & 15) == 0) {
    auto go = [&](auto kernel) { pdl_launch(kernel, plane_blocks(q), 256, smem, src, o, iy, ix, q, t); };
    if (k == 3) go(maxpool_forward_planes_kernel<3, TH>); else go(maxpool_forward_planes_kernel<2, TH>);
    check_launch("maxpool_forward");
    return;
  }
  // lanes per plane: as many as it has window columns, up to a warp; wider planes are cut into tiles of 32 columns
  const long cells_h = (H + 1) / 2, cells_w = (W + 1) / 2;
  const int LP = cells_w <= 8 ? 8 : cells_w <= 16 ? 16 : 32;
  const PoolGeom pg{planes, (int)H, (int)W, (int)oH, (int)oW, (int)(((TH ? cells_w : oW) + LP - 1) / LP), (int)(((TH ? cells_h : oH) + kBand - 1) / kBand)};
  auto go = [&](auto kernel) { pdl_launch(kernel, band_blocks(pg, 32 / LP), 256, 0, src, o, iy, ix, pg, t); };
  if (k == 3) { if (LP == 8) go(maxpool_forward_band_kernel<3, 8, TH>); else if (LP == 16) go(maxpool_forward_band_kernel<3, 16, TH>); else go(maxpool_forward_band_kernel<3, 32, TH>); }
  else { if (LP == 8) go(maxpool_forward_band_kernel<2, 8, TH>); else if (LP == 16) go(maxpool_forward_band_kernel<2, 16, TH>); else go(maxpool_forward_band_kernel<2, 32, TH>); }
  check_launch("maxpool_forward");
}
static bool banded(int kW, int kH, int dW, int dH) { return dH == 2 && dW == 2 && kH == kW && (kH == 2 || kH == 3); }
// False: windows or sizes of another kind, nothing has been done.
template <bool TH>
static bool backward_cells(const float *g, const float *iy, const float *ix, float *gi, long planes, long H, long W, long oH, long oW, int k,
                           const ThresholdPass &t) {
  size_t smem = 0;
  const PlaneGeom q = plane_geom(planes, H, W, oH, oW, k, true, TH, smem);
  if (q.G && (TH || !rows_alone(q, k, true)) && (((uintptr_t)gi | (uintptr_t)t.in | (uintptr_t)t.out) & 15) == 0) {
    auto go = [&](auto kernel) { pdl_launch(kernel, plane_blocks(q), 256, smem, g, iy, ix, gi, q, t); };
    if (k == 3) go(maxpool_backward_planes_kernel<3, TH>); else go(maxpool_backward_planes_kernel<2, TH>);
    check_launch("maxpool_backward");
    return true;
  }
  const long cells_h = (H + 1) / 2, cells_w = (W + 1) / 2;
  if (k == 3) {
    const int LP = cells_w <= 8 ? 8 : cells_w <= 16 ? 16 : 32;
    const int xtiles = cells_w <= 32 ? 1 : (int)((cells_w + 30) / 31);
    const PoolGeom pg{planes, (int)H, (int)W, (int)oH, (int)oW, xtiles, (int)((cells_h + kBand - 1) / kBand)};
    auto go = [&](auto kernel) { pdl_launch(kernel, band_blocks(pg, 32 / LP), 256, 0, g, iy, ix, gi, pg, t); };
    if (LP == 8) go(maxpool3_backward_kernel<8, TH>); else if (LP == 16) go(maxpool3_backward_kernel<16, TH>); else go(maxpool3_backward_kernel<32, TH>);
    check_launch("maxpool_backward");
    return true;
  }
  if (cells_w >= (1l << 24)) return false;
  const bool vec = W % 4 == 0 && (((uintptr_t)gi | (uintptr_t)t.in | (uintptr_t)t.out) & 15) == 0;
  const long rows = planes * cells_h, per = vec ? cells_w / 2 : cells_w;
  const unsigned bx = (unsigned)std::min<long>((64 * per + 255) / 256, 16);
  const unsigned by = (unsigned)std::min<long>((rows + 63) / 64, std::max<long>(1, ctx().sm_count * 32l / bx));
  auto go = [&](auto kernel) {
    pdl_launch(kernel, dim3(bx, by), 256, 0, g, iy, ix, gi, rows, (int)H, (int)W, (int)oH, (int)oW, (int)cells_h, (int)cells_w, Div32::make(per), t);
  };
  if (vec) go(maxpool2_backward_kernel<2, TH>); else go(maxpool2_backward_kernel<1, TH>);
  check_launch("maxpool_backward");
  return true;
}
static dim3 plane_grid(long planes, long per_plane) {
  long gx = (per_plane + 255) / 256;
  if (gx > 64) gx = 64;
  long gy = planes;
  const long cap = (long)ctx().sm_count * 32;
  if (gx * gy > cap) gy = cap / gx > 0 ? cap / gx : 1;
  if (gy > 65535) gy = 65535;
  return dim3((unsigned)gx, (unsigned)gy, 1);
}

// ---- SpatialAveragePooling (gputorch/lib/THC/gpunn-impl/SpatialAveragePooling.cpp:9-62 forward, :130-182
// backward; CPU mcw_nn/generic/SpatialAveragePooling.c:5-80, :84-150).  In this code base the module writes the
// window SUM, neither path divides by the window size.  Forward: one thread per output, the window summed in
// FP32 row by row as the CPU does.  Backward: one thread per INPUT pixel adds the gradOutput of every window that
// covers it in ascending (y, x) order, the order in which the CPU's scatter reaches that pixel, so the result is
// bit-equal to the CPU's and overlapping windows work (the reference GPU path refuses dW != kW, :194-195).
static __global__ void __launch_bounds__(256) sumpool_forward_kernel(const float *__restrict__ in, float *__restrict__ out,
                                                                     long planes, int H, int W, int oH, int oW, int kH, int kW,
                                                                     int dH, int dW) {
  pdl_begin();
  const long total = planes * oH * oW;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const int x = (int)(t % oW);
    const long q = t / oW;
    const int y = (int)(q % oH);
    const long pl = q / oH;
    const float *p = in + (pl * H + (long)y * dH) * W + (long)x * dW;
    float sum = 0.f;
    for (int ky = 0; ky < kH; ky++, p += W)
      for (int kx = 0; kx < kW; kx++) sum += p[kx];
    out[t] = sum;
  }
}
static __global__ void __launch_bounds__(256) sumpool_backward_kernel(const float *__restrict__ gout, float *__restrict__ gin,
                                                                      long planes, int H, int W, int oH, int oW, int kH, int kW,
                                                                      int dH, int dW) {
  pdl_begin();
  const long total = planes * H * W;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const int w = (int)(t % W);
    const long q = t / W;
    const int h = (int)(q % H);
    const long pl = q / H;
    // windows (y, x) with y*dH <= h < y*dH + kH
    int y0 = h - kH + 1; y0 = y0 <= 0 ? 0 : (y0 + dH - 1) / dH;
    int x0 = w - kW + 1; x0 = x0 <= 0 ? 0 : (x0 + dW - 1) / dW;
    int y1 = h / dH; if (y1 > oH - 1) y1 = oH - 1;
    int x1 = w / dW; if (x1 > oW - 1) x1 = oW - 1;
    const float *g = gout + pl * oH * oW;
    float sum = 0.f;
    for (int y = y0; y <= y1; y++)
      for (int x = x0; x <= x1; x++) sum += g[y * oW + x];
    gin[t] = sum;
  }
}

}  // namespace thc

using namespace thc;

THC_API int THGPUNN_SpatialMaxPooling_updateOutput(THGPUTensor *input, THGPUTensor *output, THGPUTensor *indices,
                                                   int kW, int kH, int dW, int dH) {
  THC_BEGIN
  THC_ARG(input->nDimension == 3 || input->nDimension == 4, 2, "3D or 4D (batch) tensor expected");
  THC_ARG(kW > 0 && kH > 0 && dW > 0 && dH > 0, 1, "invalid kernel / stride");
  const bool batch = input->nDimension == 4;
  const int o = batch ? 1 : 0;
  const long N = batch ? input->size[0] : 1, C = input->size[o], H = input->size[o + 1], W = input->size[o + 2];
  THC_ARG(W >= kW && H >= kH, 2, "input image smaller than kernel size");
  const long oH = (H - kH) / dH + 1, oW = (W - kW) / dW + 1;
  TensorRef in(tensor_new_contiguous(input));
  if (batch) {
    const long s[4] = {N, C, oH, oW}, si[5] = {2, N, C, oH, oW};
    resize_nd(output, 4, s, nullptr);
    resize_nd(indices, 5, si, nullptr);
  } else {
    const long s[3] = {C, oH, oW}, si[4] = {2, C, oH, oW};
    resize_nd(output, 3, s, nullptr);
    resize_nd(indices, 4, si, nullptr);
  }
  THC_CHECK(is_contiguous(output) && is_contiguous(indices), "output / indices must be contiguous");
  const long total = N * C * oH * oW;
  THC_CHECK(H * W < (1l << 31), "image plane too large");
  if (total > 0) {
    const float *src = data_ptr(in);
    float *o = data_ptr(output), *iy = data_ptr(indices), *ix = iy + total;
    if (banded(kW, kH, dW, dH)) {
      forward_bands<false>(src, o, iy, ix, N * C, H, W, oH, oW, kH, {});
    } else {
      pdl_launch(maxpool_forward_kernel, plane_grid(N * C, oH * oW), 256, 0, src, o, iy, ix, N * C, (int)H, (int)W, (int)oH, (int)oW,
                                                                               Div32::make(oW), kH, kW, dH, dW);
      check_launch("maxpool_forward");
    }
  }
  return 0;
  THC_END(1)
}

THC_API int THGPUNN_SpatialMaxPooling_updateGradInput(THGPUTensor *input, THGPUTensor *gradOutput, THGPUTensor *gradInput,
                                                      THGPUTensor *indices, int kW, int kH, int dW, int dH) {
  THC_BEGIN
  THC_ARG(input->nDimension == 3 || input->nDimension == 4, 2, "3D or 4D (batch) tensor expected");
  const bool batch = input->nDimension == 4;
  const int o = batch ? 1 : 0;
  const long N = batch ? input->size[0] : 1, C = input->size[o], H = input->size[o + 1], W = input->size[o + 2];
  THC_ARG(W >= kW && H >= kH, 2, "input image smaller than kernel size");
  const long oH = (H - kH) / dH + 1, oW = (W - kW) / dW + 1;
  THC_ARG(gradOutput->nDimension == input->nDimension && gradOutput->size[o] == C && gradOutput->size[o + 1] == oH &&
              gradOutput->size[o + 2] == oW && (!batch || gradOutput->size[0] == N), 3, "gradOutput has the wrong size");
  THC_ARG(nelem(indices) == 2 * N * C * oH * oW, 1, "indices do not belong to this input");
  TensorRef go(tensor_new_contiguous(gradOutput)); TensorRef ind(tensor_new_contiguous(indices));
  tensor_resize_as(gradInput, input);
  THC_CHECK(is_contiguous(gradInput), "gradInput must be contiguous");
  const long total = N * C * H * W, ototal = N * C * oH * oW;
  THC_CHECK(H * W < (1l << 31), "image plane too large");
  if (total > 0) {
    const float *g = data_ptr(go), *iy = data_ptr(ind), *ix = iy + ototal;
    float *gi = data_ptr(gradInput);
    if (banded(kW, kH, dW, dH) && backward_cells<false>(g, iy, ix, gi, N * C, H, W, oH, oW, kH, {})) return 0;
    // shared memory holds (position, value) of up to kMaxWin windows per work item
    const int kMaxWin = 5120;
    int G = 1, band_rows = (int)H, bands = 1;
    if (oH * oW <= kMaxWin) {
      // whole planes; several per block when they are small, so that a block has ~8 K pixels between barriers
      G = (int)(8192 / (H * W));
      if (G < 1) G = 1;
      if (G * oH * oW > kMaxWin) G = (int)(kMaxWin / (oH * oW));
      if (G > N * C) G = (int)(N * C);
    } else {
      long wrows = kMaxWin / oW;            // window rows that fit
      THC_CHECK(wrows >= 2 + (kH + dH - 1) / dH, "pooling window row too wide for the backward kernel");
      band_rows = (int)((wrows - 1 - (kH + dH - 1) / dH) * dH);
      if (band_rows < 1) band_rows = 1;
      bands = (int)((H + band_rows - 1) / band_rows);
    }
    const long items = ((N * C + G - 1) / G) * bands;
    // shared memory actually needed per work item: (position, value) per window
    const size_t smem = bands > 1 ? (size_t)kMaxWin * 8 : (size_t)G * oH * oW * 8;
    long blocks = items;
    const long cap = (long)ctx().sm_count * 8;
    if (blocks > cap) blocks = cap;
    pdl_launch(maxpool_backward_kernel, (unsigned)blocks, 256, smem, g, iy, ix, gi, N * C, (int)H, (int)W, Div32::make(W), (int)oH, (int)oW,
                                                                       Div32::make(oW), kH, kW, dH, dW, Div32::make(dH), Div32::make(dW), G,
                                                                       band_rows, bands);
    check_launch("maxpool_backward");
  }
  return 0;
  THC_END(1)
}

// nn.Threshold followed by nn.SpatialMaxPooling.  What the two entry points in turn give, to the bit, and by them wherever the pass over
// both does not apply: other windows, strided or overlapping tensors, arguments that one of them refuses.
// Whether resizing and writing any of `results` leaves the others and `sources` as they are: no storage is shared, and none of a result's memory,
// which goes back when the result outgrows it, is borrowed by another (THGPUStorage_newWithData).  `sources`: contiguous.
static bool apart(std::initializer_list<const THGPUTensor *> results, std::initializer_list<const THGPUTensor *> sources) {
  auto meets = [](const THGPUTensor *r, const THGPUTensor *o, const float *a, long n) {
    return o == r || (r->storage && (o->storage == r->storage || (a && a < r->storage->data + r->storage->size && r->storage->data < a + n)));
  };
  for (const THGPUTensor *r : results) {
    for (const THGPUTensor *o : results)
      if (o < r && meets(r, o, o->storage ? o->storage->data : nullptr, o->storage ? o->storage->size : 0)) return false;
    for (const THGPUTensor *o : sources)
      if (meets(r, o, data_ptr(o), nelem(o))) return false;
  }
  return true;
}
static bool pooled_shape(const THGPUTensor *t, int kW, int kH, int dW, int dH, long s[6]) {   // planes, H, W, oH, oW, and N for a batch (else 0)
  if ((t->nDimension != 3 && t->nDimension != 4) || !banded(kW, kH, dW, dH) || !is_contiguous(t)) return false;
  const int o = t->nDimension - 3;
  s[5] = o ? t->size[0] : 0;
  s[0] = (o ? t->size[0] : 1) * t->size[o]; s[1] = t->size[o + 1]; s[2] = t->size[o + 2];
  if (s[0] <= 0 || s[1] < kH || s[2] < kW || s[1] * s[2] >= (1l << 31)) return false;
  s[3] = (s[1] - kH) / 2 + 1; s[4] = (s[2] - kW) / 2 + 1;
  return true;
}

THC_API int THGPUNN_Threshold_SpatialMaxPooling_updateOutput(THGPUTensor *input, THGPUTensor *thresholded, THGPUTensor *output, THGPUTensor *indices,
                                                             double threshold, double val, int kW, int kH, int dW, int dH) {
  THC_BEGIN
  long s[6];
  if (thresholded != output && thresholded != indices && output != indices && pooled_shape(input, kW, kH, dW, dH, s) &&
      apart({thresholded, output, indices}, {input})) {
    const long C = s[0] / (s[5] ? s[5] : 1), so[4] = {s[5], C, s[3], s[4]}, si[5] = {2, s[5], C, s[3], s[4]}, si3[4] = {2, C, s[3], s[4]};
    tensor_resize_as(thresholded, input);
    if (s[5]) { resize_nd(output, 4, so, nullptr); resize_nd(indices, 5, si, nullptr); }
    else { resize_nd(output, 3, so + 1, nullptr); resize_nd(indices, 4, si3, nullptr); }
    if (is_contiguous(thresholded) && is_contiguous(output) && is_contiguous(indices)) {
      float *ind = data_ptr(indices);
      forward_bands<true>(data_ptr(input), data_ptr(output), ind, ind + nelem(output), s[0], s[1], s[2], s[3], s[4], kH,
                          ThresholdPass{nullptr, data_ptr(thresholded), (float)threshold, (float)val});
      return 0;
    }
  }
  const int bad = THGPUNN_Threshold_updateOutput(input, thresholded, threshold, val);
  return bad ? bad : THGPUNN_SpatialMaxPooling_updateOutput(thresholded, output, indices, kW, kH, dW, dH);
  THC_END(1)
}

THC_API int THGPUNN_Threshold_SpatialMaxPooling_updateGradInput(THGPUTensor *input, THGPUTensor *thresholded, THGPUTensor *gradOutput,
                                                                THGPUTensor *poolGradInput, THGPUTensor *gradInput, THGPUTensor *indices,
                                                                double threshold, int kW, int kH, int dW, int dH) {
  THC_BEGIN
  long s[6];
  if (pooled_shape(input, kW, kH, dW, dH, s) && THGPUTensor_isSameSizeAs(input, thresholded) && gradOutput->nDimension == input->nDimension &&
      is_contiguous(gradOutput) && is_contiguous(indices)) {
    const int o = input->nDimension - 3;
    const long m = s[0] * s[3] * s[4];
    const bool sizes = (!o || gradOutput->size[0] == input->size[0]) && gradOutput->size[o] == input->size[o] && gradOutput->size[o + 1] == s[3] &&
                       gradOutput->size[o + 2] == s[4] && nelem(indices) == 2 * m;
    if (sizes && poolGradInput != gradInput && apart({poolGradInput, gradInput}, {input, gradOutput, indices}) && poolGradInput != thresholded &&
        gradInput != thresholded) {
      tensor_resize_as(poolGradInput, input);
      tensor_resize_as(gradInput, input);
      const float *ind = data_ptr(indices);
      if (is_contiguous(poolGradInput) && is_contiguous(gradInput) &&
          backward_cells<true>(data_ptr(gradOutput), ind, ind + m, data_ptr(poolGradInput), s[0], s[1], s[2], s[3], s[4], kH,
                               ThresholdPass{data_ptr(input), data_ptr(gradInput), (float)threshold, 0.f}))
        return 0;
    }
  }
  const int bad = THGPUNN_SpatialMaxPooling_updateGradInput(thresholded, gradOutput, poolGradInput, indices, kW, kH, dW, dH);
  return bad ? bad : THGPUNN_Threshold_updateGradInput(input, poolGradInput, gradInput, threshold);
  THC_END(1)
}

THC_API int THGPUNN_SpatialAveragePooling_updateOutput(THGPUTensor *input, THGPUTensor *output, int kW, int kH, int dW, int dH) {
  THC_BEGIN
  THC_ARG(input->nDimension == 3 || input->nDimension == 4, 2, "3D or 4D(batch mode) tensor expected");
  THC_ARG(kW > 0 && kH > 0 && dW > 0 && dH > 0, 1, "invalid kernel / stride");
  const bool batch = input->nDimension == 4;
  const int o = batch ? 1 : 0;
  const long N = batch ? input->size[0] : 1, C = input->size[o], H = input->size[o + 1], W = input->size[o + 2];
  THC_ARG(W >= kW && H >= kH, 2, "input image smaller than kernel size");
  const long oH = (H - kH) / dH + 1, oW = (W - kW) / dW + 1;
  TensorRef in(tensor_new_contiguous(input));
  if (batch) { const long s[4] = {N, C, oH, oW}; resize_nd(output, 4, s, nullptr); }
  else { const long s[3] = {C, oH, oW}; resize_nd(output, 3, s, nullptr); }
  THC_CHECK(is_contiguous(output), "output must be contiguous");
  const long total = N * C * oH * oW;
  if (total > 0) {
    long blocks = (total + 255) / 256;
    if (blocks > (long)ctx().sm_count * 16) blocks = (long)ctx().sm_count * 16;
    pdl_launch(sumpool_forward_kernel, (unsigned)blocks, 256, 0, data_ptr(in), data_ptr(output), N * C, (int)H, (int)W, (int)oH,
                                                                  (int)oW, kH, kW, dH, dW);
    check_launch("SpatialAveragePooling_updateOutput");
  }
  return 0;
  THC_END(1)
}

THC_API int THGPUNN_SpatialAveragePooling_updateGradInput(THGPUTensor *input, THGPUTensor *gradOutput, THGPUTensor *gradInput,
                                                          int kW, int kH, int dW, int dH) {
  THC_BEGIN
  THC_ARG(input->nDimension == 3 || input->nDimension == 4, 2, "3D or 4D(batch mode) tensor expected");
  THC_ARG(kW > 0 && kH > 0 && dW > 0 && dH > 0, 1, "invalid kernel / stride");
  const bool batch = input->nDimension == 4;
  const int o = batch ? 1 : 0;
  const long N = batch ? input->size[0] : 1, C = input->size[o], H = input->size[o + 1], W = input->size[o + 2];
  THC_ARG(W >= kW && H >= kH, 2, "input image smaller than kernel size");
  const long oH = (H - kH) / dH + 1, oW = (W - kW) / dW + 1;
  THC_ARG(gradOutput->nDimension == input->nDimension && gradOutput->size[o] == C && gradOutput->size[o + 1] == oH &&
              gradOutput->size[o + 2] == oW && (!batch || gradOutput->size[0] == N), 3, "gradOutput has the wrong size");
  TensorRef go(tensor_new_contiguous(gradOutput));
  tensor_resize_as(gradInput, input);
  THC_CHECK(is_contiguous(gradInput), "gradInput must be contiguous");
  const long total = N * C * H * W;
  if (total > 0) {
    long blocks = (total + 255) / 256;
    if (blocks > (long)ctx().sm_count * 16) blocks = (long)ctx().sm_count * 16;
    pdl_launch(sumpool_backward_kernel, (unsigned)blocks, 256, 0, data_ptr(go), data_ptr(gradInput), N * C, (int)H, (int)W, (int)oH,
                                                                   (int)oW, kH, kW, dH, dW);
    check_launch("SpatialAveragePooling_updateGradInput");
  }
  return 0;
  THC_END(1)
}
