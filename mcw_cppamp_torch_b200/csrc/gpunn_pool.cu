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
  int H, W, oH, oW, xtiles, bands;   // bands of output rows (forward) or cell rows (backward)
};

// Forward.  Lane `sub` owns window column x and reads input columns 2x and 2x + 1 of each row once (column 2x + 2 is the right-hand
// lane's first); a row's maximum over the window's columns serves both windows it belongs to: 4.5 loads an output where a
// thread per output issues 9.
template <int K, int LP>
static __global__ void __launch_bounds__(256) maxpool_forward_band_kernel(const float *__restrict__ in, float *__restrict__ out,
                                                                          float *__restrict__ indy, float *__restrict__ indx, const PoolGeom p) {
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
template <int LP>
static __global__ void __launch_bounds__(256) maxpool3_backward_kernel(const float *__restrict__ gout, const float *__restrict__ indy,
                                                                       const float *__restrict__ indx, float *__restrict__ gin, const PoolGeom p) {
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
    float *dst = gin + (plane * p.H + 2 * y0) * (long)p.W + 2 * b;
    bool odd = (reinterpret_cast<uintptr_t>(dst) & 4) != 0;
    auto put = [&](float p0, float p1) {
      const float left = __shfl_up_sync(full, p1, 1, LP);
      if (!odd) {
        if (c1) *reinterpret_cast<float2 *>(dst) = make_float2(p0, p1);
        else if (c0) dst[0] = p0;
      } else {
        // the pair (2b - 1, 2b); the first lane of a row has no left column, the last column of an even row no right one
        if (c0) {
          if (sub > (halo ? 1 : 0)) *reinterpret_cast<float2 *>(dst - 1) = make_float2(left, p0);
          else dst[0] = p0;
        }
        if (c1 && (sub == LP - 1 || 2 * b + 2 >= p.W)) dst[1] = p1;
      }
      dst += p.W;
      odd ^= (p.W & 1) != 0;
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
      put(p00, p01);
      if (2 * (y0 + d - 1) + 1 < p.H) put(p10, p11);
      pt = t; pv = x; plt = lt; plv = lx;
    }
  }
}

// Backward for windows of 2 x 2 at stride 2: every pixel belongs to one window.  A thread owns V neighbouring windows and writes
// their 2 x 2V pixels (V = 2 where 16-byte stores are possible); rows and columns below and right of the last window are zero.
template <int V>
static __global__ void __launch_bounds__(256) maxpool2_backward_kernel(const float *__restrict__ gout, const float *__restrict__ indy,
                                                                       const float *__restrict__ indx, float *__restrict__ gin, long rows,
                                                                       int H, int W, int oH, int oW, int cells_h, int cells_w, Div32 dcw) {
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
      float top[2 * V], low[2 * V];
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
      float *d = gin + (plane * H + 2 * y) * (long)W + 2 * x;
      if constexpr (V == 2) {
        *reinterpret_cast<float4 *>(d) = make_float4(top[0], top[1], top[2], top[3]);
        if (2 * y + 1 < H) *reinterpret_cast<float4 *>(d + W) = make_float4(low[0], low[1], low[2], low[3]);
      } else {
        const bool second = 2 * x + 1 < W;
        d[0] = top[0];
        if (second) d[1] = top[1];
        if (2 * y + 1 < H) {
          d[W] = low[0];
          if (second) d[W + 1] = low[1];
        }
      }
    }
  }
}

static unsigned band_blocks(const PoolGeom &p, int planes_per_warp) {
  const long items = (p.planes + planes_per_warp - 1) / planes_per_warp * p.xtiles * p.bands;
  return (unsigned)std::min((items + 7) / 8, (long)ctx().sm_count * 64);
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
    if (dH == 2 && dW == 2 && kH == kW && (kH == 2 || kH == 3)) {
      // lanes per plane: as many as it has window columns, up to a warp; wider planes are cut into tiles of 32 columns
      const int LP = (W + 1) / 2 <= 8 ? 8 : (W + 1) / 2 <= 16 ? 16 : 32;
      const int xtiles = (int)((oW + LP - 1) / LP);
      const PoolGeom pg{N * C, (int)H, (int)W, (int)oH, (int)oW, xtiles, (int)((oH + kBand - 1) / kBand)};
#define THC_POOL_FWD(K, LPV) pdl_launch(maxpool_forward_band_kernel<K, LPV>, band_blocks(pg, 32 / LP), 256, 0, src, o, iy, ix, pg)
      if (kH == 3) { if (LP == 8) THC_POOL_FWD(3, 8); else if (LP == 16) THC_POOL_FWD(3, 16); else THC_POOL_FWD(3, 32); }
      else { if (LP == 8) THC_POOL_FWD(2, 8); else if (LP == 16) THC_POOL_FWD(2, 16); else THC_POOL_FWD(2, 32); }
#undef THC_POOL_FWD
    } else {
      pdl_launch(maxpool_forward_kernel, plane_grid(N * C, oH * oW), 256, 0, src, o, iy, ix, N * C, (int)H, (int)W, (int)oH, (int)oW,
                                                                               Div32::make(oW), kH, kW, dH, dW);
    }
    check_launch("maxpool_forward");
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
    const long cells_h = (H + 1) / 2, cells_w = (W + 1) / 2;
    if (dH == 2 && dW == 2 && kH == 3 && kW == 3) {
      const int LP = cells_w <= 8 ? 8 : cells_w <= 16 ? 16 : 32;
      const int xtiles = cells_w <= 32 ? 1 : (int)((cells_w + 30) / 31);
      const PoolGeom pg{N * C, (int)H, (int)W, (int)oH, (int)oW, xtiles, (int)((cells_h + kBand - 1) / kBand)};
#define THC_POOL_BWD3(LPV) pdl_launch(maxpool3_backward_kernel<LPV>, band_blocks(pg, 32 / LP), 256, 0, g, iy, ix, gi, pg)
      if (LP == 8) THC_POOL_BWD3(8); else if (LP == 16) THC_POOL_BWD3(16); else THC_POOL_BWD3(32);
#undef THC_POOL_BWD3
      check_launch("maxpool_backward");
      return 0;
    }
    if (dH == 2 && dW == 2 && kH == 2 && kW == 2 && cells_w < (1l << 24)) {
      const bool vec = W % 4 == 0 && ((uintptr_t)gi & 15) == 0;
      const long rows = N * C * cells_h, per = vec ? cells_w / 2 : cells_w;
      const unsigned bx = (unsigned)std::min<long>((64 * per + 255) / 256, 16);
      const unsigned by = (unsigned)std::min<long>((rows + 63) / 64, std::max<long>(1, ctx().sm_count * 32l / bx));
      if (vec) pdl_launch(maxpool2_backward_kernel<2>, dim3(bx, by), 256, 0, g, iy, ix, gi, rows, (int)H, (int)W, (int)oH, (int)oW, (int)cells_h, (int)cells_w, Div32::make(per));
      else pdl_launch(maxpool2_backward_kernel<1>, dim3(bx, by), 256, 0, g, iy, ix, gi, rows, (int)H, (int)W, (int)oH, (int)oW, (int)cells_h, (int)cells_w, Div32::make(per));
      check_launch("maxpool_backward");
      return 0;
    }
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
