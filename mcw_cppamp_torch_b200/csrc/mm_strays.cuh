// Values that FP16 pairs do not hold (Stray, mm_problem.cuh), added to the results of products in FP32.
//
// Each result takes the strays of one operand against all of the other operand, and the strays of that against what the pairs hold of the
// first.  A block owns the results it changes and takes the strays in their listed order, so that sums repeat exactly.  Without
// strays, the usual case of all but the largest tensors, a launch looks at two counts and ends (about 2 us as a programmatic
// dependent); each stray of an activation costs a block about a microsecond, one of the weights a pass over a plane.
// The weight gradient's are added by UnpackGradPass (mm_planes.cuh).
#ifndef THC_MM_STRAYS_CUH
#define THC_MM_STRAYS_CUH

#include "mm_planes.cuh"

namespace thc {
namespace mm {

// Forward: src = input, out [N][K][oH][oW]; GRAD_INPUT: src = gradOutput, out [N][C][H][W].  Block (a, b) owns the images a, a + gridDim.x,
// ... of the result's planes b, b + gridDim.y, ...
template <bool GRAD_INPUT>
static __global__ void __launch_bounds__(256) window_strays_kernel(const float *src, const float *w, float *out, const LayerShape l,
                                                                   const Measured act, const Measured weight, const Ranges ranges) {
  pdl_begin();
  const bool wide = ranges.wide();
  const int na = act.strays(wide), nw = weight.strays(wide);
  if (na + nw == 0) return;
  const int Cs = GRAD_INPUT ? l.K : l.C, Hs = GRAD_INPUT ? l.oH : l.H, Ws = GRAD_INPUT ? l.oW : l.W;
  const int Co = GRAD_INPUT ? l.C : l.K, Ho = GRAD_INPUT ? l.H : l.oH, Wo = GRAD_INPUT ? l.W : l.oW;
  const int taps = l.kH * l.kW, mine = (Co - (int)blockIdx.y + (int)gridDim.y - 1) / (int)gridDim.y;   // (gridDim.y <= Co)
  for (int e = 0; e < na; e++) {
    const long at = act.list[e].at, row = at / Ws, plane = row / Hs, n = plane / Cs;
    if (n % gridDim.x != blockIdx.x) continue;
    const int x = (int)(at - row * Ws), y = (int)(row - plane * Hs), c = (int)(plane - n * Cs);
    const float v = act.list[e].v;
    for (long t = threadIdx.x; t < (long)mine * taps; t += 256) {
      const int co = (int)(blockIdx.y + t / taps * gridDim.y), tap = (int)(t % taps), i = tap / l.kW, j = tap - i * l.kW;
      int oy, ox;
      if (GRAD_INPUT) {
        oy = y * l.dH + i - l.pad; ox = x * l.dW + j - l.pad;
        if (oy < 0 || ox < 0) continue;
      } else {
        const int ty = y + l.pad - i, tx = x + l.pad - j;
        oy = ty / l.dH; ox = tx / l.dW;
        if (ty < 0 || tx < 0 || oy * l.dH != ty || ox * l.dW != tx) continue;
      }
      if (oy >= Ho || ox >= Wo) continue;
      const long k = GRAD_INPUT ? (long)c * l.C + co : (long)co * l.C + c;
      out[((n * Co + co) * Ho + oy) * (long)Wo + ox] += v * w[k * taps + tap];
    }
    __syncthreads();   // (another thread may take the same result next)
  }
  const unsigned limit = stray_limit(act.rec->max_bits) - 1u;
  for (int e = 0; e < nw; e++) {
    const long at = weight.list[e].at, k = at / taps;
    const int tap = (int)(at - k * taps), i = tap / l.kW, j = tap - i * l.kW, ko = (int)(k / l.C), ci = (int)(k - (long)ko * l.C);
    const int co = GRAD_INPUT ? ci : ko, c = GRAD_INPUT ? ko : ci;
    if (co % gridDim.y != blockIdx.y) continue;
    const float v = weight.list[e].v;
    for (long n = blockIdx.x; n < l.N; n += gridDim.x)
      for (int t = threadIdx.x; t < Ho * Wo; t += 256) {
        const int oy = t / Wo, ox = t - oy * Wo;
        int y, x;
        if (GRAD_INPUT) {
          const int ty = oy + l.pad - i, tx = ox + l.pad - j;
          y = ty / l.dH; x = tx / l.dW;
          if (ty < 0 || tx < 0 || y * l.dH != ty || x * l.dW != tx) continue;
        } else {
          y = oy * l.dH + i - l.pad; x = ox * l.dW + j - l.pad;
          if (y < 0 || x < 0) continue;
        }
        if (y >= Hs || x >= Ws) continue;
        const float s = src[((n * Cs + c) * Hs + y) * (long)Ws + x];
        if ((__float_as_uint(s) & 0x7fffffffu) - 1u >= limit) out[((n * Co + co) * Ho + oy) * (long)Wo + ox] += v * s;   // (zeros pass)
      }
    __syncthreads();
  }
}

// D(m, n) += alpha * ...: element (r, l) of a side at p[r * ld + l] (along_k) or p[l * ld + r], measured as `run` values a line.  Block (a, b)
// owns the columns of a 256-wide chunk, rows b, b + gridDim.y, ...; a thread owns a column, then a row.
struct StraySide { const float *p; long ld, run; int along_k; Measured m; };
static __global__ void __launch_bounds__(256) matrix_strays_kernel(const StraySide x, const StraySide y, long M, long N, const Epilogue epi,
                                                                   const Ranges ranges) {
  pdl_begin();
  const bool wide = ranges.wide();
  const int nx = x.m.strays(wide), ny = y.m.strays(wide);
  if (nx + ny == 0) return;
  auto place = [](const StraySide &s, int e, long &r, long &l) {
    const long at = s.m.list[e].at, line = at / s.run, c = at - line * s.run;
    r = s.along_k ? line : c;
    l = s.along_k ? c : line;
  };
  const unsigned limit = stray_limit(x.m.rec->max_bits) - 1u;
  for (long n0 = blockIdx.x * 256l; n0 < N; n0 += gridDim.x * 256l) {
    const long n = n0 + threadIdx.x;
    for (int e = 0; n < N && e < nx; e++) {
      long r, l;
      place(x, e, r, l);
      if (r % gridDim.y == blockIdx.y)
        epi.out[epi.moff(r) + n * epi.nstride] += epi.alpha * (x.m.list[e].v * y.p[y.along_k ? n * y.ld + l : l * y.ld + n]);
    }
    __syncthreads();   // rows, from here on
    for (int e = 0; e < ny; e++) {
      long c, l;
      place(y, e, c, l);
      if (c < n0 || c >= n0 + 256) continue;
      for (long m = blockIdx.y + (long)threadIdx.x * gridDim.y; m < M; m += 256l * gridDim.y) {
        const float s = x.p[x.along_k ? m * x.ld + l : l * x.ld + m];
        if ((__float_as_uint(s) & 0x7fffffffu) - 1u >= limit) epi.out[epi.moff(m) + c * epi.nstride] += epi.alpha * (y.m.list[e].v * s);
      }
    }
    __syncthreads();
  }
}

}  // namespace mm
}  // namespace thc

#endif
