// Passes over operands and results of the matrix-multiply engines: ranges and FP16 pairs, channels-last planes and cells, repacked
// weights, folds of partial sums.
#ifndef THC_MM_PLANES_CUH
#define THC_MM_PLANES_CUH

#include "mm_problem.cuh"

namespace thc {
namespace mm {

// The halves of scaled values; strays (subnormal hi) leave zeros.
__device__ __forceinline__ void split_pair(float a, float b, __half2 &hi, __half2 &lo) {
  a = fabsf(a) < 0x1p-14f ? 0.f : a;
  b = fabsf(b) < 0x1p-14f ? 0.f : b;
  hi = __floats2half2_rn(a, b);
  const float2 h = __half22float2(hi);
  lo = __floats2half2_rn((a - h.x) * 2048.f, (b - h.y) * 2048.f);
}
__device__ __forceinline__ float join_pair(__half hi, __half lo, float unscale) { return (__half2float(hi) + __half2float(lo) * 0x1p-11f) * unscale; }
__device__ __forceinline__ unsigned half2_bits(const __half2 &h) { return *reinterpret_cast<const unsigned *>(&h); }

// Ranges of up to two operands (blockIdx.y), `lines` x `run` values with pitch ld.  A warp looks at a set of 512 values at a time, in
// four groups of 128: neighbours in memory (`flat`), or 128 neighbours in each of four lines.  The last block to finish lists the
// strays: from the smallest value of each block's sets and of each set (set_low) it knows where to look again, so that
// the few strays of a large tensor cost it a few microseconds.  The list is in the order of `at`: results do not depend on who came first.
struct RangeJob {
  const float *p;
  long lines, run, ld;
  int flat, vec;
  RangeRec *rec;
  Stray *list;
  unsigned blocks;      // that look at it, of the launch's
  uint2 *block_range;   // a block's largest and smallest
  unsigned *set_low;
};
constexpr int kRangeBlocks = 2048;   // a launch has no more for an operand
struct RangeSets {
  const RangeJob &j;
  long total, segs, count;
  __device__ __forceinline__ RangeSets(const RangeJob &job) : j(job) {
    total = j.lines * j.run;
    segs = j.flat ? (total + 511) / 512 : (j.run + 127) / 128;
    count = j.flat ? segs : segs * ((j.lines + 3) / 4);
  }
  // the 16 values of this lane; at[g]: the place of the first of group g
  __device__ __forceinline__ void load(long s, int lane, unsigned (&v)[4][4], long (&at)[4]) const {
    const long q = j.flat ? 0 : s / segs, c0 = j.flat ? s * 512 : (s - q * segs) * 128;
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const long line = j.flat ? 0 : q * 4 + g, c = c0 + (j.flat ? g * 128 : 0) + lane * 4, end = j.flat ? total : line < j.lines ? j.run : 0;
      const float *src = j.p + line * j.ld + c;
      at[g] = line * j.run + c;
      if (j.vec && c + 4 <= end) {
        const uint4 u = __ldg(reinterpret_cast<const uint4 *>(src));
        v[g][0] = u.x; v[g][1] = u.y; v[g][2] = u.z; v[g][3] = u.w;
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) v[g][i] = c + i < end ? __float_as_uint(__ldg(src + i)) : 0u;
      }
    }
  }
};
static __global__ void __launch_bounds__(256, 5) range_kernel(const RangeJob ja, const RangeJob jb) {
  pdl_begin();
  const RangeJob &j = blockIdx.y ? jb : ja;
  if (blockIdx.x >= j.blocks) return;
  const RangeSets sets(j);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long warps = j.blocks * 8l, me = (long)blockIdx.x * 8 + warp;
  unsigned most = 0, low = ~0u;   // the lows as bits - 1: zero becomes the largest
  for (long k = me; k < sets.count; k += warps) {
    const long s = sets.count - 1 - k;   // from the end, which whoever wrote the operand has left in L2, to the start, which the next pass reads first
    unsigned v[4][4], m = ~0u;
    long at[4];
    sets.load(s, lane, v, at);
#pragma unroll
    for (int g = 0; g < 4; g++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const unsigned x = v[g][i] & 0x7fffffffu;
        most = max(most, x);
        m = min(m, x - 1u);
      }
    m = __reduce_min_sync(0xffffffffu, m);
    if (lane == 0) j.set_low[s] = m;
    low = min(low, m);
  }
  __shared__ unsigned sm[2][8];
  __shared__ int last, found, nblocks;
  __shared__ Stray buf[kStrays];
  __shared__ unsigned short blocks[kRangeBlocks];
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0) { sm[0][warp] = most; sm[1][warp] = low; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) { most = max(most, sm[0][w]); low = min(low, sm[1][w]); }
    j.block_range[blockIdx.x] = make_uint2(most, low);
    __threadfence();
    last = atomicAdd(&j.rec->ticket, 1u) == j.blocks - 1;
    found = nblocks = 0;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  uint2 r[kRangeBlocks / 256];   // all of them on the way at once
#pragma unroll
  for (int i = 0; i < kRangeBlocks / 256; i++) r[i] = i * 256 + threadIdx.x < j.blocks ? __ldcg(j.block_range + i * 256 + threadIdx.x) : make_uint2(0, ~0u);
  most = 0;
#pragma unroll
  for (int i = 0; i < kRangeBlocks / 256; i++) most = max(most, r[i].x);
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0) sm[0][warp] = most;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; w++) most = max(most, sm[0][w]);
  if (threadIdx.x == 0) j.rec->max_bits = most;
  const unsigned limit = stray_limit(most) - 1u;   // (as the lows: bits - 1)
  if (!most || max_is_wide(most)) return;
  const int allowed = (int)min((long)kStrays, stray_allowance(sets.total));
#pragma unroll
  for (int i = 0; i < kRangeBlocks / 256; i++)
    if (r[i].y < limit) blocks[atomicAdd(&nblocks, 1)] = (unsigned short)(i * 256 + threadIdx.x);
  __syncthreads();
  // a warp takes a block's sets, 128 at a time: set q is the block's warp q % 8's in its round q / 8
  const long rounds = (sets.count + warps - 1) / warps;
  bool stop = false;   // the same for a warp's lanes, as all that the loops below depend on
  for (int b = warp; b < nblocks && !stop; b += 8) {
    const long first = blocks[b] * 8l;
    for (long q0 = 0; q0 < rounds * 8 && !stop; q0 += 128) {
      unsigned l[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const long q = q0 + i * 32 + lane, k = q / 8 * warps + first + q % 8;
        l[i] = k < sets.count ? __ldcg(j.set_low + sets.count - 1 - k) : ~0u;
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
        for (unsigned hit = __ballot_sync(0xffffffffu, l[i] < limit); hit && !stop; hit &= hit - 1) {
          const long q = q0 + i * 32 + __ffs(hit) - 1;
          unsigned v[4][4];
          long at[4];
          sets.load(sets.count - 1 - (q / 8 * warps + first + q % 8), lane, v, at);
#pragma unroll
          for (int g = 0; g < 4; g++)
#pragma unroll
            for (int e = 0; e < 4; e++)
              if ((v[g][e] & 0x7fffffffu) - 1u < limit) {
                const int n = atomicAdd(&found, 1);
                if (n < kStrays) buf[n] = Stray{at[g] + e, __uint_as_float(v[g][e])};
              }
          __syncwarp();
          stop = __shfl_sync(0xffffffffu, *const_cast<volatile int *>(&found), 0) > allowed;
        }
    }
  }
  __syncthreads();
  const int n = found;
  if (n > allowed) {
    if (threadIdx.x == 0) j.rec->wide = 1;
    return;
  }
  for (int i = threadIdx.x; i < n; i += 256) {
    int rank = 0;
    for (int o = 0; o < n; o++) rank += buf[o].at < buf[i].at;
    j.list[rank] = buf[i];
  }
  if (threadIdx.x == 0) j.rec->strays = n;
}

// Passes that do not read one another's results share a launch: the blocks of `first`, then those of `second`, then `main`'s.  Each is a
// struct of its arguments with run(block), its number of blocks of 256 threads (none: not asked for) and how many an SM has to have room for
// (kPerSM, of `main`).  A launch of its own, by the time
// the next one has waited for it, costs a small pass two to four microseconds more than its work.
struct NoPass {
  static constexpr int kPerSM = 1;
  static constexpr unsigned blocks = 0;
  __device__ __forceinline__ void run(unsigned) const {}
};
template <class Main, class First, class Second>
static __global__ void __launch_bounds__(256, Main::kPerSM) passes_kernel(const __grid_constant__ Main main, const __grid_constant__ First first,
                                                            const __grid_constant__ Second second) {
  pdl_begin();
  unsigned block = blockIdx.x;
  if (block < first.blocks) { first.run(block); return; }
  block -= first.blocks;
  if (block < second.blocks) { second.run(block); return; }
  main.run(block - second.blocks);
}

// What a kernel that writes an operand's planes needs in kPairs.
struct PairForm {
  Ranges ranges;
  KeptRange *keep = nullptr;     // where the operand's measures go when the planes outlive the call ...
  const Stray *list = nullptr;   // ... and its list
  __device__ __forceinline__ void end(bool wide, unsigned block) const {
    if (!keep || block) return;
    const RangeRec r = *ranges.rec[0];
    const int n = wide ? 0 : (int)r.strays;
    if (threadIdx.x == 0) {
      keep->rec = r;
      keep->rec.wide = wide; keep->rec.ticket = 0; keep->rec.strays = n;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) keep->strays[i] = list[i];
  }
};

// Kept planes back to FP32, in place, where another operand asks for it: 24 bits of almost every value (22 next to the strays, whose
// places stay zero).  A block takes `px` pixels of Cp channels at a time, U times eight channels a thread, all of them in registers before the
// first is written.  Not made from the input again: what the input's memory holds may have changed since the planes were written.
// In the launch that transposes gradOutput: 256 images of 64 x 56 x 56, both passes 135 us (77 where nothing is to be brought back), 64 of 128 x 112 x 112 261 (146); through
// 4 to 14 KB of shared memory 201 and 384, in two launches through 24 KB 167 and 322.
template <int U>
struct UnpairPass {
  static constexpr int kPerSM = 1, kMost = 2048 * U;   // channels that a block can take
  unsigned blocks = 0;
  void *planes;
  long pixels;
  int Cp, px;
  Ranges ranges;
  RangeRec *kept;
  static UnpairPass of(void *planes, long pixels, int Cp, const Ranges &ranges, RangeRec *kept, long most) {
    const long px = std::max(1, kMost / Cp);
    return UnpairPass{(unsigned)std::min((pixels + px - 1) / px, most), planes, pixels, Cp, (int)px, ranges, kept};
  }
  __device__ __forceinline__ void run(unsigned block) const {
    if (!ranges.wide() || *const_cast<const volatile unsigned *>(&kept->wide)) return;
    const float unscale = pair_unscale(*kept);
    const int q = Cp / 8;
    int from[U], to[U];   // 16-byte pieces: of hi (lo is q further), of the values
#pragma unroll
    for (int k = 0; k < U; k++) {
      const int i = threadIdx.x + 256 * k, p = i / q, c = i - p * q;
      from[k] = 2 * p * q + c; to[k] = 2 * (p * q + c);
    }
    for (long p0 = (long)block * px; p0 < pixels; p0 += (long)blocks * px) {
      const int n = (int)min((long)px, pixels - p0) * q;
      uint4 *at = reinterpret_cast<uint4 *>(planes) + p0 * 2 * q;
      uint4 hi[U], lo[U];
#pragma unroll
      for (int k = 0; k < U; k++)
        if ((int)threadIdx.x + 256 * k < n) { hi[k] = at[from[k]]; lo[k] = at[from[k] + q]; }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < U; k++) {
        if ((int)threadIdx.x + 256 * k >= n) break;
        const __half *h = reinterpret_cast<const __half *>(&hi[k]), *l = reinterpret_cast<const __half *>(&lo[k]);
        float4 v[2];
        float *f = reinterpret_cast<float *>(v);
#pragma unroll
        for (int e = 0; e < 8; e++) f[e] = join_pair(h[e], l[e], unscale);
        reinterpret_cast<float4 *>(at)[to[k]] = v[0];
        reinterpret_cast<float4 *>(at)[to[k] + 1] = v[1];
      }
    }
    // every block has looked at the flag before the last one sets it
    if (threadIdx.x == 0 && atomicAdd(&kept->ticket, 1u) == blocks - 1) { kept->ticket = 0; kept->wide = 1; }
  }
};

// ---------------------------------------------------------------------------------------------
// Channels-last planes of an activation tensor, FP32 or BF16, channels padded with zeros to Cp = a multiple of KV.
//
// NCHW fp32 -> [img][pixel][Cp]; kPairs: [img][pixel][hi: Cp][lo: Cp], or FP32 values in the same place.  CT channels x PT pixels per pass through
// shared memory: reads coalesced along pixels, writes in whole 128-byte lines along channels.  Bound by latency: a thread has 16 or 32
// loads on the way before the barrier.  128 pixels a pass where they fill it (198 M values as pairs, 1.6 GB: 322 -> 277 us), 64 where
// planes would leave much of the wider tile empty (13 x 13: 92 us with 128, 83 with 64).
// SUMS: `chan_partial` is [blocks][C] sums over the pixels that a block transposed, per channel: the gradBias
// reduction of a convolution rides on the transposition of gradOutput instead of reading the tensor a second time.
// A channel of a tile belongs to one warp, tiles are taken in a fixed order, so the sums are reproducible.  Blocks that stay with one tile of
// channels and keep the sums in registers to the end save 15 % of the pass (a per cent of a step of 128 images), but another order of these
// sums is another training run: of small batches, one that ends in NaN where this one does not, or the other way round.
template <int PREC, int PT, bool SUMS>
struct PlanesPass {
  // (left alone, 128 registers with sums.  Six blocks for TF32 and for BF16's 64 pixels are faster from cold caches, 512 planes of 62 x 62, 30 images 95 -> 85 us in BF16, but not
  // behind the kernel that left the tensor in L2: a small TF32 block 68.6 -> 69.6, AlexNet's BF16 step 3350 -> 3366.)
  static constexpr int CT = PREC == kTf32 ? 32 : 64, kPerSM = PT == 128 ? 4 : 5;
  unsigned blocks = 0;
  const float *src;
  long N;
  int C, HW, Cp;
  void *dst;
  float *chan_partial;
  PairForm form;
  __device__ __forceinline__ void run(unsigned block) const {
    bool wide = false;
    float scale = 1.f;
    if constexpr (PREC == kPairs) {
      wide = form.ranges.wide();
      if (!wide) scale = pair_scale(*form.ranges.rec[0]);
    }
    __shared__ float tile[CT][PT + 1];
    extern __shared__ float4 pass_sm[];
    float *chan_sum = reinterpret_cast<float *>(pass_sm);   // [C] (SUMS)
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const unsigned ptiles = (unsigned)((HW + PT - 1) / PT), ctiles = (unsigned)(Cp / CT);
    const long ntiles = N * ptiles * ctiles;
    if constexpr (SUMS) {
      for (int c = threadIdx.x; c < C; c += blockDim.x) chan_sum[c] = 0.f;
      __syncthreads();
    }
    for (long t = block; t < ntiles; t += blocks) {
      const unsigned r = (unsigned)(t % (ptiles * ctiles));
      const long img = t / (ptiles * ctiles);
      const int ct = (int)(r / ptiles), p0 = (int)(r - ct * ptiles) * PT, c0 = ct * CT;
      const int np = min(HW - p0, PT), nc = min(C - c0, CT);
      const float *s = src + (img * C + c0) * HW + p0 + tx;
      float v[CT / 8][PT / 32];
#pragma unroll
      for (int j = 0; j < CT / 8; j++)
#pragma unroll
        for (int g = 0; g < PT / 32; g++)
          v[j][g] = (g * 32 + tx < np && ty + 8 * j < nc) ? s[(long)(ty + 8 * j) * HW + g * 32] : 0.f;
#pragma unroll
      for (int j = 0; j < CT / 8; j++) {
        float part = 0.f;
#pragma unroll
        for (int g = 0; g < PT / 32; g++) {
          tile[ty + 8 * j][g * 32 + tx] = v[j][g];
          if (SUMS) part += v[j][g];
        }
        if constexpr (SUMS) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
          if (tx == 0 && ty + 8 * j < nc) chan_sum[c0 + ty + 8 * j] += part;
        }
      }
      __syncthreads();
      const long o0 = (img * HW + p0) * Cp + c0;
#pragma unroll 8
      for (int j = ty; j < np; j += 8) {
        if constexpr (PREC == kBf16) {
          reinterpret_cast<__nv_bfloat162 *>(dst)[(o0 + (long)j * Cp) / 2 + tx] = __floats2bfloat162_rn(tile[2 * tx][j], tile[2 * tx + 1][j]);
        } else if constexpr (PREC == kPairs) {
          const float a = tile[2 * tx][j] * scale, b = tile[2 * tx + 1][j] * scale;
          float *px = reinterpret_cast<float *>(dst) + o0 - c0 + (long)j * Cp;
          if (wide) {
            reinterpret_cast<float2 *>(px + c0)[tx] = make_float2(a, b);
          } else {
            __half2 hi, lo;
            split_pair(a, b, hi, lo);
            __half2 *h = reinterpret_cast<__half2 *>(px) + c0 / 2 + tx;
            h[0] = hi;
            h[Cp / 2] = lo;
          }
        } else {
          reinterpret_cast<float *>(dst)[o0 + (long)j * Cp + tx] = tile[tx][j];
        }
      }
      __syncthreads();
    }
    if constexpr (SUMS)
      for (int c = threadIdx.x; c < C; c += blockDim.x) chan_partial[(long)block * C + c] = chan_sum[c];
    if constexpr (PREC == kPairs) form.end(wide, block);
  }
};
// out[c] += scale * sum_b partial[b][c], eight channels a block: 32 row slices per channel, folded in a fixed order.  The partials are a few
// MB at most; what this pass costs is the chain of dependent loads per thread, hence a sector of channels per block and
// sixteen loads in flight.
struct ChanFinishPass {
  static constexpr int kPerSM = 1;
  unsigned blocks = 0;
  const float *partial;
  int nblocks;
  long C;
  float *out, scale;
  __device__ __forceinline__ void run(unsigned block) const {
    __shared__ float sm[32][9];
    const int lane = threadIdx.x & 7, s = threadIdx.x >> 3;
    const long c = (long)block * 8 + lane;
    float a[8];
#pragma unroll
    for (int i = 0; i < 8; i++) a[i] = 0.f;
    if (c < C) {
      int b = s;
      for (; b + 15 * 32 < nblocks; b += 16 * 32) {
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = partial[(long)(b + 32 * i) * C + c];
#pragma unroll
        for (int i = 0; i < 16; i++) a[i & 7] += v[i];
      }
      if (b + 7 * 32 < nblocks) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = partial[(long)(b + 32 * i) * C + c];
#pragma unroll
        for (int i = 0; i < 8; i++) a[i] += v[i];
        b += 8 * 32;
      }
      float v[7];
#pragma unroll
      for (int i = 0; i < 7; i++) v[i] = b + 32 * i < nblocks ? partial[(long)(b + 32 * i) * C + c] : 0.f;
#pragma unroll
      for (int i = 0; i < 7; i++)
        if (b + 32 * i < nblocks) a[0] += v[i];
    }
    const float a0 = a[0] + a[4], a1 = a[1] + a[5], a2 = a[2] + a[6], a3 = a[3] + a[7];
    sm[s][lane] = (a0 + a1) + (a2 + a3);
    __syncthreads();
    if (s == 0 && c < C) {
      float acc = 0.f;
      for (int k = 0; k < 32; k++) acc += sm[k][lane];
      out[c] += scale * acc;
    }
  }
};

// A convolution layer restated over "cells": pixel (Y, X) of the restated input carries, as channels, the eH x eW input
// pixels at offsets (dy, dx) from (Y * dH - pad, X * dW - pad), all planes of each:
//   S[n][Y][X][ch = (dy * eW + dx) * Cq + c] = in[n][c][Y * dH + dy - pad][X * dW + dx - pad]
// and filter tap (i, j) is tap ((i - dy) / stepH, (j - dx) / stepW) at the channels of (dy, dx).  Per axis either
//   fold    e = min(d, k): the pixels of a stride cell become channels, ceil(k / d) taps remain, or
//   unfold  e = k: one tap remains (along both axes: the column matrix).
// `direct`: the input's own planes (e = 1, all taps, stride and padding left to the TMA window map).
// Which one costs least depends on how far the channel count is from a multiple of KV: see restate() in gpunn_conv.cu.
struct Cells {
  int C, kH, kW, dH, dW, pad;      // the layer
  int H, W;
  int eH, eW, kHs, kWs, stepH, stepW;
  int Cq;                          // channels per offset: C, or padded where that costs no further span
  int Cr, Cs;                      // eH * eW * Cq, and that padded to a multiple of KV
  int Hs, Ws;                      // grid of S
  bool direct;
  // place of channel `ch`; false: padding
  __host__ __device__ __forceinline__ bool channel(int ch, int &c, int &dy, int &dx) const {
    const int q = ch / Cq;
    c = ch - q * Cq;
    dy = q / eW;
    dx = q - dy * eW;
    return ch < Cr && c < C;
  }
};

// S of one image row per block.  A thread produces 16 bytes of a pixel: 4 FP32 or 8 BF16 channels, whose source offsets it
// looks up in a table; neighbouring threads hold neighbouring channels, i.e. neighbouring columns of a few input rows.  More
// channels than the table holds (kCellTable: 48 KB of it) are found by division, once per 16 bytes.
constexpr int kCellTable = 6144;
// kPairs: [pixel][hi: Cs][lo: Cs], 8 channels a thread.
template <int PREC, bool TABLE>
__device__ __forceinline__ void cells_row(const float *__restrict__ in, void *__restrict__ S, long row, const Cells &u, const int2 *chan_src, bool wide,
                                          float scale, unsigned part, unsigned parts) {
  constexpr int V = PREC != kTf32 ? 8 : 4;
  const long n = row / u.Hs;
  const int Y = (int)(row - n * u.Hs);
  const int q = u.Cs / V, chunks = u.Ws * q, y0 = Y * u.dH - u.pad;
  const float *img = in + n * u.C * (long)u.H * u.W;
  uint4 *dst = reinterpret_cast<uint4 *>(S) + ((n * u.Hs + Y) * u.Ws) * (long)q * (PREC == kPairs ? 2 : 1);
  for (int o = part * blockDim.x + threadIdx.x; o < chunks; o += parts * blockDim.x) {
    const int X = o / q, ch0 = (o - X * q) * V, x0 = X * u.dW - u.pad;
    float v[V];
    if constexpr (TABLE) {
      const float *base = img + (long)y0 * u.W + x0;
#pragma unroll
      for (int e = 0; e < V; e++) {
        const int2 s = chan_src[ch0 + e];
        const int y = y0 + (s.y >> 16), x = x0 + (s.y & 0xffff);
        v[e] = s.y >= 0 && (unsigned)y < (unsigned)u.H && (unsigned)x < (unsigned)u.W ? __ldg(base + s.x) : 0.f;
      }
    } else {
      int c, dy, dx;
      u.channel(ch0, c, dy, dx);
#pragma unroll
      for (int e = 0; e < V; e++) {
        const int y = y0 + dy, x = x0 + dx;
        v[e] = ch0 + e < u.Cr && c < u.C && (unsigned)y < (unsigned)u.H && (unsigned)x < (unsigned)u.W
                   ? __ldg(img + ((long)c * u.H + y) * u.W + x) : 0.f;
        if (++c == u.Cq) {
          c = 0;
          if (++dx == u.eW) { dx = 0; dy++; }
        }
      }
    }
    if constexpr (PREC == kBf16) {
      __nv_bfloat162 h[4];
#pragma unroll
      for (int e = 0; e < 4; e++) h[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
      dst[o] = *reinterpret_cast<const uint4 *>(h);
    } else if constexpr (PREC == kPairs) {
      if (wide) {
        float4 *d = reinterpret_cast<float4 *>(dst) + 2 * (long)o;
        d[0] = make_float4(v[0], v[1], v[2], v[3]);
        d[1] = make_float4(v[4], v[5], v[6], v[7]);
      } else {
        __half2 hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; e++) split_pair(v[2 * e] * scale, v[2 * e + 1] * scale, hi[e], lo[e]);
        uint4 *d = dst + X * 2l * q + ch0 / V;
        d[0] = *reinterpret_cast<const uint4 *>(hi);
        d[q] = *reinterpret_cast<const uint4 *>(lo);
      }
    } else {
      dst[o] = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
    }
  }
}
template <int PREC, bool TABLE>
struct CellsPass {
  // as many as the pass has by itself: with the registers of the weights' repacking an SM held five (16 images of 3 x 224 x 224 as 4 x 4 cells 11.3 -> 9.6 us)
  static constexpr int kPerSM = PREC == kTf32 ? 8 : PREC == kBf16 ? (TABLE ? 7 : 6) : TABLE ? 4 : 6;
  unsigned blocks = 0, rows;   // a row of cells is shared by blocks / rows blocks
  const float *in;
  void *S;
  Cells u;
  PairForm form;
  __device__ __forceinline__ void run(unsigned block) const {
    bool wide = false;
    float scale = 1.f;
    if constexpr (PREC == kPairs) {
      wide = form.ranges.wide();
      if (!wide) scale = pair_scale(*form.ranges.rec[0]);
    }
    extern __shared__ float4 pass_sm[];
    int2 *chan_src = reinterpret_cast<int2 *>(pass_sm);      // per channel: offset in the image, (dy << 16 | dx) or -1
    if constexpr (TABLE) {
      for (int ch = threadIdx.x; ch < u.Cs; ch += blockDim.x) {
        int c, dy, dx;
        chan_src[ch] = u.channel(ch, c, dy, dx) ? make_int2((c * u.H + dy) * u.W + dx, dy << 16 | dx) : make_int2(0, -1);
      }
      __syncthreads();
    }
    const unsigned part = block / rows;
    cells_row<PREC, TABLE>(in, S, block - part * rows, u, chan_src, wide, scale, part, blocks / rows);   // (a loop over rows costs 98 -> 117 us at 256 images)
    if constexpr (PREC == kPairs) form.end(wide, block);
  }
};

// The same where a row's input fits shared memory and each thread keeps the channels it writes (Cs / V divides the block): the
// C * eH input rows are read once, in order, with zeros around them, and every value leaves from there without a bounds check
// or a table look-up.  Bound by the latency of a row's reads and by its shared-memory reads (lines 16 banks apart, the least
// conflicts for cells of four columns); for long rows (see restate_input).  3 planes of 224 x 224 as 4 x 4 cells: 1024 images as pairs (1.47 GB) 493 -> 338 us,
// 256 images in FP32 78 -> 70.
template <int PREC>
struct StagedCellsPass {
  static constexpr int kPerSM = 4;   // 1024 images as pairs 341 us unbounded (76 registers), 329 so, 366 with five
  unsigned blocks = 0;
  const float *in;
  void *S;
  long N;
  Cells u;
  int Wp, ld;
  PairForm form;
  __device__ __forceinline__ void run(unsigned block) const {
    bool wide = false;
    float scale = 1.f;
    if constexpr (PREC == kPairs) {
      wide = form.ranges.wide();
      if (!wide) scale = pair_scale(*form.ranges.rec[0]);
    }
    constexpr int V = PREC == kPairs ? 8 : 4;
    extern __shared__ float4 pass_sm[];
    float *rows_in = reinterpret_cast<float *>(pass_sm);   // [C][eH][ld]
    const int lines = u.C * u.eH, q = u.Cs / V, ch0 = (int)(threadIdx.x % q) * V, lane = threadIdx.x & 31;
    int at[V];                           // this thread's channels within the window of column 0
#pragma unroll
    for (int e = 0; e < V; e++) {
      int c, dy, dx;
      at[e] = u.channel(ch0 + e, c, dy, dx) ? (c * u.eH + dy) * ld + dx : -1;
    }
    // a warp takes up to 128 columns of four lines at a time, all loads in flight before the first store; its first piece of the next
    // row is on the way while this row leaves
    const int warp = threadIdx.x >> 5, parts = (Wp + 127) / 128, pieces = (lines + 3) / 4 * parts;
    float piece[4][4];
    auto load = [&](long row, int g) {
      const long n = row / u.Hs;
      const int Y = (int)(row - n * u.Hs), y0 = Y * u.dH - u.pad, l0 = g / parts * 4, t0 = (g - g / parts * parts) * 128 + lane;
      const float *img = in + n * u.C * (long)u.H * u.W;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const int l = l0 + a, c = l / u.eH, y = y0 + l - c * u.eH;
        const bool inside = l < lines && (unsigned)y < (unsigned)u.H;
        const float *src = img + ((long)c * u.H + y) * u.W - u.pad;
#pragma unroll
        for (int b = 0; b < 4; b++) piece[a][b] = inside && (unsigned)(t0 + 32 * b - u.pad) < (unsigned)u.W ? __ldg(src + t0 + 32 * b) : 0.f;
      }
    };
    auto keep = [&](int g) {
      const int l0 = g / parts * 4, t0 = (g - g / parts * parts) * 128 + lane;
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
          if (l0 + a < lines && t0 + 32 * b < Wp) rows_in[(l0 + a) * ld + t0 + 32 * b] = piece[a][b];
    };
    const long rows = N * u.Hs;
    if (warp < pieces && block < rows) load(block, warp);
    for (long row = block; row < rows; row += blocks) {
      if (warp < pieces) keep(warp);
      for (int g = warp + 8; g < pieces; g += 8) { load(row, g); keep(g); }
      __syncthreads();
      if (warp < pieces && row + blocks < rows) load(row + blocks, warp);
      uint4 *dst = reinterpret_cast<uint4 *>(S) + row * u.Ws * (long)q * (PREC == kPairs ? 2 : 1);
      for (int X = (int)threadIdx.x / q; X < u.Ws; X += 256 / q) {
        float v[V];
#pragma unroll
        for (int e = 0; e < V; e++) v[e] = at[e] >= 0 ? rows_in[at[e] + X * u.dW] : 0.f;
        if (PREC == kPairs && !wide) {
          __half2 hi[4], lo[4];
#pragma unroll
          for (int e = 0; e < 4; e++) split_pair(v[(2 * e) % V] * scale, v[(2 * e + 1) % V] * scale, hi[e], lo[e]);
          uint4 *d = dst + X * 2l * q + ch0 / V;
          d[0] = *reinterpret_cast<const uint4 *>(hi);
          d[q] = *reinterpret_cast<const uint4 *>(lo);
        } else {
          float4 *d = reinterpret_cast<float4 *>(dst) + ((long)X * q + ch0 / V) * (V / 4);
#pragma unroll
          for (int e = 0; e < V; e += 4) d[e / 4] = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
        }
      }
      __syncthreads();
    }
    if constexpr (PREC == kPairs) form.end(wide, block);
  }
};

// The column matrix in BF16 with eight channels per tap (Cq = 8, C <= 8): 16 bytes of S are one tap of one pixel.  A block makes
// the rows of one output row: the kH input rows it needs go to shared memory once, as 16-byte pixels, and leave from there
// kH * kW times over, so that the kernel is bound by the writes (gathering each value from the image took four times as
// long: 1105 -> 280 us for 256 images under the 11 x 11 / 4 filter, 1.6 GB).
struct Columns8Pass {
  static constexpr int kPerSM = 1;
  unsigned blocks = 0;
  const float *in;
  uint4 *S;
  Cells u;
  __device__ __forceinline__ void run(unsigned block) const {
    extern __shared__ float4 pass_sm[];
    uint4 *px_rows = reinterpret_cast<uint4 *>(pass_sm);   // [kH][W + 2 pad]
    const long n = block / u.Hs;
    const int Y = (int)(block - n * u.Hs), Wp = u.W + 2 * u.pad, taps = u.kH * u.kW, q = u.Cs / 8;
    const float *img = in + n * u.C * (long)u.H * u.W;
    for (int t = threadIdx.x; t < u.kH * Wp; t += blockDim.x) {
      const int i = t / Wp, y = Y * u.dH + i - u.pad, x = t - i * Wp - u.pad;
      float v[8];
#pragma unroll
      for (int c = 0; c < 8; c++)
        v[c] = c < u.C && (unsigned)y < (unsigned)u.H && (unsigned)x < (unsigned)u.W ? __ldg(img + ((long)c * u.H + y) * u.W + x) : 0.f;
      __nv_bfloat162 h[4];
#pragma unroll
      for (int e = 0; e < 4; e++) h[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
      px_rows[t] = *reinterpret_cast<const uint4 *>(h);
    }
    __syncthreads();
    uint4 *dst = S + (n * u.Hs + Y) * u.Ws * (long)q;
    const int chunks = u.Ws * q, step_x = (int)blockDim.x / q, step_t = (int)blockDim.x - step_x * q;
    int X = (int)threadIdx.x / q, tap = (int)threadIdx.x - X * q;
    for (int o = threadIdx.x; o < chunks; o += blockDim.x) {
      const int i = tap / u.kW, j = tap - i * u.kW;
      dst[o] = tap < taps ? px_rows[i * Wp + X * u.dW + j] : make_uint4(0, 0, 0, 0);
      X += step_x; tap += step_t;
      if (tap >= q) { tap -= q; X++; }
    }
  }
};

// An image of eight-plane BF16 pixels (planes past C and pixels around the input are zeros) that the windows of a layer cover:
// [n][rows][pitch], row (y, x) is input pixel (y - pad, x - pad).  See GatheredWindowOperand.  Bound by its writes.
struct Pixels8Pass {
  static constexpr int kPerSM = 1;
  unsigned blocks = 0;
  const float *in;
  uint4 *out;
  long N;
  int C, H, W, pad, rows, pitch;
  __device__ __forceinline__ void run(unsigned block) const {
    const long lines = N * rows;
    // a warp takes up to 128 pixels of a line, all loads on the way before the first store
    const int lane = threadIdx.x & 31, parts = (pitch + 127) / 128;
    for (long l = (long)block * 8 + (threadIdx.x >> 5); l < lines * parts; l += (long)blocks * 8) {
      const long line = l / parts, n = line / rows;
      const int x0 = (int)(l - line * parts) * 128 + lane, y = (int)(line - n * rows) - pad;
      const float *src = in + (n * C * H + y) * (long)W - pad;
      float v[4][8];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int c = 0; c < 8; c++)
          v[a][c] = c < C && (unsigned)y < (unsigned)H && (unsigned)(x0 + 32 * a - pad) < (unsigned)W ? __ldg(src + (long)c * H * W + x0 + 32 * a) : 0.f;
#pragma unroll
      for (int a = 0; a < 4; a++) {
        __nv_bfloat162 h[4];
#pragma unroll
        for (int e = 0; e < 4; e++) h[e] = __floats2bfloat162_rn(v[a][2 * e], v[a][2 * e + 1]);
        if (x0 + 32 * a < pitch) out[line * pitch + x0 + 32 * a] = *reinterpret_cast<const uint4 *>(h);
      }
    }
  }
};

// Weights of the restated layer in the k order of the window operand, four values per thread:
//   FLIP false: out[ko][(bi, bj, ch)]           (forward)
//   FLIP true : out[ch][(bi', bj', ko)], bi' = kHs - 1 - bi: gradInput as a forward pass over gradOutput (channels padded to
//               `chans`) under the filter rotated by 180 degrees
// pair_shift > 0 (pixel-pair mode, see Epilogue): the filter is widened to kWs + pair_shift columns and
// stored twice, rows [0, rows) as it is (output parity 0) and rows [rows, 2 rows) shifted right by pair_shift
// columns (parity 1, whose window starts one stride later); the new columns are zero.
// kPairs: a row is [hi: its values][lo: its values].
template <int PREC, bool FLIP>
struct RepackPass {
  unsigned blocks = 0;
  const float *w;
  Cells u;
  int K, rows, chans, pair_shift;
  void *out;
  Ranges ranges;
  __device__ __forceinline__ void run(unsigned block) const {
    bool wide = false;
    float scale = 1.f;
    if constexpr (PREC == kPairs) {
      wide = ranges.wide();
      if (!wide) scale = pair_scale(*ranges.rec[0]);
    }
    const int kWe = u.kWs + pair_shift, quads = u.kHs * kWe * (chans / 4);
    const unsigned total = (unsigned)((pair_shift ? 2 : 1) * rows) * (unsigned)quads;
    for (unsigned t = block * blockDim.x + threadIdx.x; t < total; t += blocks * blockDim.x) {
      int r = (int)(t / (unsigned)quads);
      const long row = r;
      const int k = (int)(t - (unsigned)r * quads) * 4, tap = k / chans, k0 = k - tap * chans;
      const int par = r >= rows ? 1 : 0;
      r -= par * rows;
      int bi = tap / kWe, bj = tap - bi * kWe - par * pair_shift;
      if (FLIP) { bi = u.kHs - 1 - bi; bj = u.kWs - 1 - bj; }
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int ch = FLIP ? r : k0 + e, ko = FLIP ? k0 + e : r;
        int c, dy, dx;
        const bool real = u.channel(ch, c, dy, dx);
        const int i = dy + bi * u.stepH, j = dx + bj * u.stepW;
        v[e] = real && ko < K && bj >= 0 && bj < u.kWs && i < u.kH && j < u.kW ? __ldg(w + ((((long)ko * u.C + c) * u.kH + i) * u.kW + j)) : 0.f;
      }
      if (PREC == kPairs && !wide) {
        __half2 hi[2], lo[2];
        split_pair(v[0] * scale, v[1] * scale, hi[0], lo[0]);
        split_pair(v[2] * scale, v[3] * scale, hi[1], lo[1]);
        uint2 *o = reinterpret_cast<uint2 *>(out) + row * 2 * quads + k / 4;
        o[0] = make_uint2(half2_bits(hi[0]), half2_bits(hi[1]));
        o[quads] = make_uint2(half2_bits(lo[0]), half2_bits(lo[1]));
      } else if constexpr (PREC == kBf16) {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
        reinterpret_cast<uint2 *>(out)[t] = make_uint2(*reinterpret_cast<const unsigned *>(&a), *reinterpret_cast<const unsigned *>(&b));
      } else {
        reinterpret_cast<float4 *>(out)[t] = make_float4(v[0], v[1], v[2], v[3]);
      }
    }
  }
};

template <int PREC, bool FLIP>
static __global__ void __launch_bounds__(256) repack_weight_kernel(const float *__restrict__ w, const Cells u, int K, int rows, int chans, int pair_shift,
                                                                   void *__restrict__ out, const Ranges ranges) {
  pdl_begin();
  RepackPass<PREC, FLIP>{gridDim.x, w, u, K, rows, chans, pair_shift, out, ranges}.run(blockIdx.x);
}

// gw[ko][(c, i, j)] += scale * T at the restated tap and channel of (c, i, j).  ko_stride, ch_stride, bi_stride, bj_stride: where T
// keeps them (bj counted from the other end when bj_stride is negative: `first` is then the place of tap (0, 0)).
// `copies` partial sums of each, copy_stride apart.
struct WgradPlace { long ko_stride, ch_stride, bi_stride, bj_stride, first; int copies; long copy_stride; };
// The product that the strays of its operands are added to: a layer over N images, [N][C][H][W] -> [N][K][oH][oW].
struct LayerShape { long N; int C, H, W, K, oH, oW, kH, kW, dH, dW, pad; };
struct WgradStrays {
  Measured act, gout;
  Ranges ranges;
  long n0;              // image of act's record and list that the planes start with
  const void *planes;   // of the input (pairs, where gout has strays)
  const float *go;
  LayerShape l;
};
// One value of restated planes in pairs: input pixel (y, x) of plane c, which some window covers.
__device__ __forceinline__ float plane_value(const void *planes, const Cells &u, long n, int c, int y, int x, float unscale) {
  int ch = c;
  if (!u.direct) {
    y += u.pad; x += u.pad;
    const int Y = min(y / u.dH, u.Hs - 1), X = min(x / u.dW, u.Ws - 1);
    ch += ((y - Y * u.dH) * u.eW + x - X * u.dW) * u.Cq;
    y = Y; x = X;
  }
  const __half *p = reinterpret_cast<const __half *>(planes) + ((n * u.Hs + y) * u.Ws + x) * 2 * u.Cs + ch;
  return join_pair(p[0], p[u.Cs], unscale);
}
struct StrayPlaces { int n[kStrays], c[kStrays], y[kStrays], x[kStrays]; float v[kStrays]; };
__device__ __forceinline__ void find_strays(StrayPlaces &s, const Stray *list, int count, int C, int H, int W, long n0) {
  for (int i = threadIdx.x; i < count; i += blockDim.x) {
    const long at = list[i].at, row = at / W, plane = row / H;
    s.x[i] = (int)(at - row * W); s.y[i] = (int)(row - plane * H);
    s.n[i] = (int)(plane / C - n0); s.c[i] = (int)(plane % C);
    s.v[i] = list[i].v;
  }
}
struct WgradDivs {
  FastDiv per, kHW, kW, stepH, stepW;
  static WgradDivs of(const Cells &u) {
    const long kHW = (long)u.kH * u.kW;
    return WgradDivs{FastDiv::make(u.C * kHW), FastDiv::make(kHW), FastDiv::make(u.kW), FastDiv::make(u.stepH), FastDiv::make(u.stepW)};
  }
};
// kPairs: with the strays of the input against all of gradOutput, and those of gradOutput against what the planes hold of the input.
// ALONE: not next to the fold of gradBias.  Bound by its instructions and by how many blocks an SM holds: 9.4 M weights took 80 us with the
// fold's 56 registers and five divisions in hardware a weight, 57 with these by multiplication, 33 with 32 registers as well.
template <bool PAIRS, bool ALONE>
struct UnpackGradPass {
  static constexpr int kPerSM = ALONE ? 8 : 4;
  unsigned blocks = 0;
  const float *T;
  float *gw;
  Cells u;
  int K;
  WgradDivs div;
  WgradPlace p;
  float scale;
  WgradStrays q;
  __device__ __forceinline__ void run(unsigned block) const {
    __shared__ StrayPlaces sa, sg;   // (kPairs)
    int na = 0, ng = 0;
    float unscale = 1.f;
    const LayerShape &l = q.l;
    if constexpr (PAIRS) {
      const bool wide = q.ranges.wide();
      na = q.act.strays(wide); ng = q.gout.strays(wide);
      if (na) find_strays(sa, q.act.list, na, l.C, l.H, l.W, q.n0);
      if (ng) { find_strays(sg, q.gout.list, ng, l.K, l.oH, l.oW, 0); unscale = pair_unscale(*q.act.rec); }
      __syncthreads();
    }
    const unsigned total = (unsigned)K * div.per.d;
    for (unsigned t = block * blockDim.x + threadIdx.x; t < total; t += blocks * blockDim.x) {
      unsigned ko, r, c, tap, i, j, bi = 0, dy, bj = 0, dx;
      div.per.divmod(t, ko, r);
      div.kHW.divmod(r, c, tap);
      div.kW.divmod(tap, i, j);
      dy = i; dx = j;
      if (u.kHs > 1) div.stepH.divmod(i, bi, dy);
      if (u.kWs > 1) div.stepW.divmod(j, bj, dx);
      const long ch = (int)(dy * u.eW + dx) * u.Cq + (int)c;
      const float *s = T + (p.first + ko * p.ko_stride + ch * p.ch_stride + (int)bi * p.bi_stride + (int)bj * p.bj_stride);
      float sum = *s;
      for (int b = 1; b < p.copies; b++) sum += s[b * p.copy_stride];
      if constexpr (PAIRS) {
        for (int e = 0; e < na; e++) {
          const StrayPlaces &f = sa;
          if (f.c[e] != (int)c || f.n[e] < 0 || f.n[e] >= l.N) continue;
          const int ty = f.y[e] + l.pad - (int)i, tx = f.x[e] + l.pad - (int)j, oy = ty / l.dH, ox = tx / l.dW;
          if (ty < 0 || tx < 0 || oy * l.dH != ty || ox * l.dW != tx || oy >= l.oH || ox >= l.oW) continue;
          sum += f.v[e] * q.go[(((long)f.n[e] * l.K + ko) * l.oH + oy) * l.oW + ox];
        }
        for (int e = 0; e < ng; e++) {
          const StrayPlaces &f = sg;
          if (f.c[e] != (int)ko) continue;
          const int y = f.y[e] * l.dH + (int)i - l.pad, x = f.x[e] * l.dW + (int)j - l.pad;
          if ((unsigned)y < (unsigned)l.H && (unsigned)x < (unsigned)l.W) sum += f.v[e] * plane_value(q.planes, u, f.n[e], (int)c, y, x, unscale);
        }
      }
      gw[t] += scale * sum;
    }
  }
};

// gin[n][c][h][w] = gS[n][ch][Y][X], the inverse of a fold along both axes (a bijection between the input pixels that any
// window reaches and the cells' channels; the others get zero).  gS: [N][Cr][Hs][Ws].
// Blocks take groups of G planes pixel by pixel, whatever the planes' shape, four loads of a thread on the way, divisions by multiplication.
// From cold caches (us; pixel by pixel with divisions in hardware / a warp per line / so): 16 images of 3 x 224 x 224 14.4 / 11.7 / 11.8; 512 of 512 x
// 7 x 7 233 / 376 / 49; 256 of 256 x 14 x 14 92 / 186 / 48; one of 3 x 2048 x 2048 164 / 46 / 43, of 4 x 262144 51 / 2666 / 6.6.
struct UnfoldGeom {
  long planes;
  int G;
  FastDiv HW, C, W, dH, dW;
};
static __global__ void __launch_bounds__(256) unfold_grad_input_kernel(const float *__restrict__ gS, float *__restrict__ gin, const Cells u,
                                                                       const UnfoldGeom q) {
  pdl_begin();
  const unsigned HW = q.HW.d;
  const long step = (long)u.Hs * u.Ws;
  for (long p0 = (long)blockIdx.y * q.G; p0 < q.planes; p0 += (long)gridDim.y * q.G) {
    const long n0 = p0 / u.C;
    const unsigned c0 = (unsigned)(p0 - n0 * u.C), pixels = (unsigned)min((long)q.G, q.planes - p0) * HW;
    for (unsigned t0 = blockIdx.x * 1024 + threadIdx.x; t0 < pixels; t0 += gridDim.x * 1024) {
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        unsigned pl, r, n, c, y, x, Y, dy, X, dx;
        q.HW.divmod(t0 + 256 * k, pl, r);
        q.C.divmod(c0 + pl, n, c);
        q.W.divmod(r, y, x);
        q.dH.divmod(y + u.pad, Y, dy);
        q.dW.divmod(x + u.pad, X, dx);
        const bool reached = t0 + 256 * k < pixels && (int)Y < u.Hs && (int)X < u.Ws && (int)dy < u.eH && (int)dx < u.eW;
        v[k] = reached ? __ldg(gS + ((n0 + n) * u.Cr + (long)(dy * u.eW + dx) * u.Cq + c) * step + (long)Y * u.Ws + X) : 0.f;
      }
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (t0 + 256 * k < pixels) gin[p0 * HW + t0 + 256 * k] = v[k];
    }
  }
}

// Up to two matrices (blockIdx.y) as FP16 pairs: lines of `run` values become [hi: ldp][lo: ldp], ldp = run padded with zeros to whole
// spans, or lines of ldp FP32 values.  A warp takes 512 values of a line, all loads in flight before the first store.
struct PairJob { const float *src; void *dst; long lines, run, ld, ldp; int vec; Ranges ranges; };
static __global__ void __launch_bounds__(256) split_matrix_kernel(const PairJob a, const PairJob b) {
  pdl_begin();
  const PairJob &j = blockIdx.y ? b : a;
  const bool wide = j.ranges.wide();
  const float scale = wide ? 1.f : pair_scale(*j.ranges.rec[0]);
  const int lane = threadIdx.x & 31;
  const long warps = (long)gridDim.x * 8, parts = (j.ldp + 511) / 512;
  for (long w = (long)blockIdx.x * 8 + (threadIdx.x >> 5); w < j.lines * parts; w += warps) {
    const long l = w / parts, c0 = (w - l * parts) * 512 + lane * 4;
    const float *s = j.src + l * j.ld;
    float4 v[4];
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const long c = c0 + g * 128;
      if (j.vec && c + 4 <= j.run) v[g] = __ldg(reinterpret_cast<const float4 *>(s + c));
      else v[g] = make_float4(c < j.run ? s[c] : 0.f, c + 1 < j.run ? s[c + 1] : 0.f, c + 2 < j.run ? s[c + 2] : 0.f, c + 3 < j.run ? s[c + 3] : 0.f);
    }
    float *d = reinterpret_cast<float *>(j.dst) + l * j.ldp;
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const long c = c0 + g * 128;
      if (c >= j.ldp) break;
      if (wide) {
        *reinterpret_cast<float4 *>(d + c) = v[g];
      } else {
        __half2 hi[2], lo[2];
        split_pair(v[g].x * scale, v[g].y * scale, hi[0], lo[0]);
        split_pair(v[g].z * scale, v[g].w * scale, hi[1], lo[1]);
        uint2 *h = reinterpret_cast<uint2 *>(reinterpret_cast<__half *>(d) + c);
        h[0] = make_uint2(half2_bits(hi[0]), half2_bits(hi[1]));
        h[j.ldp / 4] = make_uint2(half2_bits(lo[0]), half2_bits(lo[1]));
      }
    }
  }
}

// BF16 plane of a strided matrix: element (r, k) at src[r*rs + k*ks]; out [rows][ld], zero for k >= K (ld a multiple of 64).
// 64 x 64 tiles: along k as they lie, else through shared memory.
static __global__ void __launch_bounds__(256) bf16_rows_kernel(const float *__restrict__ src, long rs, long ks, long rows, long K,
                                                               __nv_bfloat16 *__restrict__ out, long ld) {
  pdl_begin();
  __shared__ float tile[64][65];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long tiles_k = ld / 64;
  const long ntiles = ((rows + 63) / 64) * tiles_k;
  for (long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const long r0 = (t / tiles_k) * 64, k0 = (t % tiles_k) * 64;
    if (rs == 1 && ks != 1) {   // memory runs along the rows: warp = k, lanes = rows
      float v[8][2];
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const long r = r0 + tx + 32 * h, k = k0 + ty + 8 * j;
          v[j][h] = (r < rows && k < K) ? src[r + k * ks] : 0.f;
        }
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) tile[tx + 32 * h][ty + 8 * j] = v[j][h];
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const long r = r0 + ty + 8 * j;
        if (r < rows)
          *reinterpret_cast<__nv_bfloat162 *>(out + r * ld + k0 + 2 * tx) = __floats2bfloat162_rn(tile[ty + 8 * j][2 * tx], tile[ty + 8 * j][2 * tx + 1]);
      }
      __syncthreads();
    } else {
      float v[8][2];
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const long r = r0 + ty + 8 * j, k = k0 + 2 * tx + h;
          v[j][h] = (r < rows && k < K) ? src[r * rs + k * ks] : 0.f;
        }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const long r = r0 + ty + 8 * j;
        if (r < rows) *reinterpret_cast<__nv_bfloat162 *>(out + r * ld + k0 + 2 * tx) = __floats2bfloat162_rn(v[j][0], v[j][1]);
      }
    }
  }
}

// Folds split-K partials (fixed order -> deterministic) and applies the epilogue.  grid.y walks n, threads walk
// m, which is contiguous in the workspace.
static __global__ void __launch_bounds__(256) splitk_finish_kernel(const float *__restrict__ ws, int splits, long M, long N,
                                                            Epilogue epi) {
  pdl_begin();
  const long m = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  const bool pair = epi.pair_K != 0;
  const long mo = pair ? epi.moff<true>(m) : epi.moff<false>(m);
  const float row_b = epi.rb(m);
  for (long n = blockIdx.y; n < N; n += gridDim.y) {
    float acc = 0.f;
    for (int z = 0; z < splits; z++) acc += ws[((long)z * N + n) * M + m];
    if (pair) epi.store<true>(mo, n, acc);
    else epi.store<false>(mo, n, acc, row_b);
  }
}

// The same for the tile-local partials of the two-SM engine (Problem::tail_first): block (t, y) folds columns COLS * y .. + COLS - 1, COLS *
// (y + gridDim.y), ... of tail tile t; a thread owns one of the tile's 256 rows, which are contiguous in the workspace.  Bound by
// latency: four columns at once where that leaves blocks enough (8 -> 5 us for a round of tiles in two to four slices), one where
// few tiles are cut into many slices (a tile in 70: 11.5 us, 18 with four).
template <int COLS>
static __global__ void __launch_bounds__(256) tail_finish_kernel(const float *__restrict__ ws, int splits, int bn2, long tail_first,
                                                          long gm, long M, long N, Epilogue epi) {
  pdl_begin();
  const long tile = tail_first + blockIdx.x;
  const long nt = Epilogue::quotient(tile, gm), mt = tile - nt * gm;
  const long m = mt * 256 + threadIdx.x;
  if (m >= M) return;
  const bool pair = epi.pair_K != 0;
  const long mo = pair ? epi.moff<true>(m) : epi.moff<false>(m);
  const float row_b = epi.rb(m);
  const float *base = ws + (long)blockIdx.x * splits * bn2 * 256 + threadIdx.x;
  for (int c = COLS * blockIdx.y; c < bn2; c += COLS * gridDim.y) {
    const long n = nt * bn2 + c;
    if (n >= N) break;
    float acc[COLS];
#pragma unroll
    for (int j = 0; j < COLS; j++) acc[j] = 0.f;
#pragma unroll (COLS == 1 ? 8 : 4)
    for (int z = 0; z < splits; z++)
#pragma unroll
      for (int j = 0; j < COLS; j++) acc[j] += base[((long)z * bn2 + c + j) * 256];
    if constexpr (COLS == 4) {
      float *o = epi.out + mo + n;
      if (!pair && epi.nstride == 1 && n + 3 < N && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {   // the columns are neighbours in memory
        float4 old = make_float4(0.f, 0.f, 0.f, 0.f);
        if (epi.beta != 0.f) old = *reinterpret_cast<const float4 *>(o);
        const float4 v = make_float4(epi.value(n, acc[0], row_b, old.x), epi.value(n + 1, acc[1], row_b, old.y), epi.value(n + 2, acc[2], row_b, old.z),
                                     epi.value(n + 3, acc[3], row_b, old.w));
        *reinterpret_cast<float4 *>(o) = v;
        continue;
      }
    }
#pragma unroll
    for (int j = 0; j < COLS; j++) {
      if (n + j >= N) break;
      if (pair) epi.store<true>(mo, n + j, acc[j]);
      else epi.store<false>(mo, n + j, acc[j], row_b);
    }
  }
}

}  // namespace mm
}  // namespace thc

#endif
