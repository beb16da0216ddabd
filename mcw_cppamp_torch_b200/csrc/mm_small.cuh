// Products that are too small or too narrow for the two-SM tcgen05 tiles: FP32-accurate through warp-level TF32 MMAs.
//
// A 256 x 64 tile of the raw-operand engine needs its cluster, tensor memory, tensor maps and a deep ring before the
// first result, about 10 us however little there is to do, and it cannot fetch operands whose pitch is no multiple
// of 16 bytes.  What runs here is bound by latency (a few tiles) or by one operand's bytes (a weight matrix against a
// handful of rows), not by the tensor pipe, so the wide tile buys nothing: one launch reads the FP32 operands as
// they lie (either may run along k or along its rows, any pitch, any alignment), splits them into TF32 hi and lo
// parts in registers and multiplies with mma.sync.
//
//   block   128 threads, a BM x BN tile of D over one k slice; 32-k stages through a ring of cp.async copies
//           (16 bytes where the operand allows it, else 4)
//   split   hi = tf32(x), lo = tf32(x - hi); hi*hi goes into one accumulator and the
//           two cross products into another, both started afresh every 32 k and added into FP32 registers with
//           round-to-nearest (the tensor core truncates when it accumulates; chains here are 4 and 8 long)
//   slices  k is cut until the tiles fill the device; partial sums go to the workspace and the block that finishes
//           last on a tile (ticket) adds them in slice order and applies the epilogue, in the same launch
#ifndef THC_MM_SMALL_CUH
#define THC_MM_SMALL_CUH

#include <type_traits>

#include "mm_tc.cuh"

namespace thc {
namespace mm {

// Matrix with element (r, k) at base[r * ld + k] (along_k) or base[k * ld + r].
struct SmallOperand {
  const float *base;
  long ld;
  int vec4;   // base 16-byte aligned and ld a multiple of 4
};
struct SmallProblem {
  SmallOperand a, b;
  int M, N, K;
  float *c;                  // D(m, n) at c[m * sm + n * sn]
  long sm, sn;
  float alpha, beta;
  const float *bias;         // added at bias[m * bias_m + n * bias_n]; may be null
  int bias_m, bias_n;
  int slices, tiles_per_slice;   // k slices and 32-k tiles in each
  float *ws;                 // [tile][slice][value][thread] partial sums
  unsigned *tickets;         // one zero word per tile
  const int *stalled;        // the stream's stall flag (StallCtl::dev_flag): behind a stalled kernel nothing is written
};

constexpr int SM_THREADS = 128;
constexpr int SM_STAGES = 4;
// A 32-k tile of ROWS rows in shared memory.  Which row or k a fragment register stands for is free as long as both
// operands (k) and the epilogue (rows) agree, so the assignment is the one that lets a thread read its fragments with
// the widest accesses:
//   along k : [row][32 k], 16-byte chunk index XOR 4 on odd rows (the two rows of a quarter-warp access then fall into
//             different halves of the banks).  One 16-byte read per row gives k = 4t .. 4t + 3 of a 16-k group: the slots
//             (t, t + 4) of two consecutive 8-k MMAs.
//   along rows : [k][ROWS + 8].  One read of two to four neighbouring rows at each of k = 4t .. 4t + 3.
template <int ROWS, bool ALONG_K> struct SmallTile {
  static constexpr int PITCH = ALONG_K ? TC_BK : ROWS + 8;
  static constexpr int FLOATS = ALONG_K ? ROWS * PITCH : TC_BK * PITCH;
  static constexpr int RUN = ALONG_K ? TC_BK : ROWS, LINES = ALONG_K ? ROWS : TC_BK;   // a line of the tile runs along memory
  static __device__ __forceinline__ int at(int line, int c) {
    // lines of an along-rows tile lie transposed within groups of 16, so that k = q, 4 + q, 8 + q, 12 + q are neighbours
    const int l = ALONG_K ? line : (line & 16) | ((line & 3) << 2) | ((line >> 2) & 3);
    return l * PITCH + (ALONG_K ? c ^ ((line & 1) << 4) : c);
  }
};

__device__ __forceinline__ void cp_async16_part(uint32_t dst, const float *src, int bytes) {
  asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"((const void *)src), "r"(bytes) : "memory");
}
// One thread's share of the copies of an operand's tiles.  What lies beyond the matrix arrives as zeros.
template <int ROWS, bool ALONG_K>
struct SmallFetch {
  typedef SmallTile<ROWS, ALONG_K> Tile;
  static constexpr int CHUNKS = Tile::RUN / 4, TOTAL = CHUNKS * Tile::LINES, N = (TOTAL + SM_THREADS - 1) / SM_THREADS;
  static constexpr int STEP = SM_THREADS / CHUNKS;      // lines between a thread's chunks (SM_THREADS % CHUNKS == 0)
  static_assert(SM_THREADS % CHUNKS == 0, "thread mapping");
  const float *src;   // this thread's first chunk of the next tile
  int line, c;        // its place in the tile
  long line_step, tile_step;
  __device__ __forceinline__ void init(const SmallOperand &o, int r0, int k0) {
    line = (int)threadIdx.x / CHUNKS; c = (int)threadIdx.x % CHUNKS * 4;
    src = o.base + (long)((ALONG_K ? r0 : k0) + line) * o.ld + (ALONG_K ? k0 : r0) + c;
    line_step = (long)STEP * o.ld;
    tile_step = ALONG_K ? TC_BK : (long)TC_BK * o.ld;
  }
  __device__ __forceinline__ void issue(const SmallOperand &o, int rows, int K, int r0, int k0, uint32_t dst) {
    const int lines = (ALONG_K ? rows - r0 : K - k0) - line, run = (ALONG_K ? K - k0 : rows - r0) - c;   // what is left of both
    const float *s = src;
    if (o.vec4) {
      const int bytes = run >= 4 ? 16 : run > 0 ? 4 * run : 0;
#pragma unroll
      for (int i = 0; i < N; i++) {
        if (TOTAL % SM_THREADS == 0 || line + i * STEP < Tile::LINES) {
          const int n = i * STEP < lines ? bytes : 0;
          cp_async16_part(dst + (uint32_t)Tile::at(line + i * STEP, c) * 4, n ? s : o.base, n);
        }
        s += line_step;
      }
    } else {
#pragma unroll
      for (int i = 0; i < N; i++) {
        if (TOTAL % SM_THREADS == 0 || line + i * STEP < Tile::LINES) {
#pragma unroll
          for (int e = 0; e < 4; e++)
            cp_async4(dst + (uint32_t)Tile::at(line + i * STEP, c + e) * 4, i * STEP < lines && e < run ? s + e : nullptr, o.base);
        }
        s += line_step;
      }
    }
    src += tile_step;
  }
};
template <int VEC> __device__ __forceinline__ void lds_vec(const float *p, float (&v)[VEC]) {
  if constexpr (VEC == 4) { const float4 q = *reinterpret_cast<const float4 *>(p); v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w; }
  else if constexpr (VEC == 2) { const float2 q = *reinterpret_cast<const float2 *>(p); v[0] = q.x; v[1] = q.y; }
  else v[0] = *p;
}
// d += a * b, or d = a * b
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2], bool fresh = false) {
  if (fresh) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
    return;
  }
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// hi = tf32(x) rounded to nearest in integer arithmetic, lo = x - hi scaled by 1 + 2^-12, of which the tensor core drops the
// low 13 bits (within 3/4 of a unit of the nearest): the conversion instruction shares a pipe that takes a quarter of
// the ALU's rate and was what bounded this kernel (4096 x 1 x 9216: 45 us with it, 37 without).
// A value next to the largest rounds to infinity, and lo to its opposite; an infinite one or a NaN has a NaN in lo.  All of
// them leave a NaN in every sum they reach, whatever the other operand: fp32_sum().
__device__ __forceinline__ void split_tf32(float x, uint32_t &hi, uint32_t &lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  const float d = x - __uint_as_float(hi);
  lo = __float_as_uint(fmaf(d, 0x1p-12f, d));
}

// The sum over [k0, k1) in plain FP32, for one that came out as NaN: values near the largest and infinities then give what FP32
// arithmetic gives.  (Keeping hi finite by a clamp in split_tf32 costs 2 - 14 % of the whole kernel, 4096 x 16 x 4096 27.0 -> 30.7
// us; a second pass over the tiles with the clamp costs the 64 x 64 tile its registers.)
template <bool A_K, bool B_K>
__device__ __forceinline__ float fp32_sum(const SmallProblem &p, long m, long n, int k0, int k1) {
  const float *a = p.a.base + (A_K ? m * p.a.ld + k0 : m + k0 * p.a.ld), *b = p.b.base + (B_K ? n * p.b.ld + k0 : n + k0 * p.b.ld);
  float sum = 0.f;
#pragma unroll 1
  for (int k = k0; k < k1; k++, a += A_K ? 1 : p.a.ld, b += B_K ? 1 : p.b.ld) sum = fmaf(*a, *b, sum);
  return sum;
}

// WM x WN warps, each (BM / WM) x (BN / WN)
template <int BM, int BN, int WM, int WN, bool A_K, bool B_K>
__global__ void __launch_bounds__(SM_THREADS) small_kernel(const SmallProblem p) {
  pdl_begin();
  static_assert(WM * WN * 32 == SM_THREADS && BM % (16 * WM) == 0 && BN % (8 * WN) == 0, "warp layout");
  constexpr int MT = BM / WM / 16, NT = BN / WN / 8;
  constexpr int A_FLOATS = SmallTile<BM, A_K>::FLOATS, B_FLOATS = SmallTile<BN, B_K>::FLOATS, STAGE = A_FLOATS + B_FLOATS;
  extern __shared__ float small_smem[];
  __shared__ bool is_last;
  const int stalled = *reinterpret_cast<const volatile int *>(p.stalled);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int wm = (warp % WM) * (BM / WM), wn = (warp / WM) * (BN / WN);
  const int kt0 = blockIdx.z * p.tiles_per_slice;
  const int nk = min(p.tiles_per_slice, (p.K + TC_BK - 1) / TC_BK - kt0);
  // the rows a thread's fragment registers stand for: fragment row r = 16 i + g + 8 e (A) or 8 j + g (B) of a warp's share
  // is this row of it
  auto a_row = [&](int i, int gr, int e) { return wm + (A_K ? 16 * i + gr + 8 * e : gr * 2 * MT + 2 * i + e); };
  auto b_row = [&](int j, int gr) { return wn + (B_K ? 8 * j + gr : gr * NT + j); };
  SmallFetch<BM, A_K> fa;
  SmallFetch<BN, B_K> fb;
  fa.init(p.a, m0, kt0 * TC_BK);
  fb.init(p.b, n0, kt0 * TC_BK);
  auto fetch = [&](int it) {
    if (it < nk) {
      const uint32_t st = smem_u32(small_smem + (it % SM_STAGES) * STAGE);
      fa.issue(p.a, p.M, p.K, m0, (kt0 + it) * TC_BK, st);
      fb.issue(p.b, p.N, p.K, n0, (kt0 + it) * TC_BK, st + A_FLOATS * 4);
    }
    cp_async_commit();
  };
  float acc[MT][NT][4];
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[i][j][e] = 0.f;
#pragma unroll
  for (int it = 0; it < SM_STAGES - 1; it++) fetch(it);
  for (int it = 0; it < nk; it++) {
    cp_async_wait<SM_STAGES - 2>();
    __syncthreads();             // tile `it` is there for everybody, and everybody has left tile it - 1
    fetch(it + SM_STAGES - 1);   // into the stage of tile it - 1
    const float *as = small_smem + (it % SM_STAGES) * STAGE, *bs = as + A_FLOATS;
    float big[MT][NT][4], cross[MT][NT][4];
#pragma unroll
    for (int k = 0; k < TC_BK; k += 16) {
      // x[..][2 s + h]: slot t + 4 h of 8-k step s
      float ax[MT][2][4], bx[NT][4];
      if constexpr (A_K) {
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
          for (int e = 0; e < 2; e++) lds_vec<4>(as + SmallTile<BM, true>::at(a_row(i, g, e), k + 4 * t), ax[i][e]);
      } else {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          float v[2 * MT];
          lds_vec<2 * MT>(as + SmallTile<BM, false>::at(k + 4 * t + q, a_row(0, g, 0)), v);
#pragma unroll
          for (int i = 0; i < MT; i++) { ax[i][0][q] = v[2 * i]; ax[i][1][q] = v[2 * i + 1]; }
        }
      }
      if constexpr (B_K) {
#pragma unroll
        for (int j = 0; j < NT; j++) lds_vec<4>(bs + SmallTile<BN, true>::at(b_row(j, g), k + 4 * t), bx[j]);
      } else {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          float v[NT];
          lds_vec<NT>(bs + SmallTile<BN, false>::at(k + 4 * t + q, b_row(0, g)), v);
#pragma unroll
          for (int j = 0; j < NT; j++) bx[j][q] = v[j];
        }
      }
#pragma unroll
      for (int s8 = 0; s8 < 2; s8++) {
        uint32_t ah[MT][4], al[MT][4];
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
          for (int e = 0; e < 4; e++) split_tf32(ax[i][e & 1][2 * s8 + (e >> 1)], ah[i][e], al[i][e]);
#pragma unroll
        for (int j = 0; j < NT; j++) {
          uint32_t bh[2], bl[2];
#pragma unroll
          for (int e = 0; e < 2; e++) split_tf32(bx[j][2 * s8 + e], bh[e], bl[e]);
          const bool fresh = k == 0 && s8 == 0;
#pragma unroll
          for (int i = 0; i < MT; i++) {
            mma_tf32(cross[i][j], al[i], bh, fresh);
            mma_tf32(big[i][j], ah[i], bh, fresh);
            mma_tf32(cross[i][j], ah[i], bl);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][j][e] += big[i][j][e] + cross[i][j][e];
  }
  cp_async_wait<0>();
  // a NaN among the sums leaves one in their sum, added up in four chains (so may opposite infinities, which costs a look at each)
  float any[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) any[e] += acc[i][j][e];
  const float all4 = (any[0] + any[1]) + (any[2] + any[3]);
  if (all4 != all4) {
    const int k0 = kt0 * TC_BK, k1 = min(p.K, k0 + nk * TC_BK);
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int m = m0 + a_row(i, g, e >> 1), n = n0 + b_row(j, 2 * t + (e & 1));
          if (acc[i][j][e] != acc[i][j][e] && m < p.M && n < p.N) acc[i][j][e] = fp32_sum<A_K, B_K>(p, m, n, k0, k1);
        }
  }
  if (p.slices > 1) {
    const long tile = (long)blockIdx.y * gridDim.x + blockIdx.x;
    constexpr int NV = MT * NT * 4;
    float *mine = p.ws + (tile * p.slices + blockIdx.z) * (NV * SM_THREADS) + tid;
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) mine[((i * NT + j) * 4 + e) * SM_THREADS] = acc[i][j][e];
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      is_last = atomicAdd(p.tickets + tile, 1u) == (unsigned)p.slices - 1;
      if (is_last) p.tickets[tile] = 0;   // ready for the next launch on this stream
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int j = 0; j < NT; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][j][e] = 0.f;
    const float *all = p.ws + tile * p.slices * (long)(NV * SM_THREADS) + tid;
    constexpr int UZ = NV >= 32 ? 1 : 32 / NV;   // about 32 loads in flight
#pragma unroll UZ
    for (int z = 0; z < p.slices; z++)
#pragma unroll
      for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
          for (int e = 0; e < 4; e++) acc[i][j][e] += __ldcg(all + ((long)z * NV + (i * NT + j) * 4 + e) * SM_THREADS);
  }
  if (stalled) return;
  auto store = [&](auto accumulate) {
    constexpr bool OLD = decltype(accumulate)::value;
    // Old values are asked for together, before the first store: otherwise each waits for its own round trip, up to 32 of them one
    // after the other (1574 x 1276 x 2 with beta = 1: 53 us, 18 with the loads ahead; 15 with beta = 0).
    float old[OLD ? MT : 1][OLD ? NT : 1][4];
    if constexpr (OLD) {
#pragma unroll
      for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int m = m0 + a_row(i, g, e >> 1), n = n0 + b_row(j, 2 * t + (e & 1));
            old[i][j][e] = m < p.M && n < p.N ? p.c[(long)m * p.sm + (long)n * p.sn] : 0.f;
          }
    }
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int e2 = 0; e2 < 2; e2++) {
        const int m = m0 + a_row(i, g, e2);
        if (m >= p.M) continue;
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
          for (int e1 = 0; e1 < 2; e1++) {
            const int n = n0 + b_row(j, 2 * t + e1);
            if (n >= p.N) continue;
            float v = p.alpha * acc[i][j][2 * e2 + e1];
            if (p.bias) v += p.bias[m * p.bias_m + n * p.bias_n];
            if constexpr (OLD) v += p.beta * old[i][j][2 * e2 + e1];
            p.c[(long)m * p.sm + (long)n * p.sn] = v;
          }
      }
  };
  if (p.beta != 0.f) store(std::true_type());
  else store(std::false_type());
}

// A long K-major matrix against a handful of K-major rows (a fully connected layer over one to eight images): the
// matrix's bytes are the bound, each is used R times, and FP32 multiply-adds keep up with them.  A warp takes RA rows of
// the matrix and every (8 / groups)-th 128-k chunk, the RA x UNROLL 16-byte loads of UNROLL chunks in flight before the
// first multiply-add (8 to 16, as registers allow); the 8 warps of a block are `groups` sets of rows times 8 / groups
// interleaved slices of k, whose sums meet in shared memory, so no second launch or workspace follows.  The warps of a slice
// read the same chunk of the few rows at about the same time, which the L1 serves.  In a loop over one
// matrix, against the tiles above: 9216 -> 4096 outputs (151 MB) 42.5 -> 26 us for one and two rows (5.8 TB/s), 33 for four;
// 4096 -> 1000 (16 MB, which then stays in L2) 12.5 -> 6.5; 512 -> 512 5.0 -> 3.3.  With the matrix in DRAM: 32, 18 (4096 -> 4096) and
// 11 us, i.e. 4.7, 3.7 and 1.5 TB/s: the shorter the launch, the more of it is its start.
template <int R, int RA, int UNROLL>
__global__ void __launch_bounds__(256) few_rows_kernel(const SmallProblem p, int groups) {
  pdl_begin();
  __shared__ float part[8][RA * R];
  const int stalled = *reinterpret_cast<const volatile int *>(p.stalled);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nslices = 8 / groups, slice = warp / groups, group = warp % groups;
  const int m0 = ((int)blockIdx.x * groups + group) * RA;
  float acc[RA][R];
  const float *a[RA], *b[R];
#pragma unroll
  for (int i = 0; i < RA; i++) a[i] = p.a.base + (long)min(m0 + i, p.M - 1) * p.a.ld;
#pragma unroll
  for (int j = 0; j < R; j++) b[j] = p.b.base + (long)min(j, p.N - 1) * p.b.ld;
#pragma unroll
  for (int i = 0; i < RA; i++)
#pragma unroll
    for (int j = 0; j < R; j++) acc[i][j] = 0.f;
  const int step = nslices * 128;
  for (int k = slice * 128 + lane * 4; k < p.K; k += UNROLL * step) {   // K is a multiple of 4
    float4 w[UNROLL][RA];
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      const bool in = k + u * step < p.K;
#pragma unroll
      for (int i = 0; i < RA; i++)
        w[u][i] = in ? __ldcs(reinterpret_cast<const float4 *>(a[i] + k + u * step)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < UNROLL; u++) {
      if (k + u * step >= p.K) break;
#pragma unroll
      for (int j = 0; j < R; j++) {
        const float4 x = *reinterpret_cast<const float4 *>(b[j] + k + u * step);
#pragma unroll
        for (int i = 0; i < RA; i++)
          acc[i][j] = fmaf(w[u][i].w, x.w, fmaf(w[u][i].z, x.z, fmaf(w[u][i].y, x.y, fmaf(w[u][i].x, x.x, acc[i][j]))));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RA; i++)
#pragma unroll
    for (int j = 0; j < R; j++) {
      float v = acc[i][j];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) part[warp][i * R + j] = v;
    }
  __syncthreads();
  if (stalled) return;
  for (int e = threadIdx.x; e < groups * RA * R; e += 256) {
    const int g = e / (RA * R), i = e / R % RA, n = e % R, m = ((int)blockIdx.x * groups + g) * RA + i;
    if (m >= p.M || n >= p.N) continue;
    float sum = 0.f;
    for (int z = 0; z < nslices; z++) sum += part[z * groups + g][i * R + n];
    float *o = p.c + (long)m * p.sm + (long)n * p.sn;
    float v = p.alpha * sum;
    if (p.bias) v += p.bias[m * p.bias_m + n * p.bias_n];
    if (p.beta != 0.f) v += p.beta * *o;
    *o = v;
  }
}

}  // namespace mm
}  // namespace thc

#endif
