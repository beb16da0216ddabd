// Two-SM tcgen05 engine over operands fetched by TMA: FP32 values as 3xTF32 products split inside the SM, FP32 values that come as
// FP16 pairs, or BF16 values.
//
// A cluster of two CTAs on neighbouring SMs computes one 256 x BN2 tile of D (BN2 = 64, 128, 192 or 256): CTA r of the pair
// stages rows [128 r, 128 r + 128) of the A tile and rows [BN2/2 r, BN2/2 (r+1)) of the B tile in its own shared
// memory; the MMAs, issued by CTA 0, read both CTAs' shared memory and leave rows [128 r, +128) of the result in CTA
// r's tensor memory, so that every byte fetched from L2 feeds twice the arithmetic of a one-SM tile.
//
// FP32: TMA brings the values themselves (four bytes per element) straight into the `hi` slot of a stage, in the swizzled
// layout the MMAs read; kind::tf32 ignores the low 13 mantissa bits of its operands, so that slot already is the
// hi operand, hi = trunc_tf32(x).  Four splitter warps per CTA read the slot back and write lo = tf32(x - hi) into
// the `lo` slot at the same offsets (both slots share one layout, K-major or MN-major alike).  Twelve MMAs per 32-k tile,
// Alo*Bhi + Ahi*Blo + Ahi*Bhi, go into one of two TMEM buffers and are added into FP32 registers with
// round-to-nearest (the tensor core's own accumulation truncates, so chains stay 12 MMAs long).
//
// FP16 pairs (RangeRec, mm_problem.cuh): the same three products from halves that a pass over the operands has made, at twice the
// rate of TF32 and without the splitters' shared-memory traffic.  A ring slot holds one half of a 64-k tile, lo before hi, and
// twelve kind::f16 MMAs multiply a tile: Alo*Bhi + Ahi*Blo at 2^11 times their size, which the first of Ahi*Bhi scales back
// (scale-input-d).  Each tile has an accumulator of its own, as in TF32, whose chain of full-size additions is as long (four MMAs)
// over twice the k, so that the error is smaller: 4096^3 of normal values 1.95e-7 of the result's norm against 2.94e-7 (2048^3
// 1.70e-7 / 2.61e-7, 8192^3 2.44e-7 / 3.60e-7).  Time with the passes over the operands: 4096^3 659 -> 430 us, 8192^3 4.78 -> 2.69 ms;
// the 256-wide convolution launches of 1024 images run 500-570 TFLOP/s where TF32 had 240-250 (its ceiling 277).
// What bounds it: the wide tiles the tensor pipe under the power cap (570-600 TFLOP/s = 1.7-1.8 PFLOP/s of MMAs).
//
// 16-bit operands of either kind: the loads of both CTAs complete on CTA 0's `full` barrier directly, tiles of up to 128 columns have
// four accumulator buffers (they end an item every few microseconds, and the MMAs run on while its results are stored), and
// the warp that issues the loads carries its coordinates on by additions.  A relayed barrier, two
// buffers and divisions for every load took, at 1024 images: first layer forward 1121 -> 986 us, its weight gradient 971 -> 728,
// gradInput 64 <- 192 1625 -> 1525, the 256-wide weight gradients 357 -> 340; 128 images 3207 -> 3115 us a step.
//
// BF16 (opt-in math mode): no splitters and no lo slots, four kind::f16 MMAs per 64-k tile; products are exact
// in FP32 and the tolerance of the mode is BF16's, so four k tiles (16 MMAs) chain in one accumulator before a drain.  No pipe is
// full (4096^3: 136 us, 1.0 PFLOP/s, tensor pipe 47 % busy): 7.9 TB/s cross from L2 into the SMs, 64 KB per 256 x 256 x 64
// step of the pair, near the most any engine here has moved.
//
// Rings: R `hi` slots (loads in flight, tiles being split, tiles being multiplied) and L <= R `lo` slots
// (only tiles being split or multiplied), so that the load queue can be deep.
//
// Roles (512 threads per CTA):
//   warps 0-3   splitters, two groups of two warps taking alternate k tiles: wait for the tile's TMA bytes
//               (`raw_full`, CTA-local) and for its lo slot to be free, split, publish to the async proxy,
//               arrive on CTA 0's `full`.  16-bit operands have nothing to split: there these warps are idle, or (GatheredWindowOperand) copy
//               the A rows of their CTA by cp.async, each a quarter of every tile, and arrive on CTA 0's `full` as the copies land.
//   warps 4, 6  (CTA 0) issue the MMAs of the even and the odd k tiles (16-bit operands: warp 4 all).
//   warp 5      issues the TMA loads of this CTA's A rows and B rows, R - 1 tiles ahead,
//               as soon as the MMAs that read a slot have completed (`empty`).
//   warps 8-15  drain: tcgen05.ld every finished partial tile and add it into FP32 registers; then the epilogue.
// The issuing warps run their loops with all lanes and elect a thread for each tile's instructions (elect_one, mm_tc.cuh).  With a
// single thread in the loop the MMAs of narrow tiles were bound by their issue: 512 images, forward 64 -> 192 (192 columns) 596 -> 500
// us, gradInput 64 <- 192 (pixel pairs, 128) 839 -> 645, 64 -> 128 of 112 x 112 (128) 399 -> 320, in BF16 278 -> 240 and (64 columns)
// 566 -> 464; tiles of 256 columns, which the power cap holds, 3 %.
// Registers are rebalanced with setmaxnreg: the drain warps hold BN2/2 accumulators per thread.
// The kernel is persistent: see tc2r_kernel.
// Every wait is bounded; on expiry the CTA tells its peer, raises the stall flags (StallCtl, mm_tc.cuh), skips
// its stores and still joins the final cluster barrier.
#ifndef THC_MM_TC2R_CUH
#define THC_MM_TC2R_CUH

#include "mm_tc.cuh"

namespace thc {
namespace mm {

constexpr int T2_PRODUCERS = 128;
constexpr int T2_MMA_WARP = 4;
constexpr int T2_DRAIN_WARP0 = 8;
constexpr int T2_DRAIN_WARPS = 8;
constexpr int T2_THREADS = 512;
constexpr int T2R_HALF_CHAIN = 4;   // BF16: k tiles accumulated in tensor memory before the drain warps fold them
constexpr int kGatherAhead = 4;     // tiles on the way to a warp that gathers A
constexpr int T2R_TMA_WARP = 5;
constexpr int T2R_MMA_WARP2 = 6;

template <int BN2, int PREC> struct Tc2rCfg {
  static constexpr bool HALF = PREC != kTf32;
  static constexpr int BH = BN2 / 2;
  static constexpr int A_BYTES = TC_BM * 128;
  static constexpr int B_BYTES = BH * 128;
  static constexpr int SLOT_BYTES = A_BYTES + B_BYTES;          // one precision of this CTA's A rows and B rows
  static constexpr int LO_SLOTS = HALF ? 0 : 3;
  static constexpr int HI_MAX = (227 * 1024 - 1024 - 512) / SLOT_BYTES - LO_SLOTS;
  static constexpr int HI_SLOTS = HI_MAX > (HALF ? 8 : 6) ? (HALF ? 8 : 6) : HI_MAX;
  static constexpr int ACCS = HALF && BN2 <= 128 ? 4 : 2;       // accumulator buffers
  static constexpr int TMEM_COLS = ACCS * BN2 > 256 ? 512 : 256;
  static constexpr int SMEM_BYTES = (HI_SLOTS + LO_SLOTS) * SLOT_BYTES + 512 + 1024;
  static_assert(HI_SLOTS >= LO_SLOTS, "ring sizes");
  static_assert(HALF || HI_SLOTS % 2 == 0 || HI_SLOTS <= LO_SLOTS + 2, "an odd hi ring must not be longer than the lo ring + 2 (parity waits of the two MMA warps)");
};

// What a launch asks for: one over pairs may have to run as kTf32.
template <int BN2, int PREC> __host__ __device__ constexpr int tc2r_smem_bytes() {
  constexpr int own = Tc2rCfg<BN2, PREC>::SMEM_BYTES, wide = Tc2rCfg<BN2, kTf32>::SMEM_BYTES;
  return PREC == kPairs && wide > own ? wide : own;
}

// lo = tf32(x - trunc_tf32(x)) of four values
__device__ __forceinline__ uint4 tf32_lo4(const uint4 &v) {
  uint4 l;
  l.x = to_tf32(__uint_as_float(v.x) - __uint_as_float(v.x & 0xffffe000u));
  l.y = to_tf32(__uint_as_float(v.y) - __uint_as_float(v.y & 0xffffe000u));
  l.z = to_tf32(__uint_as_float(v.z) - __uint_as_float(v.z & 0xffffe000u));
  l.w = to_tf32(__uint_as_float(v.w) - __uint_as_float(v.w & 0xffffe000u));
  return l;
}
// Volatile without a memory clobber: these keep their order among themselves and against the (volatile) barrier
// waits and fences around them, which is all the splitter needs, and leave the compiler free to keep values
// in registers across them.
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4 &v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w));
}

// Tiled TMA loads of one CTA's share of a plain matrix operand: K-major, one {32 k, ROWS} box; MN-major, one
// {32 rows, 32 k} box per 32-row block (4096 bytes each).  Completion in bytes on this CTA's `mbar`.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void *tmap, int x, int y, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"((unsigned long long)tmap), "r"(mbar), "r"(x), "r"(y)
      : "memory");
}
// The loads of one CTA's share of an operand, ROWS rows from row0 on, k tile after k tile.  PREC: the form the operand's buffer is in;
// `lo`: the second half of a pair.  One warp issues them all, and what it does between two loads is on the engine's
// critical path: coordinates are found by division once per item and carried on by additions.
template <int ROWS, int PREC, bool WIDE, class Op> struct TileLoader;
template <int ROWS, int PREC, bool WIDE, bool MN, int OWN>
struct TileLoader<ROWS, PREC, WIDE, RawOperand<MN, OWN>> {
  static constexpr int KV = PREC == kTf32 ? 32 : 64;
  int row, k;
  __device__ __forceinline__ TileLoader(const RawOperand<MN, OWN> &, long row0, long k0) : row((int)row0), k((int)k0) {}
  __device__ __forceinline__ void issue(const RawOperand<MN, OWN> &op, uint32_t dst, bool lo, uint32_t mbar) const {
    if constexpr (MN) {
      static_assert(ROWS % KV == 0, "whole row blocks");
#pragma unroll
      for (int a = 0; a < ROWS / KV; a++) tma_load_2d(dst + a * KV * 128, op.map(WIDE), row + KV * a + op.half(lo), k, mbar);
    } else {
      tma_load_2d(dst, op.map(WIDE), k + op.half(lo), row, mbar);
    }
  }
  __device__ __forceinline__ void next(const RawOperand<MN, OWN> &) { k += KV; }
};
// Convolution windows as rows (K-major): one im2col load of KV channels of ROWS = 128 consecutive windows.
template <int ROWS, int PREC, bool WIDE, int OWN>
struct TileLoader<ROWS, PREC, WIDE, PlanesWindowOperand<OWN>> {
  static constexpr int KV = PREC == kTf32 ? 32 : 64;
  static_assert(ROWS == TC_BM, "the window map loads 128 windows");
  int x, y, img, i, j, c;
  __device__ __forceinline__ TileLoader(const PlanesWindowOperand<OWN> &op, long row0, long k0) {
    op.tile_origin(row0, x, y, img);
    op.tile_tap((unsigned)k0, i, j, c);
  }
  __device__ __forceinline__ void issue(const PlanesWindowOperand<OWN> &op, uint32_t dst, bool lo, uint32_t mbar) const {
    tma_load_windows(dst, op.map(WIDE), c + op.half(lo), x, y, img, j, i, mbar);
  }
  __device__ __forceinline__ void next(const PlanesWindowOperand<OWN> &op) {
    c += KV;
    if (c == (int)op.C.d) {
      c = 0;
      if (++j == (int)op.kW.d) { j = 0; i++; }
    }
  }
};
// Convolution windows as the reduction (MN-major): per KV-row block, KV channels of KV consecutive windows.
template <int ROWS, int PREC, bool WIDE, int OWN>
struct TileLoader<ROWS, PREC, WIDE, WindowRowsOperand<OWN>> {
  static constexpr int KV = PREC == kTf32 ? 32 : 64, BLOCKS = ROWS / KV;
  static_assert(ROWS % KV == 0, "whole row blocks");
  int x, y, img, i0, j0, c0;   // the other blocks' taps by addition each time: kept, they would spill
  __device__ __forceinline__ TileLoader(const WindowRowsOperand<OWN> &op, long row0, long k0) {
    op.pixel(k0, x, y, img);
    op.row_tap(row0, i0, j0, c0);
  }
  __device__ __forceinline__ void issue(const WindowRowsOperand<OWN> &op, uint32_t dst, bool lo, uint32_t mbar) const {
    const int cx = x * op.ks.sx + op.ks.x0, cy = y * op.ks.sy + op.ks.y0;
    int i = i0, j = j0, c = c0;
#pragma unroll
    for (int a = 0; a < BLOCKS; a++) {
      tma_load_windows(dst + a * KV * 128, op.map(WIDE), c + op.half(lo), cx, cy, img, j, i, mbar);
      c += KV;
      if (c == (int)op.C.d) {
        c = 0;
        if (++j == (int)op.kW.d) { j = 0; i++; }
      }
    }
  }
  __device__ __forceinline__ void next(const WindowRowsOperand<OWN> &op) {   // KV pixels on
    const WindowStep &s = op.step[PREC == kTf32 ? 0 : 1];
    x += s.x; y += s.y; img += s.img;
    if (x >= (int)op.ks.XW.d) { x -= (int)op.ks.XW.d; y++; }
    if (y >= op.oH) { y -= op.oH; img++; }
  }
};

// Windows that the splitter warps gather.
template <int ROWS, int PREC, bool WIDE>
struct TileLoader<ROWS, PREC, WIDE, GatheredWindowOperand> {
  __device__ __forceinline__ TileLoader(const GatheredWindowOperand &, long, long) {}
  __device__ __forceinline__ void issue(const GatheredWindowOperand &, uint32_t, bool, uint32_t) const {}
  __device__ __forceinline__ void next(const GatheredWindowOperand &) {}
};

// ---- item hand-out ------------------------------------------------------------------------------------------
// The clusters of a launch take their work items from a counter in device memory, first come first served, so a
// cluster that starts late (its SMs were still busy with another stream's kernel: a collective, a parameter
// update) simply takes fewer items instead of leaving its fixed share to run alone at the end.  One thread of the
// leader CTA fetches the next item number when the leader's TMA warp, the role that runs furthest ahead, starts on
// the current one (`go` barrier): one item of look-ahead hides the counter's round trip, and a cluster never holds
// claims on work it is not about to do.  The numbers go into a ring of T2R_SCHED slots that exists in both CTAs;
// every role of both CTAs reads the ring in the same order.  Slot protocol: `full` (one per CTA, count 1) completes
// when the number is there; `empty` (leader CTA only) collects one arrival per reading role of either CTA.  The
// peer's copy travels as st.async, whose completion is counted in bytes on the peer's `full` barrier: the peer
// sees the number when it sees the phase.
constexpr int T2R_SCHED = 8;
constexpr int T2R_SCHED_WARP = 7;
constexpr uint32_t T2R_NO_ITEM = 0xffffffffu;
constexpr int T2R_ITEM_WAIT_SHIFT = 6;   // item-level waits may take 64 k-tile limits (see mbar_wait)
// readers per slot: TMA warp, 4 splitter warps (16-bit operands: none, or the 4 that gather A), 8 drain warps in each CTA, the MMA warps in the leader
template <bool HALF, bool GATHERED> struct Tc2rReaders { static constexpr uint32_t count = 2 * (1 + (HALF && !GATHERED ? 0 : 4) + T2_DRAIN_WARPS) + (HALF ? 1 : 2); };

__device__ __forceinline__ void mbar_arrive_local(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void sched_publish_peer(uint32_t peer_item, uint32_t peer_full, uint32_t w) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(peer_full), "r"(4u) : "memory");
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];"
               ::"r"(peer_item), "r"(w), "r"(peer_full) : "memory");
}
struct Tc2rSched {
  uint32_t full, empty_leader, ring;   // shared-memory addresses: this CTA's `full` barriers and ring, the leader's `empty`
  // The n-th item number of this cluster (T2R_NO_ITEM: no more work), or false when the wait ran out.  A warp calls
  // this with all lanes; its lane 0 (or the single calling thread) then reports the slot read with done().
  __device__ __forceinline__ bool next(uint32_t n, uint32_t &w, volatile WaitCtl *ctl) const {
    const uint32_t slot = n % T2R_SCHED;
    if (!mbar_wait(full + 8 * slot, (n / T2R_SCHED) & 1u, ctl, kWaitItemNumber, T2R_ITEM_WAIT_SHIFT)) return false;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w) : "r"(ring + 4 * slot) : "memory");
    return true;
  }
  __device__ __forceinline__ void done(uint32_t n) const { mbar_arrive_cluster(empty_leader + 8 * (n % T2R_SCHED)); }
};

// One work item of a launch: a 256 x BN2 tile of the product over one split-K slice.
struct Tc2rItem {
  long m_tile0, n_tile0, k_begin;
  long z;      // k slice of a tail tile, -1 for a whole-reduction tile
  long slot;   // partial-sum block of the workspace (tail items only)
  int num_k_tiles;
};

// Persistent: the launch has as many clusters as the device runs at once; cluster c starts with item c and takes
// further items from `sched_counter` (zero at launch) as it finishes (m tiles fastest, so that clusters running
// side by side share their B rows in L2).  All
// rings, barrier phases and accumulator buffers run on with a k-tile count `g` that spans the items, so the
// loads, splits and first MMAs of an item run under the previous item's epilogue stores, and the barrier and
// tensor-memory set-up is paid once per launch.
// PREC: what is multiplied; WIDE: operands meant as FP16 pairs that are in FP32 (kTf32 then).
template <class P, int BN2, int PREC, bool WIDE>
__device__ __forceinline__ void tc2r_run(const P &p, const StallCtl &ctl, unsigned *sched_counter) {
  constexpr bool HALF = PREC != kTf32;     // operands of 16 bits: nothing is split here
  constexpr bool PAIRS = PREC == kPairs, GATHERED = P::OpA::GATHERED;
  constexpr int PARTS = PAIRS ? 2 : 1;     // ring slots of a k tile: lo, then hi, which is needed longest
  constexpr int KV = HALF ? 64 : 32;
  constexpr int CHAIN = PAIRS ? 1 : T2R_HALF_CHAIN;
  typedef Tc2rCfg<BN2, PREC> Cfg;
  constexpr int R = Cfg::HI_SLOTS, L = Cfg::LO_SLOTS, LM = L > 0 ? L : 1, ACCS = Cfg::ACCS;
  constexpr int BH = Cfg::BH;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t *lo_ring = smem + R * Cfg::SLOT_BYTES;
  uint8_t *aux = lo_ring + L * Cfg::SLOT_BYTES;
  // full[R], empty[R], raw_full[R] (kTf32), acc_full[ACCS], acc_empty[ACCS], lo_empty[L], sched_full[T2R_SCHED], sched_empty[T2R_SCHED], sched_go
  uint64_t *bars = reinterpret_cast<uint64_t *>(aux);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3 * R + 2 * ACCS + L + 2 * T2R_SCHED + 1);
  volatile WaitCtl *abort_flag = reinterpret_cast<volatile WaitCtl *>(tmem_slot + 2);
  uint32_t *sched_ring = tmem_slot + 2 + sizeof(WaitCtl) / 4;
  static_assert((3 * R + 2 * ACCS + L + 2 * T2R_SCHED + 1) * 8 + 8 + sizeof(WaitCtl) + 4 * T2R_SCHED <= 512, "auxiliary shared memory");

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // warp: as a value that a warp has once
  const uint32_t rank = cluster_ctarank();
  // item counts fit 32 bits (checked by the launcher): the decode below runs once per item in every role
  const uint32_t gm = (uint32_t)((p.M + 255) / 256), gn = (uint32_t)((p.N + BN2 - 1) / BN2);
  const uint32_t tiles = gm * gn, tail_first = p.ws ? (uint32_t)p.tail_first : tiles;
  const uint32_t tail_tiles = tiles - tail_first;
  const uint32_t items = tail_first + tail_tiles * (uint32_t)p.tail_splits, cluster_id = blockIdx.x >> 1, clusters = gridDim.x >> 1;
  // Items 0 .. tail_first - 1 are whole tiles; the rest are the k slices of the tail tiles, slice-major (clusters
  // running side by side then work on neighbouring tiles of one k range and share its B rows in L2).
  auto item_at = [&](uint32_t w) {
    Tc2rItem t;
    uint32_t tile = w;
    t.z = -1;
    t.k_begin = 0;
    long k_end = p.K;
    if (w >= tail_first) {
      const uint32_t r = w - tail_first, z = r / tail_tiles;
      tile = tail_first + (r - z * tail_tiles);
      t.z = z;
      t.slot = (long)(tile - tail_first) * p.tail_splits + z;
      t.k_begin = (long)z * p.k_per_split;
      k_end = t.k_begin + p.k_per_split;
      if (k_end > p.K) k_end = p.K;
    }
    const uint32_t nt = tile / gm, mt = tile - nt * gm;
    t.m_tile0 = (long)mt * 256; t.n_tile0 = (long)nt * BN2;
    t.num_k_tiles = (int)((k_end - t.k_begin + KV - 1) / KV);
    return t;
  };

  const uint32_t bar_full = smem_u32(bars), bar_empty = smem_u32(bars + R), bar_raw = smem_u32(bars + 2 * R);
  const uint32_t bar_acc_full = smem_u32(bars + 3 * R), bar_acc_empty = smem_u32(bars + 3 * R + ACCS);
  const uint32_t bar_lo_empty = smem_u32(bars + 3 * R + 2 * ACCS);
  const uint32_t bar_sched_full = smem_u32(bars + 3 * R + 2 * ACCS + L), bar_sched_empty = bar_sched_full + 8 * T2R_SCHED;
  const uint32_t bar_sched_go = bar_sched_empty + 8 * T2R_SCHED;
  Tc2rSched sched;
  sched.full = bar_sched_full;
  sched.empty_leader = mapa_shared(bar_sched_empty, 0);
  sched.ring = smem_u32(sched_ring);
  if (tid == 0) {
    for (int s = 0; s < R; s++) {
      mbar_init(bar_full + 8 * s, GATHERED ? 1 + 2 * T2_PRODUCERS / 32 : HALF ? 1 : 2 * T2_PRODUCERS / 64);   // used in CTA 0: its TMA warp and both CTAs' bytes (and the four warps of each CTA that gather) / a group of two splitter warps in each CTA
      mbar_init(bar_empty + 8 * s, 1);
      mbar_init(bar_raw + 8 * s, 1);                        // this CTA's TMA warp + the bytes it announces
    }
    for (int l = 0; l < L; l++) mbar_init(bar_lo_empty + 8 * l, 1);
    for (int k = 0; k < T2R_SCHED; k++) {
      mbar_init(bar_sched_full + 8 * k, 1);
      mbar_init(bar_sched_empty + 8 * k, Tc2rReaders<HALF, GATHERED>::count);   // used in CTA 0
    }
    mbar_init(bar_sched_go, 1);                                // used in CTA 0
    for (int b = 0; b < ACCS; b++) {
      mbar_init(bar_acc_full + 8 * b, 1);
      mbar_init(bar_acc_empty + 8 * b, 2 * T2_DRAIN_WARPS);
    }
    wait_ctl_init(abort_flag, ctl, mapa_shared(smem_u32(const_cast<int *>(&abort_flag->abort)), rank ^ 1u));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == T2_MMA_WARP) tmem_alloc2(smem_u32(tmem_slot), Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = abort_flag->abort == 0;   // set on entry: an earlier kernel of this stream stalled, do no work

  if (!ok) {
    if (tid == 0) wait_ctl_give_up(abort_flag, kWaitEntry);   // the peer may have read the flag before it was set: tell it
  } else if (warp < T2_MMA_WARP) {
    // ------------------------------------------------------------ splitters
    setmaxnreg_dec<72>();
    const uint32_t full_leader = mapa_shared(bar_full, 0);
    if constexpr (GATHERED) {
      // A warp copies 32 windows' taps of a k tile: eight lanes the eight taps of one window, which are 128 bytes of the image where they
      // belong to one filter row.  kGatherAhead tiles are on the way before the first is waited for, across items.  Bound by these copies, in
      // L1 and what it misses: 256 images of the 11 x 11 / 4 layer over three planes (us) 305 with 4 tiles ahead, 330 with 2 and half the ring; past
      // L1 345, and more with more on the way (6: 356, 8: 388).  With the pass that makes the image (54) 359, where the column matrix, written
      // and read through DRAM at 1.6 GB, took 605.
      static_assert(PREC == kBf16 && kGatherAhead < R, "k = (tap, 16 bytes); a slot is free before its turn to be announced comes");
      const uint32_t ring = smem_u32(smem);
      const int c = lane & 7, r0 = warp * 32 + (lane >> 3);
      const uint32_t at[2] = {(uint32_t)(r0 * 128 + ((c ^ (lane >> 3)) << 4)), (uint32_t)((r0 + 4) * 128 + ((c ^ ((lane >> 3) + 4)) << 4))};   // 128-byte swizzle
      uint32_t s = 0, phase = 0, told = 0;
      int ahead = 0;
      bool filled = false;
      auto tell = [&]() {   // the oldest tile not announced yet has landed
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(full_leader + 8 * told);
        if (++told == R) told = 0;
      };
      for (uint32_t n = 0; ok; n++) {
        uint32_t w = T2R_NO_ITEM;
        ok = __all_sync(0xffffffffu, sched.next(n, w, abort_flag));
        if (!ok) break;
        if (lane == 0) sched.done(n);
        if (w == T2R_NO_ITEM) break;
        const Tc2rItem item = item_at(w);
        const uint4 *row[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const long m = min(item.m_tile0 + (long)rank * TC_BM + r0 + 4 * i, p.M - 1);   // (rows past the end are not stored)
          unsigned img, px, y, x;
          p.a.rows.PP.divmod((unsigned)m, img, px);
          p.a.rows.XW.divmod(px, y, x);
          row[i] = p.a.image + ((long)img * p.a.image_pixels + (int)y * p.a.rows.sy * p.a.pitch + (int)x * p.a.rows.sx);
        }
        int tap = (int)(item.k_begin >> 3) + c, ti = tap / p.a.kW, tj = tap - ti * p.a.kW;
        for (int t = 0; t < item.num_k_tiles; t++) {
          if (filled) ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, phase ^ 1u, abort_flag, kWaitSlotEmpty));
          if (!ok) break;
          const bool there = tap < p.a.taps;
          const int off = there ? ti * p.a.pitch + tj : 0;
          const uint32_t slot = ring + s * Cfg::SLOT_BYTES;
#pragma unroll
          for (int i = 0; i < 8; i++) cp_async16(slot + at[i & 1] + (uint32_t)((i >> 1) * 1024), row[i] + off, there);
          cp_async_commit();
          if (ahead == kGatherAhead) { cp_async_wait<kGatherAhead>(); tell(); } else ahead++;
          tap += 8; tj += 8;
          while (tj >= p.a.kW) { tj -= p.a.kW; ti++; }
          if (++s == R) { s = 0; phase ^= 1u; filled = true; }
        }
      }
      cp_async_wait<0>();
      if (ok)
        for (; ahead > 0; ahead--) tell();
    } else if constexpr (!HALF) {
    // Two groups of two warps take alternate k tiles, so that one group's barrier round trips and proxy fence
    // overlap the other group's copying: under the MMAs' own shared-memory traffic every access here waits
    // hundreds of cycles.
    const int grp = warp >> 1, gtid = tid & 63;
    int g0 = 0;
    for (uint32_t n = 0; ok; n++) {
      uint32_t w = T2R_NO_ITEM;
      ok = __all_sync(0xffffffffu, sched.next(n, w, abort_flag));
      if (!ok) break;
      if (lane == 0) sched.done(n);
      if (w == T2R_NO_ITEM) break;
      const int nk = item_at(w).num_k_tiles;
      for (int it = (g0 + grp) & 1; it < nk; it += 2) {
        const int g = g0 + it;
        const int s = g % R, ls = g % LM;
        const uint32_t raw_bar = bar_raw + 8 * s, raw_par = (uint32_t)(g / R) & 1u;
        // The lo slot is free once the MMAs of tile g - L have read it.  It has a barrier of its own: the hi slots'
        // `empty` barriers can run two phases ahead of a splitter group that was slow to wake up (the other group and
        // the other MMA warp do not wait for it), and a parity wait cannot tell two completed phases from none.
        const uint32_t lo_bar = bar_lo_empty + 8 * ls, lo_par = (uint32_t)(g / LM + 1) & 1u;
        const bool r1 = mbar_try_wait(raw_bar, raw_par), r2 = g < L || mbar_try_wait(lo_bar, lo_par);
        ok = (r1 || mbar_wait(raw_bar, raw_par, abort_flag, kWaitRawTile)) && (r2 || mbar_wait(lo_bar, lo_par, abort_flag, kWaitLoSlot));
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t src = smem_u32(smem + s * Cfg::SLOT_BYTES) + (uint32_t)gtid * 16u;
        const uint32_t dst = smem_u32(lo_ring + ls * Cfg::SLOT_BYTES) + (uint32_t)gtid * 16u;
        // a quarter of the group's 16-byte chunks per batch: all loads of a batch are in flight before its first store
        constexpr int GT = T2_PRODUCERS / 2, PASSES = Cfg::SLOT_BYTES / (GT * 16), BATCH = PASSES <= 24 ? PASSES / 2 : PASSES / 4;
        static_assert(Cfg::SLOT_BYTES % (GT * 16 * 4) == 0, "slot size");
#pragma unroll
        for (int i0 = 0; i0 < PASSES; i0 += BATCH) {
          uint4 v[BATCH];
#pragma unroll
          for (int i = 0; i < BATCH; i++) v[i] = lds128(src + (uint32_t)((i0 + i) * GT * 16));
#pragma unroll
          for (int i = 0; i < BATCH; i++) sts128(dst + (uint32_t)((i0 + i) * GT * 16), tf32_lo4(v[i]));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(full_leader + 8 * s);
      }
      g0 += nk;
    }
    }
  } else if (warp < T2_DRAIN_WARP0) {
    setmaxnreg_dec<40>();
    if (HALF && warp == T2_MMA_WARP && rank == 0) {
      // ---------------------------------------------------------- MMA issuer of 16-bit operands: one warp, CHAIN k tiles per buffer
      constexpr bool A_MN = P::OpA::MN_MAJOR, B_MN = P::OpB::MN_MAJOR;
      constexpr uint32_t idesc = PAIRS ? umma2_idesc_f16(BN2, A_MN, B_MN) : umma2_idesc_bf16(BN2, A_MN, B_MN);
      const uint32_t ring = smem_u32(smem);
      uint32_t s = 0, phase = 0, buf = 0, acc_phase = 0;
      for (uint32_t n = 0; ok; n++) {
        uint32_t w = T2R_NO_ITEM;
        ok = __all_sync(0xffffffffu, sched.next(n, w, abort_flag));
        if (!ok) break;
        w = __shfl_sync(0xffffffffu, w, 0);
        if (lane == 0) sched.done(n);
        if (w == T2R_NO_ITEM) break;
        const int nk = item_at(w).num_k_tiles;
        for (int it = 0; it < nk; it++) {
          const bool first = it % CHAIN == 0, last = it % CHAIN == CHAIN - 1 || it == nk - 1;
          const uint32_t d = tmem_base + buf * BN2;
          if (first) ok = mbar_wait_spin(bar_acc_empty + 8 * buf, acc_phase ^ 1u, abort_flag, kWaitAccEmpty);
          ok = ok && mbar_wait_spin(bar_full + 8 * s, phase, abort_flag, kWaitTileFull);
          const uint32_t sl = s;
          if constexpr (PAIRS) {
            if (++s == R) { s = 0; phase ^= 1u; }
            ok = ok && mbar_wait_spin(bar_full + 8 * s, phase, abort_flag, kWaitTileFull);
          }
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            if constexpr (PAIRS) {
              const uint32_t lo = ring + sl * Cfg::SLOT_BYTES, hi = ring + s * Cfg::SLOT_BYTES;
              const uint64_t a_lo = umma_desc_half<A_MN>(lo), b_lo = umma_desc_half<B_MN>(lo + Cfg::A_BYTES);
              const uint64_t a_hi = umma_desc_half<A_MN>(hi), b_hi = umma_desc_half<B_MN>(hi + Cfg::A_BYTES);
#pragma unroll
              for (int kk = 0; kk < 4; kk++) {   // 16 k per MMA; these two carry 2^11
                const uint64_t adv_a = (uint64_t)((kk * umma_kstep_bytes_half<A_MN>()) >> 4), adv_b = (uint64_t)((kk * umma_kstep_bytes_half<B_MN>()) >> 4);
                umma2_f16(d, a_lo + adv_a, b_hi + adv_b, idesc, kk ? 1u : 0u);
                umma2_f16(d, a_hi + adv_a, b_lo + adv_b, idesc, 1u);
              }
              umma2_commit_both(bar_empty + 8 * sl);
              umma2_f16_scale11(d, a_hi, b_hi, idesc);
#pragma unroll
              for (int kk = 1; kk < 4; kk++)
                umma2_f16(d, a_hi + (uint64_t)((kk * umma_kstep_bytes_half<A_MN>()) >> 4), b_hi + (uint64_t)((kk * umma_kstep_bytes_half<B_MN>()) >> 4), idesc, 1u);
            } else {
              const uint32_t st = ring + s * Cfg::SLOT_BYTES;
              const uint64_t a_d = umma_desc_half<A_MN>(st), b_d = umma_desc_half<B_MN>(st + Cfg::A_BYTES);
#pragma unroll
              for (int kk = 0; kk < 4; kk++) {   // 16 k per MMA
                const uint64_t adv_a = (uint64_t)((kk * umma_kstep_bytes_half<A_MN>()) >> 4), adv_b = (uint64_t)((kk * umma_kstep_bytes_half<B_MN>()) >> 4);
                umma2_f16(d, a_d + adv_a, b_d + adv_b, idesc, (kk || !first) ? 1u : 0u);
              }
            }
            umma2_commit_both(bar_empty + 8 * s);
            if (last) umma2_commit_both(bar_acc_full + 8 * buf);
          }
          __syncwarp();
          if (++s == R) { s = 0; phase ^= 1u; }
          if (last && ++buf == ACCS) { buf = 0; acc_phase ^= 1u; }
        }
      }
    } else if (!HALF && (warp == T2_MMA_WARP || warp == T2R_MMA_WARP2) && rank == 0) {
      // ---------------------------------------------------------- MMA issuers
      // Two warps take alternate k tiles (and with them alternate accumulator buffers): while one is blocked on
      // the tensor pipe's queue the other sits through its barrier polls, each a shared-memory round trip of
      // hundreds of cycles under the MMAs' own traffic.
      // With an odd number of hi slots a warp meets a slot only every second time round, so its parity wait for
      // tile g sees the phase of tile g - 2R as "the previous one".  That is safe because the phase of tile g - R
      // is over by then: the warp has waited for tile g - 2, which was split only after the MMAs of tile g - 5
      // released its lo slot (three lo slots), and R = 5 is the only odd ring size in use (static_assert below).
      // A scheme in which a warp skips whole revolutions (alternate ITEMS instead of alternate tiles) loses that
      // guarantee and stalls.
      constexpr bool A_MN = P::OpA::MN_MAJOR, B_MN = P::OpB::MN_MAJOR;
      constexpr uint32_t idesc = umma2_idesc_tf32(BN2, A_MN, B_MN);
      const int buf = warp == T2_MMA_WARP ? 0 : 1;
      int g0 = 0;
      for (uint32_t n = 0; ok; n++) {
        uint32_t w = T2R_NO_ITEM;
        ok = __all_sync(0xffffffffu, sched.next(n, w, abort_flag));
        if (!ok) break;
        w = __shfl_sync(0xffffffffu, w, 0);
        if (lane == 0) sched.done(n);
        if (w == T2R_NO_ITEM) break;
        const int nk = item_at(w).num_k_tiles;
        for (int it = (g0 + buf) & 1; it < nk; it += 2) {
          const int g = g0 + it;
          const int s = g % R, ls = g % LM;
          const uint32_t phase = (uint32_t)(g / R) & 1u, acc_phase = (uint32_t)(g >> 1) & 1u;
          ok = mbar_wait_spin(bar_acc_empty + 8 * buf, acc_phase ^ 1u, abort_flag, kWaitAccEmpty);
          ok = __all_sync(0xffffffffu, ok && mbar_wait_spin(bar_full + 8 * s, phase, abort_flag, kWaitTileFull));
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
            const uint32_t hs = smem_u32(smem + s * Cfg::SLOT_BYTES), lsl = smem_u32(lo_ring + ls * Cfg::SLOT_BYTES);
            const uint64_t a_hi = umma_desc_sw128<A_MN>(hs), a_lo = umma_desc_sw128<A_MN>(lsl);
            const uint64_t b_hi = umma_desc_sw128<B_MN>(hs + Cfg::A_BYTES), b_lo = umma_desc_sw128<B_MN>(lsl + Cfg::A_BYTES);
            const uint32_t d = tmem_base + (uint32_t)(buf * BN2);
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {   // 8 k per MMA
              const uint64_t adv_a = (uint64_t)((kk * umma_kstep_bytes<A_MN>()) >> 4);
              const uint64_t adv_b = (uint64_t)((kk * umma_kstep_bytes<B_MN>()) >> 4);
              umma2_tf32(d, a_lo + adv_a, b_hi + adv_b, idesc, kk ? 1u : 0u);
              umma2_tf32(d, a_hi + adv_a, b_lo + adv_b, idesc, 1u);
            }
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {   // 8 k per MMA
              const uint64_t adv_a = (uint64_t)((kk * umma_kstep_bytes<A_MN>()) >> 4);
              const uint64_t adv_b = (uint64_t)((kk * umma_kstep_bytes<B_MN>()) >> 4);
              umma2_tf32(d, a_hi + adv_a, b_hi + adv_b, idesc, 1u);
            }
            umma2_commit_both(bar_empty + 8 * s);
            umma2_commit_both(bar_lo_empty + 8 * ls);
            umma2_commit_both(bar_acc_full + 8 * buf);
          }
          __syncwarp();
        }
        g0 += nk;
      }
    } else if (warp == T2R_TMA_WARP) {
      // ---------------------------------------------------------- TMA issuer (one warp per CTA)
      // 16-bit tiles are ready as they land: the bytes of both CTAs complete on CTA 0's `full`.  The peer's may come before CTA 0 has
      // announced them: the phase still waits for that arrival, and the peer's slot was free only after the phase before.
      const uint32_t full_leader = mapa_shared(bar_full, 0), ring = smem_u32(smem);
      uint32_t s = 0, phase = 0;
      bool filled = false;   // every slot has been used
      for (uint32_t n = 0; ok; n++) {
        uint32_t w = T2R_NO_ITEM;
        ok = __all_sync(0xffffffffu, sched.next(n, w, abort_flag));
        if (!ok) break;
        w = __shfl_sync(0xffffffffu, w, 0);
        if (lane == 0) sched.done(n);
        if (w == T2R_NO_ITEM) break;
        if (rank == 0 && lane == 0) mbar_arrive_local(bar_sched_go);   // item n is under way: time to fetch the number of item n + 1
        const Tc2rItem item = item_at(w);
        TileLoader<TC_BM, PREC, WIDE, typename P::OpA> load_a(p.a, item.m_tile0 + (long)rank * TC_BM, item.k_begin);   // (gathered: nothing)
        TileLoader<BH, PREC, WIDE, typename P::OpB> load_b(p.b, item.n_tile0 + (long)rank * BH, item.k_begin);
        for (int t = 0; ok && t < item.num_k_tiles; t++) {
#pragma unroll
          for (int part = 0; part < PARTS; part++) {
            const bool lo = PAIRS && part == 0;
            if (filled) ok = __all_sync(0xffffffffu, mbar_wait(bar_empty + 8 * s, phase ^ 1u, abort_flag, kWaitSlotEmpty));
            if (!ok) break;
            if (elect_one()) {
              const uint32_t slot = ring + s * Cfg::SLOT_BYTES;
              uint32_t landed = bar_raw + 8 * s;
              if constexpr (HALF) {
                landed = full_leader + 8 * s;
                if (rank == 0) mbar_arrive_expect_tx(bar_full + 8 * s, 2u * (GATHERED ? Cfg::B_BYTES : Cfg::SLOT_BYTES));
              } else {
                mbar_arrive_expect_tx(landed, (uint32_t)Cfg::SLOT_BYTES);
              }
              load_a.issue(p.a, slot, lo, landed);
              load_b.issue(p.b, slot + Cfg::A_BYTES, lo, landed);
            }
            __syncwarp();
            if (++s == R) { s = 0; phase ^= 1u; filled = true; }
          }
          load_a.next(p.a);
          load_b.next(p.b);
        }
      }
    } else if (warp == T2R_SCHED_WARP && rank == 0 && elect_one()) {
      // ---------------------------------------------------------- item hand-out (one thread per cluster)
      const uint32_t peer_ring = mapa_shared(sched.ring, 1), peer_full = mapa_shared(bar_sched_full, 1);
      for (uint32_t n = 0;; n++) {
        const uint32_t slot = n % T2R_SCHED;
        if (n >= 1 && !mbar_wait(bar_sched_go, (n - 1) & 1u, abort_flag, kWaitItemGo, T2R_ITEM_WAIT_SHIFT)) break;
        if (n >= T2R_SCHED && !mbar_wait(bar_sched_empty + 8 * slot, (n / T2R_SCHED - 1) & 1u, abort_flag, kWaitItemSlot, T2R_ITEM_WAIT_SHIFT)) break;
        uint32_t w = n == 0 ? cluster_id : clusters + atomicAdd(sched_counter, 1u);
        if (w >= items) w = T2R_NO_ITEM;
        sched_publish_peer(peer_ring + 4 * slot, peer_full + 8 * slot, w);
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(sched.ring + 4 * slot), "r"(w) : "memory");
        mbar_arrive_local(bar_sched_full + 8 * slot);
        if (w == T2R_NO_ITEM) break;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ drain + epilogue warps
    setmaxnreg_inc<192>();
    const int q = warp & 3;
    const int h = (warp - T2_DRAIN_WARP0) >> 2;
    constexpr int NCOL = BN2 / 2;
    const uint32_t acc_empty_leader = mapa_shared(bar_acc_empty, 0);
    // Pixel-pair products over 64 planes (a 128-column tile: parity 0 in columns 0-63, parity 1 in 64-127): this warp
    // takes 32 planes in both parities instead of 64 columns of one, for the whole-line epilogue
    const bool pair_capable = P::PAIR && BN2 == 128 && p.epi.pair_K == 64 && p.epi.beta == 0.f;
    float unscale_a = 1.f, unscale_b = 1.f;
    if constexpr (PAIRS) { unscale_a = pair_unscale(*p.range_a); unscale_b = pair_unscale(*p.range_b); }
    int g0 = 0;
    for (uint32_t n = 0; ok; n++) {
      uint32_t w = T2R_NO_ITEM;
      ok = __all_sync(0xffffffffu, sched.next(n, w, abort_flag));
      if (!ok) break;
      if (lane == 0) sched.done(n);
      if (w == T2R_NO_ITEM) break;
      const Tc2rItem item = item_at(w);
      const bool pair_lines = pair_capable && item.z < 0;   // tail slices keep the plain column order for the workspace
      float acc[NCOL];
#pragma unroll
      for (int j = 0; j < NCOL; j++) acc[j] = 0.f;
      const int folds = HALF ? (item.num_k_tiles + CHAIN - 1) / CHAIN : item.num_k_tiles;   // accumulators of this item
      for (int it = 0; it < folds; it++) {
        const int g = g0 + it;
        const int buf = g % ACCS;
        const uint32_t acc_phase = (uint32_t)(g / ACCS) & 1u;
        ok = mbar_wait(bar_acc_full + 8 * buf, acc_phase, abort_flag, kWaitAccFull);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const uint32_t t0 = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN2 + (pair_lines ? h * 32 : h * NCOL));
#pragma unroll
        for (int c0 = 0; c0 < NCOL; c0 += 32) {
          uint32_t v[32];
          tmem_ld32_nowait(t0 + (pair_lines ? 2 * c0 : c0), v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j++) acc[c0 + j] += __uint_as_float(v[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty_leader + 8 * buf);
      }
      g0 += folds;
      if constexpr (PAIRS) {
#pragma unroll
        for (int j = 0; j < NCOL; j++) acc[j] = acc[j] * unscale_a * unscale_b;
      }
      if (ok) {
        const long m = item.m_tile0 + (long)rank * TC_BM + q * 32 + lane;
        if (item.z >= 0) {
          // partial sums of a tail slice: ws[slot][column][row], a warp's 32 rows side by side
          float *o = p.ws + (item.slot * BN2 + h * NCOL) * 256 + (rank * TC_BM + q * 32 + lane);
#pragma unroll
          for (int j = 0; j < NCOL; j++) o[j * 256] = acc[j];
        } else if constexpr (P::PAIR && BN2 == 128) {
          if (pair_lines) tc2_store_pair_rows<P>(p, acc, m, h * 32);
          else tc2_store_rows<P, NCOL>(p, acc, m, item.n_tile0 + h * NCOL);
        } else {
          tc2_store_rows<P, NCOL>(p, acc, m, item.n_tile0 + h * NCOL);
        }
      }
    }
  }
  if (abort_flag->abort && tid == 0) stall_raise(ctl, abort_flag->abort);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == T2_MMA_WARP) tmem_dealloc2(tmem_base, Cfg::TMEM_COLS);
}
template <class P, int BN2>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(T2_THREADS, 1) tc2r_kernel(const __grid_constant__ P p, const StallCtl ctl,
                                                                                                unsigned *sched_counter) {
  pdl_wait();
  if constexpr (P::PREC == kPairs) {
    if (p.ranges.wide()) tc2r_run<P, BN2, kTf32, true>(p, ctl, sched_counter);
    else tc2r_run<P, BN2, kPairs, false>(p, ctl, sched_counter);
  } else {
    tc2r_run<P, BN2, P::PREC, false>(p, ctl, sched_counter);
  }
}

}  // namespace mm
}  // namespace thc

#endif
