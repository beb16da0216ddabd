// PTX wrappers of the tensor-core engines: mbarriers with bounded waits and stall reporting, tcgen05 MMAs of two-CTA groups,
// tensor memory, TMA loads, asynchronous copies.
//
// Every mbarrier wait is bounded (StallCtl::limit SM cycles); on expiry the CTA raises the stall flags
// (one in device memory that every later CTA of the stream reads on entry and then does no work, one in mapped
// host memory that the host reads at its next synchronisation point), skips its stores and exits normally.
#ifndef THC_MM_TC_CUH
#define THC_MM_TC_CUH

#include "mm_problem.cuh"

namespace thc {
namespace mm {

constexpr int TC_BM = 128;  // rows of A per CTA
constexpr int TC_BK = 32;   // floats per tile row = 128 bytes = one swizzle span (BF16: 64 values)

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(2000u)  // suspend-time hint (ns): sleep in hardware instead of spinning
      : "memory");
  return ok != 0;
}
// Stall handling.  StallCtl (thc_internal.h) is a kernel parameter: `dev_flag` (device memory) is read by every
// CTA on entry, a CTA that finds it set does no work; `host_flag` (mapped pinned host memory) is what the host
// reads after it has synchronised the stream; `limit` is the number of SM cycles one wait may take.  WaitCtl is
// the per-CTA copy in shared memory that the waits poll: `abort` is set by the first wait of the CTA that runs
// out (and, in a cluster pair, in the peer CTA's copy too, through `peer_abort`), every other role leaves at its
// next poll.
struct WaitCtl {
  int abort;             // 0, or the code of the wait that gave up first (kWait*), or kWaitPeer / kWaitEntry
  uint32_t peer_abort;   // shared::cluster address of the peer CTA's `abort`, 0 outside a cluster
  long long limit;
};
// Which wait ran out: the code travels to the host flag and into the error message (names: thc_general.cu).
enum : int {
  kWaitOther = 1, kWaitRawTile = 2, kWaitLoSlot = 3, kWaitAccEmpty = 4, kWaitTileFull = 5, kWaitSlotEmpty = 6,
  kWaitAccFull = 7, kWaitItemNumber = 8, kWaitItemGo = 9, kWaitItemSlot = 10, kWaitProbe = 11,
  kWaitEntry = 254, kWaitPeer = 255
};
__device__ __forceinline__ void wait_ctl_init(volatile WaitCtl *w, const StallCtl &ctl, uint32_t peer_abort = 0) {
  w->abort = *reinterpret_cast<volatile int *>(ctl.dev_flag) != 0 ? kWaitEntry : 0;
  w->peer_abort = peer_abort;
  w->limit = ctl.limit;
}
__device__ __forceinline__ void wait_ctl_give_up(volatile WaitCtl *w, int code = kWaitOther) {
  if (w->abort == 0) w->abort = code;
  const uint32_t peer = w->peer_abort;
  if (peer) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer), "r"((uint32_t)kWaitPeer) : "memory");
}
// What a CTA does before it leaves when any of its waits ran out (or it found the flag set on entry): `code` is its
// abort word.  The host flag keeps the code of a wait that ran out in preference to "the peer / an earlier kernel did".
__device__ __forceinline__ void stall_raise(const StallCtl &ctl, int code = kWaitOther) {
  atomicExch(ctl.dev_flag, 1);
  volatile int *host = reinterpret_cast<volatile int *>(ctl.host_flag);
  if ((code != kWaitEntry && code != kWaitPeer) || *host == 0) *host = code;
  __threadfence_system();
}
// Bounded wait.  Returns false when the phase did not complete within the limit (the CTA's abort word is then
// set to `code`) or another thread already gave up.
// `shift`: the wait may take 2^shift limits.  For waits that span a whole work item rather than one k tile (the item
// hand-out of the persistent engine): when the pipeline really stands still a k-tile wait runs out first and sets
// the abort word, which these waits poll too, so the longer allowance costs no detection time, and a long item
// (or a kernel slowed a few hundred times by a profiler's instrumentation) is not taken for a stall.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile WaitCtl *w, int code = kWaitOther,
                                          int shift = 0) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  int polls = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++polls & 15) == 0) {
      if (w->abort) return false;
      if (clock64() - t0 > (w->limit << shift)) { wait_ctl_give_up(w, code); return false; }
    }
  }
  return true;
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Operand tile descriptors.
//   K-major : rows (m or n) of 128 B = 32 k, 128-byte swizzle (16-byte chunk index XOR row % 8); 8-row groups
//             1024 B apart (stride offset); leading offset unused.
//   MN-major: rows are k, each 128 B = 32 consecutive m (or n); the tile is [32-wide block][32 k][128 B].  For
//             32-bit elements the tensor core reads this form with the "128-byte swizzle, 32-byte atom" mode:
//             32-byte granule index XOR k % 4, blocks along m / n 4096 B apart (leading offset), 4-k groups
//             512 B apart (stride offset).
template <bool MN_MAJOR>
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);               // start address
  d |= (uint64_t)(MN_MAJOR ? (4096 >> 4) : 1) << 16;          // leading byte offset
  d |= (uint64_t)((MN_MAJOR ? 512 : 1024) >> 4) << 32;        // stride byte offset
  d |= (uint64_t)1 << 46;                                     // descriptor version (Blackwell)
  d |= (uint64_t)(MN_MAJOR ? 1 : 2) << 61;                    // SWIZZLE_128B_BASE32B : SWIZZLE_128B
  return d;
}
// bytes between the operand slices of consecutive MMAs (8 k each)
template <bool MN_MAJOR> __host__ __device__ constexpr int umma_kstep_bytes() { return MN_MAJOR ? 1024 : 32; }
__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ void cp_async4(uint32_t dst, const float *src, const float *any_valid) {
  // 4-byte asynchronous global -> shared copy; a null source zero-fills the destination (src-size 0:
  // nothing is read, `any_valid` only keeps the address operand well-formed)
  const unsigned n = src ? 4u : 0u;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"((const void *)(src ? src : any_valid)), "r"(n) : "memory");
}
// 16 bytes, kept in L1 for the neighbours that read them again; `there` false: zeros, nothing is read
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool there) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------- cluster / cta_group::2 PTX
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on a barrier of any CTA of the cluster (address from mapa_shared).  Default (CTA-scope release)
// semantics on purpose: a cluster-scope release costs the arriving thread one to two thousand cycles here,
// and nothing these arrivals hand over travels through the generic proxy between the CTAs: shared-memory
// tiles are published to the async proxy by the producer's own fence.proxy.async, tensor memory by
// tcgen05.fence / tcgen05.wait::ld.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// One thread of a converged warp.  The tensor-core and TMA instructions take their descriptors, coordinates and barriers from registers
// that a warp has once.  A warp that runs its loop with all lanes on values that all of them share, and issues under this predicate, has
// them there; one thread alone (`lane == 0` around the loop, an election around the loop as well) pays for bringing them there
// with every instruction.  tcgen05.mma of a CTA pair back to back at 64, 128 and 192 columns: one every 107 cycles then, the cost of its issue, and
// every 46, 68 and 100 so; 256 columns, which the pipe itself bounds, take some 130 either way.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// Bounded busy wait for the warps that issue MMAs, all lanes of which poll: polling without suspension answers within a few
// cycles of the arrival, which is what keeps the tensor pipe fed.  A poll is one instruction of the warp, as it was of a lone thread.
__device__ __forceinline__ bool mbar_wait_spin(uint32_t bar, uint32_t parity, volatile WaitCtl *w, int code = kWaitOther) {
  long long t0 = 0;
  for (int polls = 0;; polls++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((polls & 255) == 255) {
      if (w->abort) return false;
      if (t0 == 0) t0 = clock64();
      else if (clock64() - t0 > w->limit) { wait_ctl_give_up(w, code); return false; }
    }
  }
}
__device__ __forceinline__ void tmem_alloc2(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma2_tf32(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// completion of all MMAs issued so far -> one arrival on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma2_commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// kind::tf32, FP32 accumulate, M = 256 over the CTA pair
__host__ __device__ constexpr uint32_t umma2_idesc_tf32(int n, bool a_mn, bool b_mn) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// im2col TMA load of 32 channels of 128 consecutive windows (tensor {C, W, H, images}) starting at window
// corner (x, y) of image `img`, at tap offset (j, i); completion as above.
__device__ __forceinline__ void tma_load_windows(uint32_t dst, const void *tmap, int c, int x, int y, int img, int j, int i,
                                                 uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.im2col.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
      ::"r"(dst), "l"((unsigned long long)tmap), "r"(mbar), "r"(c), "r"(x), "r"(y), "r"(img), "h"((unsigned short)j),
        "h"((unsigned short)i)
      : "memory");
}
template <int N> __device__ __forceinline__ void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t *v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// BF16 operand tiles: K-major as for TF32; MN-major [64-channel block][64 pixels][128 B], plain 128-byte
// swizzle, blocks 8192 B apart (leading offset), 8-pixel groups 1024 B apart (stride offset).
template <bool MN_MAJOR>
__device__ __forceinline__ uint64_t umma_desc_half(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)(MN_MAJOR ? (8192 >> 4) : 1) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;   // SWIZZLE_128B
  return d;
}
// bytes between the operand slices of consecutive MMAs (16 k each)
template <bool MN_MAJOR> __host__ __device__ constexpr int umma_kstep_bytes_half() { return MN_MAJOR ? 2048 : 32; }
// kind::f16 with BF16 operands, FP32 accumulate, M = 256 over the CTA pair
__host__ __device__ constexpr uint32_t umma2_idesc_bf16(int n, bool a_mn, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
}
// the same with FP16 operands
__host__ __device__ constexpr uint32_t umma2_idesc_f16(int n, bool a_mn, bool b_mn) {
  return (1u << 4) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
}
__device__ __forceinline__ void umma2_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// FP16 products on top of an accumulator of 2^11 times their unit: D = A * B + D * 2^-11
__device__ __forceinline__ void umma2_f16_scale11(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.eq.b32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p, 11;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc)
      : "memory");
}

}  // namespace mm
}  // namespace thc

#endif
