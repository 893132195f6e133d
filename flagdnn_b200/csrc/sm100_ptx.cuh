// Thin inline-PTX wrappers for the sm_100a features the convolution kernels
// use: mbarrier, TMA (tiled and im2col tensor copies), tcgen05 (tensor memory
// allocation, MMA issue, commit, accumulator loads).  Every wait is bounded.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fdnn {

// Codes written into the per-device status word by a wait that ran out.
enum : uint32_t {
  kIncidentNone = 0,
  kIncidentProducerWait = 1,   // TMA producer: stage never freed
  kIncidentMmaWaitFull = 2,    // MMA issuer: stage never filled
  kIncidentMmaWaitTmem = 3,    // MMA issuer: accumulator never drained
  kIncidentEpilogueWait = 4,   // epilogue: accumulator never completed
  kIncidentDrainWait = 5,      // teardown: outstanding copies never landed
  kIncidentPartialWait = 6,    // epilogue of a split tile: another pair's partial sums never arrived
  kIncidentResidualWait = 7,   // epilogue: the residual box never landed in the staging buffer
  kIncidentDepthwiseWait = 8   // depthwise: an input row never landed in its ring slot
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}

// Shared-memory accesses by 32-bit shared address (staging buffers reached through an aligned-up base lose their
// address space in C++ and would be read through generic loads).
__device__ __forceinline__ uint16_t lds_u16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds_v2(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds_v4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_u16(uint32_t a, uint16_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(v) : "memory");
}
__device__ __forceinline__ void sts_u32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// 32 bytes to global memory in one store (32-byte aligned).
__device__ __forceinline__ void stg_v8(void* p, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void sts_v2(uint32_t a, uint2 v) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void sts_v4(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Tests whether the phase with the given parity has completed.  While it is still open the hardware may
// park the thread for up to kParkNs nanoseconds (it is woken when the phase completes) instead of
// returning at once: ten warps of a CTA re-polling their barriers every few dozen clocks cost enough
// power to lower the clock of a tensor-bound kernel by 5-9 % on B200 (measured: 50.0 -> 45.8 us on the
// 3x3 256-channel layer; hints from 0.25 to 8 us measure the same).
#ifndef FDNN_PARKED_WAIT_NS
#define FDNN_PARKED_WAIT_NS 2000
#endif
constexpr uint32_t kParkNs = FDNN_PARKED_WAIT_NS;

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  if constexpr (kParkNs > 0) {
    asm volatile(
        "{\n\t"
        ".reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(kParkNs)
        : "memory");
  } else {
    asm volatile(
        "{\n\t"
        ".reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
  }
  return ok != 0;
}

// The same without the suspend-time hint: for a role on the critical path that expects the phase to be complete (the
// hint costs some 30 clocks even then).
__device__ __forceinline__ bool mbar_try_wait_now(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  Gives up after `limit_cycles` SM clocks (about 2 s by
// default) or as soon as another role raised `*abort_flag`; on giving up it
// records `incident` in the device status word and raises the flag itself, so
// every role leaves its loop and the CTA tears down normally.
constexpr long long kWaitLimitCycles = 4000000000LL;

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  volatile uint32_t* abort_flag,
                                                  uint32_t* status_word, uint32_t incident,
                                                  long long limit_cycles = kWaitLimitCycles) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++spins & 0xf) == 0) {  // a parked poll lasts up to kParkNs, so this is still rare
      if (*abort_flag) return false;
      if (clock64() - t0 > limit_cycles) {
        atomicCAS(status_word, 0u, incident);
        *abort_flag = 1;
        __threadfence_block();
        return false;
      }
    }
  }
}

// The wait of a whole warp: every lane gets the same answer.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag,
                                               uint32_t* status_word, uint32_t incident, long long limit_cycles) {
  if (__all_sync(0xffffffffu, mbar_try_wait_now(bar, parity))) return true;
  const bool ok = mbar_wait_bounded(bar, parity, abort_flag, status_word, incident, limit_cycles);
  return __all_sync(0xffffffffu, ok);
}

// ------------------------------------------- programmatic dependent launch
// A kernel launched with the programmatic-stream-serialization attribute may
// start while the kernel before it on the stream is still draining.  It runs
// its set-up (barriers, tensor memory, descriptor prefetch), then blocks in
// griddep_wait() until that kernel has completed and its writes are visible;
// nothing before the wait may touch global memory.  griddep_launch_dependents()
// in the earlier kernel says that the next one may be scheduled as soon as
// every CTA of this grid has issued it (or exited); without it the trigger
// fires when the grid completes, which is ordinary stream order.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ------------------------------------------------- register reallocation
// The register file is handed out per warp group (four consecutive warps).  A group whose roles need
// few registers gives some back, the others take them; every warp of a group executes the same call.
template <int kRegs>
__device__ __forceinline__ void warpgroup_reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegs));
}
template <int kRegs>
__device__ __forceinline__ void warpgroup_reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegs));
}

// --------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* tm) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tm)) : "memory");
}

// Asks for a 3-D box of a tensor to be brought into L2; nothing lands in shared memory and nothing waits.
__device__ __forceinline__ void tma_prefetch_l2_3d(const CUtensorMap* tm, int32_t c0, int32_t c1, int32_t c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];"
               :
               : "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

// Tiled 3-D tensor copy global -> shared of this CTA, completion on `bar`.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* tm, uint64_t* bar,
                                            int32_t c0, int32_t c1, int32_t c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(c0),
        "r"(c1), "r"(c2)
      : "memory");
}

// Tiled 4-D tensor copy global -> shared of this CTA.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* tm, uint64_t* bar,
                                            int32_t c0, int32_t c1, int32_t c2, int32_t c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(c0),
        "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// Im2col-mode 4-D tensor copy (C, W, H, N): starts at base pixel (w, h, n) of
// the descriptor's bounding box, walks pixelsPerColumn pixels through W, H, N,
// and reads each at the filter-tap offset (off_w, off_h).  Out-of-range
// elements arrive as zero, which implements the convolution's padding.
__device__ __forceinline__ void tma_load_im2col_4d(void* smem_dst, const CUtensorMap* tm,
                                                   uint64_t* bar, int32_t c, int32_t w, int32_t h,
                                                   int32_t n, uint16_t off_w, uint16_t off_h) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(c),
        "r"(w), "r"(h), "r"(n), "h"(off_w), "h"(off_h)
      : "memory");
}

// The same over five dimensions (C, W, H, D, N), for grouped layers: D holds the images (the walk of pixelsPerColumn
// pixels goes through W, H, D), N the group.
__device__ __forceinline__ void tma_load_im2col_5d(void* smem_dst, const CUtensorMap* tm, uint64_t* bar, int32_t c,
                                                   int32_t w, int32_t h, int32_t d, int32_t n, uint16_t off_w,
                                                   uint16_t off_h) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6, %7}], [%2], {%8, %9, %10};"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar)), "r"(c),
        "r"(w), "r"(h), "r"(d), "r"(n), "h"(off_w), "h"(off_h), "h"(static_cast<uint16_t>(0))
      : "memory");
}

// Tiled 2-D tensor store shared -> global (bulk-group completion).  Rows or
// columns of the box that fall outside the tensor are not written.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tm, const void* smem_src, int32_t c0,
                                             int32_t c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* tm, const void* smem_src, int32_t c0,
                                             int32_t c1, int32_t c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               :
               : "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void bulk_commit_group() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// Waits until the bulk stores committed so far have finished READING shared memory.
__device__ __forceinline__ void bulk_wait_group_read0() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// Same, but lets the most recent group keep reading (two staging buffers in rotation).
__device__ __forceinline__ void bulk_wait_group_read1() {
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}
// Waits until the bulk stores committed so far are complete.
__device__ __forceinline__ void bulk_wait_group0() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// Makes this thread's shared-memory writes visible to the async (TMA) proxy.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Untiled bulk copies: global -> shared of this CTA with completion on an mbarrier, and shared -> global as
// part of the thread's bulk group.  Both addresses 16-byte aligned, the size a multiple of 16 bytes.
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :
               : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(gmem_src)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store_1d(void* gmem_dst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               :
               : "l"(reinterpret_cast<uint64_t>(gmem_dst)), "r"(smem_u32(smem_src)), "r"(bytes)
               : "memory");
}

// Same for writes to global memory that a later tensor copy of this CTA reads (all state spaces).
__device__ __forceinline__ void fence_proxy_async_all() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

// Shared-memory matrix descriptor for a K-major operand tile whose rows are
// 128 bytes wide and stored with the 128-byte swizzle (what a TMA box with
// CU_TENSOR_MAP_SWIZZLE_128B produces): 8-row groups are 1024 bytes apart.
//   bits [0,14)  start address >> 4
//   bits [16,30) leading byte offset >> 4 (unused for swizzled K-major; 1)
//   bits [32,46) stride byte offset >> 4  (1024 >> 4 = 64)
//   bits [46,48) descriptor version (1 on sm_100)
//   bits [61,64) layout type (2 = SWIZZLE_128B)
// The high word is a constant of the layout, the low word names the place.
constexpr uint32_t kSw128DescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
// ... of K-major rows of 64 and 32 bytes in the swizzle of that width (eight rows take 512 and 256 bytes)
constexpr uint32_t kSw64DescHi = (512u >> 4) | (1u << 14) | (4u << 29), kSw32DescHi = (256u >> 4) | (1u << 14) | (6u << 29);
__device__ __forceinline__ uint32_t sw128_desc_lo(uint32_t smem_addr) { return (smem_addr >> 4) | (1u << 16); }

// The same for an operand stored MN-major (its rows run along M or N, one reduction element each): boxes of 64 M/N
// elements (128 bytes) x 64 reduction rows, 128-byte swizzle, one after another.  Eight reduction rows take 1024 bytes
// (stride byte offset), the next 64 M/N elements are one 8192-byte box further (leading byte offset); an MMA's 16
// reduction elements take 2048 bytes.  The instruction descriptor says so with kIdescBMnMajor.
// The high word of the descriptor is that of the K-major form.
constexpr uint32_t kMnBoxElems = 64, kMnBoxBytes = 8192, kMnStepBytes = 2048;
__device__ __forceinline__ uint32_t mnmajor_desc_lo(uint32_t smem_addr) { return (smem_addr >> 4) | (kMnBoxBytes >> 4) << 16; }
constexpr uint32_t kIdescBMnMajor = 1u << 16;

// ----------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Arrives once on `bar` when every MMA issued so far by this thread is done.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

// 32 consecutive fp32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ------------------------------------------------- CTA pairs (cta_group::2)
// Two CTAs of one cluster cooperate on a 256-row tile: each stages its own 128
// rows of A and its own half of B; the leader (cluster rank 0) issues MMAs that
// read both CTAs' shared memory and write both CTAs' tensor memory.  Every
// load below is per-CTA: nothing is broadcast between CTAs.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of `local_smem_addr` as seen in CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The same without ordering this thread's earlier global stores for the whole cluster: a release at cluster scope waits
// until they are performed.  For hand-overs of tensor memory, which tcgen05 fences order.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Pair forms of the copies: data lands in THIS CTA's shared memory, the
// completion bytes are credited to the mbarrier at `bar_cluster_addr`, which
// may live in the partner CTA (the leader's "stage full" barrier).
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* tm,
                                                 uint32_t bar_cluster_addr, int32_t c0, int32_t c1,
                                                 int32_t c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cluster_addr), "r"(c0),
        "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(void* smem_dst, const CUtensorMap* tm,
                                                 uint32_t bar_cluster_addr, int32_t c0, int32_t c1,
                                                 int32_t c2, int32_t c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cluster_addr), "r"(c0),
        "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_load_im2col_4d_pair(void* smem_dst, const CUtensorMap* tm,
                                                        uint32_t bar_cluster_addr, int32_t c, int32_t w,
                                                        int32_t h, int32_t n, uint16_t off_w,
                                                        uint16_t off_h) {
  asm volatile(
      "cp.async.bulk.tensor.4d.im2col.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cluster_addr), "r"(c),
        "r"(w), "r"(h), "r"(n), "h"(off_w), "h"(off_h)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// Arrives once on the mbarrier at `bar_cluster_addr` (own or partner CTA) when
// every pair MMA issued so far by this thread is done.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar_cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar_cluster_addr)
               : "memory");
}
// The same arrival on the barrier at this offset in both CTAs of the pair.
__device__ __forceinline__ void tc_commit_both(uint32_t bar_addr) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar_addr),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
// Four MMAs D[tmem] (+)= A[smem] * B[smem] (kind::f16 covers f16 and bf16) over 64 reduction elements, from the low words of the two descriptors (the high word is the same for both):
// `acc0` of the first, the others add; the operands advance by 2 and kBStep descriptor units.  What the issuing thread does
// between two MMAs bounds narrow tiles, so that the descriptors are put together in place.
#define FDNN_MMA4(GROUP)                                        \
  asm volatile(                                                 \
      "{\n\t"                                                   \
      ".reg .pred p, q;\n\t"                                    \
      ".reg .b64 a, b;\n\t"                                     \
      ".reg .b32 x, y;\n\t"                                     \
      "setp.ne.b32 p, %5, 0;\n\t"                               \
      "setp.eq.b32 q, 0, 0;\n\t"                                \
      "mov.b64 a, {%1, %3};\n\t"                                \
      "mov.b64 b, {%2, %3};\n\t"                                \
      "tcgen05.mma." GROUP ".kind::f16 [%0], a, b, %4, p;\n\t"  \
      "add.u32 x, %1, 2;\n\t"                                   \
      "add.u32 y, %2, %6;\n\t"                                  \
      "mov.b64 a, {x, %3};\n\t"                                 \
      "mov.b64 b, {y, %3};\n\t"                                 \
      "tcgen05.mma." GROUP ".kind::f16 [%0], a, b, %4, q;\n\t"  \
      "add.u32 x, %1, 4;\n\t"                                   \
      "add.u32 y, %2, %7;\n\t"                                  \
      "mov.b64 a, {x, %3};\n\t"                                 \
      "mov.b64 b, {y, %3};\n\t"                                 \
      "tcgen05.mma." GROUP ".kind::f16 [%0], a, b, %4, q;\n\t"  \
      "add.u32 x, %1, 6;\n\t"                                   \
      "add.u32 y, %2, %8;\n\t"                                  \
      "mov.b64 a, {x, %3};\n\t"                                 \
      "mov.b64 b, {y, %3};\n\t"                                 \
      "tcgen05.mma." GROUP ".kind::f16 [%0], a, b, %4, q;\n\t"  \
      "}\n"                                                     \
      :                                                         \
      : "r"(d_tmem), "r"(a_lo), "r"(b_lo), "n"(kSw128DescHi), "r"(idesc), "r"(acc0), "n"(kBStep), "n"(2 * kBStep), "n"(3 * kBStep) \
      : "memory")
template <int kBStep = 2>
__device__ __forceinline__ void mma4_f16(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc0) {
  FDNN_MMA4("cta_group::1");
}
template <int kBStep = 2>
__device__ __forceinline__ void mma4_f16_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc0) {
  FDNN_MMA4("cta_group::2");
}
#undef FDNN_MMA4

// One MMA of a CTA pair, from the low words of its descriptors and their constant high words.
template <uint32_t kAHi, uint32_t kBHi>
__device__ __forceinline__ void mma_f16_pair_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      ".reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 a, {%1, %3};\n\t"
      "mov.b64 b, {%2, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %5, p;\n\t"
      "}\n"
      :
      : "r"(d_tmem), "r"(a_lo), "r"(b_lo), "n"(kAHi), "n"(kBHi), "r"(idesc), "r"(acc)
      : "memory");
}

// fp32 operands as TF32: low descriptor words of K-major rows in the 128-byte swizzle.  kPair: a CTA pair.
template <bool kPair = false>
__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
#define FDNN_MMA_TF32(GROUP)                                                                                      \
  asm volatile(                                                                                                   \
      "{\n\t"                                                                                                     \
      ".reg .pred p;\n\t"                                                                                         \
      ".reg .b64 a, b;\n\t"                                                                                       \
      "setp.ne.b32 p, %5, 0;\n\t"                                                                                 \
      "mov.b64 a, {%1, %3};\n\t"                                                                                  \
      "mov.b64 b, {%2, %3};\n\t"                                                                                  \
      "tcgen05.mma." GROUP ".kind::tf32 [%0], a, b, %4, p;\n\t"                                                   \
      "}\n"                                                                                                       \
      :                                                                                                           \
      : "r"(d_tmem), "r"(a_lo), "r"(b_lo), "n"(kSw128DescHi), "r"(idesc), "r"(acc)                                \
      : "memory")
  if constexpr (kPair) FDNN_MMA_TF32("cta_group::2");
  else FDNN_MMA_TF32("cta_group::1");
#undef FDNN_MMA_TF32
}

// Instruction descriptor: fp32 accumulate, both operands K-major, dense.
//   bits [4,6) D format (1 = f32); [7,10) A format; [10,13) B format
//   (0 = f16, 1 = bf16, 2 = tf32); bit 15/16 A/B major (0 = K);
//   bits [17,23) N >> 3; bits [24,29) M >> 4.
__host__ __device__ constexpr uint32_t make_idesc(uint32_t ab_format, uint32_t m, uint32_t n) {
  return (1u << 4) | (ab_format << 7) | (ab_format << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

}  // namespace fdnn
