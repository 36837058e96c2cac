// sdg_tc_ptx.cuh -- inline-PTX building blocks of the tcgen05 kernels
// (sdg_dense_tc.cu, sdg_sparse_tc.cu): mbarriers with bounded waits, TMA tile
// loads, shared-memory matrix descriptors, UMMA issue / commit and TMEM loads.
//
// Every wait is bounded by WAIT_NS of %globaltimer: a wait that runs out sets
// *status, raises the CTA's abort flag and returns false, so that a kernel
// never spins forever; the kernels then drain their own copies and MMAs,
// free TMEM and return.
#pragma once

#include <cuda.h>
#include <cstdint>

namespace sdg {
namespace tc {

constexpr uint64_t WAIT_NS = 1000000000ull;    // 1 s per wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint64_t gtimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// try_wait with a suspend-time hint: the thread sleeps until the phase
// completes or about `ns` nanoseconds pass, instead of spinning on the issue
// slots that the warps sharing its scheduler need.
__device__ __forceinline__ bool mbar_try_wait_sleep(uint64_t* bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}
constexpr uint32_t SLEEP_NS = 20000;

// Bounded wait for the phase of the given parity; false when it ran out or the
// CTA aborted (then *abort_flag is set).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          int* status) {
  if (mbar_try_wait(bar, parity)) return true;
  uint64_t t0 = 0;                           // read after a while only: %globaltimer is slow
  for (uint32_t spin = 1;; ++spin) {
    if (mbar_try_wait_sleep(bar, parity, SLEEP_NS)) return true;
    if ((spin & 255u) == 0) {
      if (*abort_flag) return false;
      if (!t0) t0 = gtimer();
      if (gtimer() - t0 > WAIT_NS) {
        *abort_flag = 1;
        atomicExch(status, 1);
        return false;
      }
    }
  }
}
// Waits (bounded, without raising anything) for a phase that work already
// issued will complete: the drain before a CTA exits.
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
  const uint64_t t0 = gtimer();
  while (!mbar_try_wait_sleep(bar, parity, SLEEP_NS) && gtimer() - t0 < WAIT_NS) {}
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
// the same from a four-dimensional map
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z,
                                            int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)map) : "memory");
}
__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Shared-memory matrix descriptor of a K-major SWIZZLE_128B tile: rows of 128
// bytes, 8-row (1024-byte) swizzle atoms stacked at SBO = 1024; LBO is unused
// for swizzled K-major operands; version 1 (bits 46-47); layout 2 = 128B
// swizzle (bits 61-63).  The tile base is 1024-byte aligned, so the base
// offset (bits 49-51) is 0; a K step of 16 16-bit elements advances the start
// by 32 B.
// As two words, so that a K step or another tile is one 32-bit addition to the
// low one (the start address, below 2^14 units of 16 bytes).
__device__ __forceinline__ uint32_t sw128_desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
constexpr uint32_t SW128_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
// One lane of the (converged) warp, the same at every call.  A loop that issues
// MMAs runs in the whole warp and only the instructions themselves are
// predicated: addresses and descriptors then stay in uniform registers.  Inside an
// `if (lane == 0)` each tcgen05.mma cost its warp 70 cycles of operand moves, and
// issuing, not the tensor pipe, set the pace.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// Instruction descriptor of kind::f16 with FP32 accumulation (bits 4-5 = 1),
// A and B of one 16-bit type (bits 7-9 and 10-12: 0 = FP16, 1 = BF16), both
// K-major (bits 15, 16 = 0), N >> 3 at bits 17-22, M >> 4 at bits 24-28.
constexpr uint32_t idesc_f16(int m, int n, bool bf16) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
// alo, blo: the descriptors' low words (sw128_desc_lo)
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t idesc,
                                            uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 a, {%1, %5};\n\t"
      "mov.b64 b, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(idesc), "r"(accum), "r"(SW128_DESC_HI)
      : "memory");
}
// Arrives on bar once every MMA this thread issued before has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
               ::"r"(smem_u32(bar))
               : "memory");
}
// ---- CTA pairs (cta_group::2): the two CTAs of a cluster of two share one
// UMMA of M = 256 (rows 0-127 of A and D in the even CTA, 128-255 in the odd
// one) whose N columns of B are split between their shared memories; every
// tcgen05 instruction of such a kernel uses cta_group::2.
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// every thread of both CTAs: orders what each did before against what
// either does after (shared memory and barrier initialisation included)
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the shared::cluster address of bar's offset in CTA `cta` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t cta) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(cta));
  return a;
}
// arrive on the barrier at the same shared-memory offset in CTA `cta` of the cluster
__device__ __forceinline__ void mbar_arrive_remote(uint64_t* bar, uint32_t cta) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr(bar, cta)) : "memory");
}
// A tile load into this CTA's shared memory whose completion is counted on
// the barrier at bar_cluster, a shared::cluster address in either CTA of the
// pair (the pair's MMA waits on the even CTA's barriers).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster, int x,
                                                 int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, "
      "%3}], [%4];"
      ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar_cluster)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster, int x,
                                                 int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, "
      "%3, %4, %5}], [%6];"
      ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar_cluster)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t idesc,
                                                 uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 a, {%1, %5};\n\t"
      "mov.b64 b, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(idesc), "r"(accum), "r"(SW128_DESC_HI)
      : "memory");
}
// Arrives on the barrier at bar's offset in every CTA of `mask` once every
// MMA this thread issued before has completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"(mask)
               : "memory");
}
// executed by one warp in each CTA of the pair
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// 32 consecutive accumulator columns of this thread's lane; the wait carries
// the registers as operands so that no use is scheduled before it
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
#define SDG_R8(o) "=r"(v[o]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]), "=r"(v[o + 4]), "=r"(v[o + 5]), \
                  "=r"(v[o + 6]), "=r"(v[o + 7])
#define SDG_P8(o) "+r"(v[o]), "+r"(v[o + 1]), "+r"(v[o + 2]), "+r"(v[o + 3]), "+r"(v[o + 4]), "+r"(v[o + 5]), \
                  "+r"(v[o + 6]), "+r"(v[o + 7])
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : SDG_R8(0), SDG_R8(8), SDG_R8(16), SDG_R8(24)
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" : SDG_P8(0), SDG_P8(8), SDG_P8(16), SDG_P8(24) :: "memory");
#undef SDG_R8
#undef SDG_P8
}

// tmem_ld32 in two halves, so that the next chunk's load is in flight while
// the current one is processed: the issue writes v, the wait (which waits for
// every load this thread issued) carries v as operands so that no use of v is
// scheduled before it.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&v)[32]) {
#define SDG_R8(o) "=r"(v[o]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]), "=r"(v[o + 4]), "=r"(v[o + 5]), \
                  "=r"(v[o + 6]), "=r"(v[o + 7])
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : SDG_R8(0), SDG_R8(8), SDG_R8(16), SDG_R8(24)
      : "r"(taddr));
#undef SDG_R8
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&v)[32]) {
#define SDG_P8(o) "+r"(v[o]), "+r"(v[o + 1]), "+r"(v[o + 2]), "+r"(v[o + 3]), "+r"(v[o + 4]), "+r"(v[o + 5]), \
                  "+r"(v[o + 6]), "+r"(v[o + 7])
  asm volatile("tcgen05.wait::ld.sync.aligned;" : SDG_P8(0), SDG_P8(8), SDG_P8(16), SDG_P8(24) :: "memory");
#undef SDG_P8
}

}  // namespace tc
}  // namespace sdg
