// PTX of kernels whose thread-block clusters are pairs of SMs that share one tcgen05.mma
// (cta_group::2): barriers and copies across the pair, tensor memory of the pair, a stage of MMAs.
#pragma once
#include "tc_common.cuh"

namespace ek {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The address of the same shared-memory place in block `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t own, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(own), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// A tile of this block's shared memory whose bytes complete on a barrier that may stand in the
// other block of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                                 uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// All MMAs issued so far by this thread: when they are done, one arrival on the barrier at this
// place in BOTH blocks of the pair.
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// One stage of the pair's product in one piece of PTX: ask the NEXT stage's barrier (test_wait: it
// answers at once and never suspends the thread, unlike try_wait), issue this stage's four MMAs (K = 16 each, 32 bytes further along the swizzled row), commit them to this stage's "empty"
// barrier in both blocks, and only then look at the barrier's answer - the thread does not wait for it
// before the MMAs are on their way.  Returns whether the next stage is full.
__device__ __forceinline__ uint32_t mma_stage_pair(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc,
                                                   uint32_t accumulate, uint32_t empty_bar, uint32_t next_full,
                                                   uint32_t next_parity) {
  uint32_t ready;
  asm volatile(
      "{\n\t.reg .pred p, q, t;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%8], %9;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "setp.eq.b32 t, %6, %6;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], %2, %3, %4, {%6, %6, %6, %6, %6, %6, %6, %6}, p;\n\t"
      "add.u64 %2, %2, 2;\n\tadd.u64 %3, %3, 2;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], %2, %3, %4, {%6, %6, %6, %6, %6, %6, %6, %6}, t;\n\t"
      "add.u64 %2, %2, 2;\n\tadd.u64 %3, %3, 2;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], %2, %3, %4, {%6, %6, %6, %6, %6, %6, %6, %6}, t;\n\t"
      "add.u64 %2, %2, 2;\n\tadd.u64 %3, %3, 2;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], %2, %3, %4, {%6, %6, %6, %6, %6, %6, %6, %6}, t;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%7], %10;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ready), "+r"(d_tmem), "+l"(da), "+l"(db)
      : "r"(idesc), "r"(accumulate), "r"(0u), "r"(empty_bar), "r"(next_full), "r"(next_parity), "h"((uint16_t)3)
      : "memory");
  return ready;
}

}  // namespace ek
