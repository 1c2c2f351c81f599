// Helpers of the kernels that run on CTA pairs (tcgen05 cta_group::2).
#pragma once
#include "cluster.cuh"
#include "common.cuh"

namespace flyb200 {

__device__ __forceinline__ void tmem_alloc2(uint32_t dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// completion of all MMAs issued so far -> one arrival on a barrier of the issuing (leader) CTA; the
// leader's relay thread passes it on to the peer
__device__ __forceinline__ void tc_commit2(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_f8_2(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t"
      "}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One arrival on an mbarrier of another CTA of the cluster. Relaxed: the arriving threads publish no
// data of their own (they pass on a completion they have observed on a local barrier); with release
// semantics at cluster scope each such arrival took ~700-900 cycles and was the bottleneck of the loop.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t local_bar, uint32_t rank) {
  const uint32_t remote = map_to_cta(local_bar, rank);
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
// Predicated, relaxed, on a barrier given by its cluster address.
__device__ __forceinline__ void mbar_arrive_cluster_if(uint32_t bar, bool pred) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "@p mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n\t"
      "}" ::"r"(bar),
      "r"(static_cast<uint32_t>(pred))
      : "memory");
}
// Three queries in flight together; the first two are answered as one, the third through `third`.
__device__ __forceinline__ bool mbar_test_2_1(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1,
                                              uint32_t bar2, uint32_t parity2, bool& third) {
  uint32_t ok, ok2;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q, r;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%2], %3;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 q, [%4], %5;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 r, [%6], %7;\n\t"
      "and.pred p, p, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "selp.u32 %1, 1, 0, r;\n\t"
      "}"
      : "=r"(ok), "=r"(ok2)
      : "r"(bar0), "r"(parity0), "r"(bar1), "r"(parity1), "r"(bar2), "r"(parity2)
      : "memory");
  third = ok2 != 0;
  return ok != 0;
}
// The same completion -> one arrival on the barrier at this offset in BOTH CTAs of the pair.
__device__ __forceinline__ void tc_commit2_both(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}

}  // namespace flyb200
