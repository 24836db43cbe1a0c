// CTA pairs (clusters of two) working on one tile with `tcgen05.mma.cta_group::2`: what the two-SM products share.
#pragma once

#include "common.cuh"

namespace mfq {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(const void* smem_ptr, uint32_t cta) {  // cluster address of a peer's variable
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(smem_ptr)), "r"(cta));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {  // one warp in EACH CTA of the pair
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// One stage: the weight tile and the token half-tile, both completing on the barrier at `bar_cluster_addr` (the leader's, from
// either CTA), which the leader arms with `bytes` (0: the peer's call, it does not arm).  Whole warp, one elected lane issues.
__device__ __forceinline__ void tma_load_stage_pair(uint32_t smem_a, uint32_t smem_b, const CUtensorMap* map_a, const CUtensorMap* map_b,
                                                    uint32_t bar_cluster_addr, uint32_t bar_local, uint32_t bytes, int x, int ya, int yb) {
  asm volatile(
      "{\n\t.reg .pred q, e;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.and.b32 e, %6, 0, q;\n\t"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%5], %6;\n\t"
      "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%7, %8}], [%4];\n\t"
      "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%3, {%7, %9}], [%4];\n\t}"
      ::"r"(smem_a), "r"(smem_b), "l"(reinterpret_cast<uint64_t>(map_a)), "l"(reinterpret_cast<uint64_t>(map_b)), "r"(bar_cluster_addr),
        "r"(bar_local), "r"(bytes), "r"(x), "r"(ya), "r"(yb)
      : "memory");
}
// One tile of a stage, likewise.
__device__ __forceinline__ void tma_load_pair(uint32_t smem, const CUtensorMap* map, uint32_t bar_cluster_addr, uint32_t bar_local, uint32_t bytes, int x,
                                              int y) {
  asm volatile(
      "{\n\t.reg .pred q, e;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.and.b32 e, %4, 0, q;\n\t"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %4;\n\t"
      "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%5, %6}], [%2];\n\t}"
      ::"r"(smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(bar_local), "r"(bytes), "r"(x), "r"(y)
      : "memory");
}
// Relaxed: what it orders are tensor-memory reads, which have completed (wait::ld, fence::before_thread_sync) before it; a
// release at cluster scope would also drain this warp's global accesses, about a microsecond per block.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

__device__ __forceinline__ void mbar_arrive_cluster_warp(uint32_t bar_cluster_addr) {  // whole warp, one elected lane, no branch
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t@q mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n\t}" ::"r"(bar_cluster_addr)
               : "memory");
}

// Four k-steps of 32 bytes into accumulator `d`, then up to two commits (shared addresses; 0 = none), each of which arrives on the
// barrier at that offset in BOTH CTAs once these MMAs have retired.  Whole warp of the leader, one elected lane issues.
#define MFQ_UMMA_BLOCK_PAIR(NAME, KIND)                                                                                              \
  __device__ __forceinline__ void NAME(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t bar0,       \
                                       uint32_t bar1) {                                                                              \
    asm volatile(                                                                                                                    \
        "{\n\t.reg .pred q, f, t, u, v;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t.reg .b16 both;\n\tmov.b16 both, 3;\n\t"               \
        "setp.ne.b32 f, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"                                                                          \
        "add.s64 a1, %1, 2;\n\tadd.s64 a2, %1, 4;\n\tadd.s64 a3, %1, 6;\n\t"                                                       \
        "add.s64 b1, %2, 2;\n\tadd.s64 b2, %2, 4;\n\tadd.s64 b3, %2, 6;\n\t"                                                       \
        "elect.sync _|q, 0xffffffff;\n\t"                                                                                            \
        "setp.ne.and.b32 u, %5, 0, q;\n\tsetp.ne.and.b32 v, %6, 0, q;\n\t"                                                           \
        "@q tcgen05.mma.cta_group::2.kind::" KIND " [%0], %1, %2, %3, f;\n\t"                                                        \
        "@q tcgen05.mma.cta_group::2.kind::" KIND " [%0], a1, b1, %3, t;\n\t"                                                        \
        "@q tcgen05.mma.cta_group::2.kind::" KIND " [%0], a2, b2, %3, t;\n\t"                                                        \
        "@q tcgen05.mma.cta_group::2.kind::" KIND " [%0], a3, b3, %3, t;\n\t"                                                        \
        "@u tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%5], both;\n\t"                \
        "@v tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%6], both;\n\t}"               \
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(bar0), "r"(bar1)                                                  \
        : "memory");                                                                                                                 \
  }
MFQ_UMMA_BLOCK_PAIR(umma_f8f6f4_block_pair, "f8f6f4")
MFQ_UMMA_BLOCK_PAIR(umma_f16_block_pair, "f16")
#undef MFQ_UMMA_BLOCK_PAIR

}  // namespace mfq
