// Shared device helpers for the sm_100a kernels: mbarrier, TMA, tcgen05/TMEM wrappers and the
// bounded-wait protocol.  Every spin in these kernels has a time budget; a wait that runs out
// records a code in a global status word, raises a CTA-wide abort flag and lets every role fall
// through to the common teardown (where TMEM is released), so a protocol bug shows up as an error
// code on the host instead of a hung device.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace mfq {

// ----- status codes written to the global status word (0 = ok) -----
enum : int {
  kStatusOk = 0,
  kStatusTimeoutProducer = 1,
  kStatusTimeoutMma = 2,
  kStatusTimeoutEpilogue = 3,
  kStatusTimeoutPeer = 4,
  kStatusBadArgument = 5,
};

constexpr unsigned long long kWaitBudgetNs = 1500ull * 1000ull * 1000ull;  // 1.5 s per wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }

// ----- mbarrier -----
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
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

// Wait for `parity` of `bar` with a time budget.  Returns false (after recording `code`) when the
// budget runs out or when another role of this CTA already aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status,
                                          int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 0x3F) == 0) {
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > kWaitBudgetNs) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, code);
        return false;
      }
    }
  }
  return true;
}

// The same by a whole warp, with one answer for all its lanes: what follows stays warp-uniform for the compiler, which then
// keeps descriptors and addresses in uniform registers.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status, int code) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, code));
}
// Looks at a barrier without waiting (whole warp, one answer): asked one block ahead, its latency hides under the current block.
__device__ __forceinline__ bool mbar_test_warp(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return __all_sync(0xffffffffu, ok != 0);
}

// ----- TMA (bulk tensor copies; loads are never cluster-multicast) -----
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* desc) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(desc)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* desc, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(desc)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* desc, uint64_t* bar, int x, int y,
                                            int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(desc)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// A stage of two tiles whose bytes complete on `bar`: optionally arm the barrier and load the first tile (`with_a`), then load the
// second.  Whole warp, one elected lane issues (see umma_f8f6f4_block for why not `if (lane == 0)`).  `az` < 0: the first tensor
// is 2-D, else its third coordinate; `x`, `xb`: the tiles' innermost coordinates.
__device__ __forceinline__ void tma_load_stage(uint32_t smem_a, uint32_t smem_b, const CUtensorMap* map_a, const CUtensorMap* map_b,
                                               uint32_t bar, uint32_t bytes, bool with_a, int x, int ya, int az, int yb, int xb) {
  const uint64_t ma = reinterpret_cast<uint64_t>(map_a), mb = reinterpret_cast<uint64_t>(map_b);
  if (az < 0) {
    asm volatile(
        "{\n\t.reg .pred q, w;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.and.b32 w, %6, 0, q;\n\t"
        "@w mbarrier.arrive.expect_tx.shared::cta.b64 _, [%4], %5;\n\t"
        "@w cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%7, %8}], [%4];\n\t"
        "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%3, {%10, %9}], [%4];\n\t}"
        ::"r"(smem_a), "r"(smem_b), "l"(ma), "l"(mb), "r"(bar), "r"(bytes), "r"(uint32_t(with_a)), "r"(x), "r"(ya), "r"(yb), "r"(xb)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred q, w;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.and.b32 w, %6, 0, q;\n\t"
        "@w mbarrier.arrive.expect_tx.shared::cta.b64 _, [%4], %5;\n\t"
        "@w cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%2, {%7, %8, %10}], [%4];\n\t"
        "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%1], [%3, {%11, %9}], [%4];\n\t}"
        ::"r"(smem_a), "r"(smem_b), "l"(ma), "l"(mb), "r"(bar), "r"(bytes), "r"(uint32_t(with_a)), "r"(x), "r"(ya), "r"(yb), "r"(az), "r"(xb)
        : "memory");
  }
}
// Bulk store of a shared-memory tile (rows and columns beyond the tensor are left out), in the issuing thread's current group.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* desc, uint32_t smem_src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(desc)), "r"(smem_src), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }  // sources may be written again
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }             // ... and the stores are done
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----- programmatic dependent launch -----
// Kernels of the decode path are launched with the programmatic-serialization attribute: a kernel may be scheduled
// while its predecessor in the stream drains, run its prologue (barrier init, TMEM allocation, index math) and
// then block in pdl_wait() until the predecessor has completed and flushed its writes.  Such a kernel calls
// pdl_trigger() first thing, so its own successor may be scheduled as early as possible, unless it takes tensor memory: then behind the
// allocation (and the block barrier that publishes it).  The successors may allocate before they wait; were one resident while a CTA
// of this grid had still to allocate, it could take the columns that this CTA needs and wait, without end, for this grid.  Once all CTAs have
// triggered, all hold what they need, and a successor that finds too little waits for them, which end without it.
// Beside that, correctness only depends on pdl_wait() preceding the first access to memory another kernel produced (and the
// first global write).  Weights are apart: products and the small router request the first of them ahead of the wait.  No kernel here writes
// any; whoever changes weights in place on the stream of their product puts a launch without this attribute between the two.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ----- tcgen05 / TMEM -----
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {  // one thread; arrives when prior MMAs retire
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T, f16/bf16 inputs, fp32 accumulate.  One thread issues.
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// fp8/fp6/fp4 element kinds: one 128-byte K block, four k-steps of 32 bytes each into accumulator `d`, then a commit to each of up to
// two barriers (shared addresses; 0 = none) -- all issued by ONE elected lane of a warp that runs this converged.  A single lane inside
// `if (lane == 0)` needs 55 cycles per tcgen05 instruction on a B200 (every operand moves to a uniform register first), four
// MMAs and their commits 320; issued like this they need 160, below the 256 cycles the tensor core works on a 128 x 128 block.
// `accumulate` applies to the first step.
__device__ __forceinline__ void umma_f8f6f4_block(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate,
                                                  uint32_t bar0, uint32_t bar1) {
  asm volatile(
      "{\n\t.reg .pred q, f, t, u, v;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
      "setp.ne.b32 f, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.s64 a1, %1, 2;\n\tadd.s64 a2, %1, 4;\n\tadd.s64 a3, %1, 6;\n\t"
      "add.s64 b1, %2, 2;\n\tadd.s64 b2, %2, 4;\n\tadd.s64 b3, %2, 6;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.and.b32 u, %5, 0, q;\n\tsetp.ne.and.b32 v, %6, 0, q;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, f;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a1, b1, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a2, b2, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a3, b3, %3, t;\n\t"
      "@u tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%5];\n\t"
      "@v tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(bar0), "r"(bar1)
      : "memory");
}

// The 16-bit form: four k-steps of 16 values; the descriptors advance by kA, kB (16-byte units) from step to step.
template <int kA = 2, int kB = 2>
__device__ __forceinline__ void umma_f16_block(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate,
                                               uint32_t bar0 = 0, uint32_t bar1 = 0) {
  asm volatile(
      "{\n\t.reg .pred q, f, t, u, v;\n\t.reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
      "setp.ne.b32 f, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.s64 a1, %1, %7;\n\tadd.s64 a2, %1, %8;\n\tadd.s64 a3, %1, %9;\n\t"
      "add.s64 b1, %2, %10;\n\tadd.s64 b2, %2, %11;\n\tadd.s64 b3, %2, %12;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.and.b32 u, %5, 0, q;\n\tsetp.ne.and.b32 v, %6, 0, q;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, f;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, t;\n\t"
      "@u tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%5];\n\t"
      "@v tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(bar0), "r"(bar1), "n"(kA), "n"(2 * kA), "n"(3 * kA), "n"(kB),
        "n"(2 * kB), "n"(3 * kB)
      : "memory");
}
__device__ __forceinline__ void umma_f16_warp(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {  // a single k-step
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit_warp(uint64_t* bar) {  // whole warp, one elected lane; arrives when its prior MMAs retire
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}

// Instruction descriptor (dense, fp32 accumulate).  fmt: kind::f8f6f4 0 = E4M3, 1 = E5M2, 5 = E2M1;
// kind::f16 0 = F16, 1 = BF16.  major: 0 = K-major, 1 = MN-major.
__host__ __device__ constexpr uint32_t umma_idesc(int m, int n, int a_fmt, int b_fmt, int a_major = 0,
                                                  int b_major = 0) {
  return (1u << 4) | (uint32_t(a_fmt) << 7) | (uint32_t(b_fmt) << 10) | (uint32_t(a_major) << 15) |
         (uint32_t(b_major) << 16) | (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

// Shared-memory matrix descriptor for a K-major tile stored as rows of 128 bytes with the 128-byte
// swizzle (what a TMA load with CU_TENSOR_MAP_SWIZZLE_128B produces): 8-row groups are 1024 B apart.
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= uint64_t((smem_addr >> 4) & 0x3FFF);  // start address
  d |= uint64_t(1) << 16;                    // leading byte offset (unused for swizzled K-major): 1
  d |= uint64_t(1024 >> 4) << 32;            // stride byte offset between 8-row groups
  d |= uint64_t(1) << 46;                    // descriptor version (Blackwell)
  d |= uint64_t(2) << 61;                    // SWIZZLE_128B
  return d;
}
// MN-major tile with the 128-byte swizzle: the tile is [k][mn] with 64 16-bit mn-elements (128 B) per row
// chunk; `mn_chunk_stride` bytes separate 64-element mn chunks, 8 k-rows form one 1024 B group.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t mn_chunk_stride_bytes) {
  uint64_t d = 0;
  d |= uint64_t((smem_addr >> 4) & 0x3FFF);
  d |= uint64_t((mn_chunk_stride_bytes >> 4) & 0x3FFF) << 16;  // leading byte offset: next mn chunk
  d |= uint64_t(1024 >> 4) << 32;                              // stride byte offset: next 8 k-rows
  d |= uint64_t(1) << 46;
  d |= uint64_t(2) << 61;
  return d;
}

// 32 lanes x 32 columns of fp32 from TMEM: thread i of the warp gets row (lane base + i), 32 columns.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// ----- misc -----
// c += {a0, a1} * s, two fp32 multiply-adds in one instruction
__device__ __forceinline__ void fma2(float& c0, float& c1, uint32_t a0, uint32_t a1, float s) {
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %4};\n\tmov.b64 z, {%0, %1};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "+f"(c0), "+f"(c1)
      : "r"(a0), "r"(a1), "f"(s));
}
// Two fp32 operations per instruction, each rounded as by itself: {a, b} * s, {a, b} + {c, d}, {a0, a1} * {b0, b1} + {c0, c1}.
__device__ __forceinline__ void scale2(float& a, float& b, float s) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %2};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}" : "+f"(a), "+f"(b) : "f"(s));
}
__device__ __forceinline__ void add2(float& a, float& b, uint32_t c, uint32_t d) {
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}" : "+f"(a), "+f"(b) : "r"(c), "r"(d));
}
__device__ __forceinline__ float2 fma_f2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float bf16_to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

struct alignas(16) U4 { uint32_t x, y, z, w; };

}  // namespace mfq

// ----- host side: tensor maps through the driver entry point (no -lcuda link dependency) -----
#include <cstdio>
namespace mfq {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || !p) return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}
// 2-D row-major tensor [rows, cols] of `elem_bytes`-sized items, box = [box_rows, box_cols], 128-byte swizzle.
// Returns 0 on success.
inline int make_tmap_2d(CUtensorMap* out, const void* base, CUtensorMapDataType dt, int elem_bytes, uint64_t rows,
                        uint64_t cols, uint64_t row_stride_bytes, uint32_t box_rows, uint32_t box_cols,
                        CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_128B) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {row_stride_bytes};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  (void)elem_bytes;
  CUresult r = fn(out, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : int(r);
}
inline int make_tmap_3d(CUtensorMap* out, const void* base, CUtensorMapDataType dt, uint64_t d0, uint64_t d1,
                        uint64_t d2, uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1,
                        uint32_t b2, CUtensorMapSwizzle swz = CU_TENSOR_MAP_SWIZZLE_128B) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -1;
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
  cuuint32_t box[3] = {b0, b1, b2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(out, dt, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : int(r);
}
}  // namespace mfq


// Host side: launch with the programmatic-serialization attribute (MFQ_PDL=0 in the environment turns it off).
#include <cstdlib>
#include <utility>
namespace mfq {
inline bool pdl_enabled() {
  static const bool on = [] { const char* e = getenv("MFQ_PDL"); return !(e && e[0] == '0'); }();
  return on;
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                 Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
// The same with the grid cut into thread-block clusters of `cluster` CTAs (distributed shared memory among them).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel_clustered(void (*kernel)(KArgs...), dim3 grid, dim3 block, dim3 cluster, size_t smem,
                                           cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster.x;
  attr[0].val.clusterDim.y = cluster.y;
  attr[0].val.clusterDim.z = cluster.z;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
}  // namespace mfq
