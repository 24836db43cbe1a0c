// 4-bit weight streaming for up to 16 tokens:  out[t, n] = sum_k x[t, k] * w[n, k] (+ residual), weights in the layout of w4_gemm.cu.
//
// A decode step of a few tokens reads every weight once, so the time to beat is 0.625 bytes per weight at the memory's rate.  The
// tcgen05 form decodes into shared memory for the tensor core and is bound there by that hand-over (28672 x 4096: 62 us whatever the
// batch, 1.2 TB/s); here the codes go from memory into registers, through the same decode (w4_decode.cuh) and straight into
// mma.sync.m16n8k16 fragments.
//
// A CTA owns 16 weight rows, its eight warps take alternate steps of 128 inputs.  In a step a thread holds 32 consecutive codes (16
// bytes) of rows g and g + 8; the four threads of a row cover two K blocks of 64 (32 bytes of a row are contiguous, eight rows 256).
// The MMA's sums do not care which input sits in which k slot as long as both operands agree, so a word of eight codes is the thread's
// share of two MMAs, against the same eight values of x.  Four steps are in flight per thread: 128 bytes of codes, requested before the
// programmatic-launch wait for the first four.  The eight partial sums of an output meet in shared memory in warp order.
#include "w4_decode.cuh"

namespace mfq {

struct W4GemvParams {
  const uint8_t* packed;   // [n_tiles][k_blocks][128 rows][32 B]
  const uint32_t* group;   // [n_tiles][groups][128 rows]
  const __nv_bfloat16* x;  // [M, K]
  __nv_bfloat16* out;      // [M, N]
  const __nv_bfloat16* residual;
  int M, N, K, groups, words_per_group;
};

__device__ __forceinline__ void w4_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: blocks of 8 tokens.  WHOLE: a thread's 32 codes lie in one group (group size a multiple of 32).
template <int NT, int KIND, bool WHOLE>
__global__ void __launch_bounds__(256, 2) w4_gemv_kernel(const W4GemvParams p) {
  pdl_trigger();
  constexpr int kRing = 4;
  __shared__ float red[8][16][8 * NT + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int n0 = blockIdx.x * 16, blocks = p.K / 64, steps = (blocks + 1) / 2;
  const int block_in_step = t4 >> 1, half = t4 & 1;
  const uint8_t* codes = p.packed + size_t(n0 >> 7) * blocks * 4096 + ((n0 & 127) + g) * 32 + half * 16;
  const uint32_t* params = p.group + size_t(n0 >> 7) * p.groups * 128 + (n0 & 127) + g;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 wa[kRing], wb[kRing];     // rows g and g + 8
  uint32_t ga[kRing], gb[kRing];  // their group parameters (WHOLE); zero parameters make the codes of a missing block zero weights
  auto fetch = [&](int step, int j) {
    const int block = step * 2 + block_in_step;
    const bool live = block < blocks;
    wa[j] = live ? __ldcs(reinterpret_cast<const uint4*>(codes + size_t(block) * 4096)) : zero;
    wb[j] = live ? __ldcs(reinterpret_cast<const uint4*>(codes + size_t(block) * 4096 + 256)) : zero;
    if (WHOLE) {
      const uint32_t* at = params + (block * 8 + half * 4) / p.words_per_group * 128;
      ga[j] = live ? __ldcs(at) : 0u;
      gb[j] = live ? __ldcs(at + 8) : 0u;
    }
  };
#pragma unroll
  for (int j = 0; j < kRing; ++j) fetch(warp + 8 * j, j);
  pdl_wait();
  const __nv_bfloat16* xr[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) xr[nt] = p.x + size_t(min(nt * 8 + g, p.M - 1)) * p.K + block_in_step * 64 + half * 32;
  // the output of this thread, and what it is added to: requested under the product instead of after it
  const int t = threadIdx.x >> 4, row = threadIdx.x & 15, n = n0 + row;
  const bool mine = t < p.M && t < 8 * NT && n < p.N;
  const size_t at = size_t(t) * p.N + n;
  const float add = mine && p.residual ? __bfloat162float(p.residual[at]) : 0.f;
  float acc[NT][4] = {};
  for (int s0 = warp; s0 < steps; s0 += 8 * kRing) {
#pragma unroll
    for (int j = 0; j < kRing; ++j) {
      const int step = s0 + 8 * j, block = step * 2 + block_in_step;
      const bool live = block < blocks;
      uint4 xv[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int w = 0; w < 4; ++w)
          xv[nt][w] = live && nt * 8 + g < p.M ? *reinterpret_cast<const uint4*>(xr[nt] + step * 128 + w * 8) : zero;
      const uint32_t ca[4] = {wa[j].x, wa[j].y, wa[j].z, wa[j].w}, cb[4] = {wb[j].x, wb[j].y, wb[j].z, wb[j].w};
      uint32_t sa, ba, sb, bb;
      if (WHOLE) {
        w4_params(ga[j], sa, ba);
        w4_params(gb[j], sb, bb);
      }
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        if (!WHOLE) {
          const uint32_t* at = params + (block * 8 + half * 4 + w) / p.words_per_group * 128;
          w4_params(live ? __ldg(at) : 0u, sa, ba);
          w4_params(live ? __ldg(at + 8) : 0u, sb, bb);
        }
        uint32_t a[4], b[4];
        w4_decode<KIND>(ca[w], sa, ba, a);
        w4_decode<KIND>(cb[w], sb, bb, b);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          w4_mma(acc[nt], a[0], b[0], a[1], b[1], xv[nt][w].x, xv[nt][w].y);
          w4_mma(acc[nt], a[2], b[2], a[3], b[3], xv[nt][w].z, xv[nt][w].w);
        }
      }
      fetch(step + 8 * kRing, j);
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const int c = nt * 8 + t4 * 2;
    red[warp][g][c] = acc[nt][0];
    red[warp][g][c + 1] = acc[nt][1];
    red[warp][g + 8][c] = acc[nt][2];
    red[warp][g + 8][c + 1] = acc[nt][3];
  }
  __syncthreads();
  if (mine) {
    float v = 0.f;
#pragma unroll
    for (int z = 0; z < 8; ++z) v += red[z][row][t];
    if (p.residual) v += add;
    p.out[at] = __float2bfloat16(v);
  }
}

template <int NT, int KIND, bool WHOLE>
static int launch_w4_gemv(const W4GemvParams& p, cudaStream_t stream) {
  // the loads in flight live in L1: ask for a small shared-memory carve-out (as dense_gemv does)
  static bool set[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -6;
  if (!set[dev]) {
    if (cudaFuncSetAttribute(w4_gemv_kernel<NT, KIND, WHOLE>, cudaFuncAttributePreferredSharedMemoryCarveout, 15 * NT) != cudaSuccess) return -6;
    set[dev] = true;
  }
  launch_kernel(w4_gemv_kernel<NT, KIND, WHOLE>, dim3((p.N + 15) / 16), dim3(256), 0, stream, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

}  // namespace mfq

// The arguments of mfq_w4_gemm for up to 16 tokens.
extern "C" int mfq_w4_gemv(const void* packed, const void* group, const void* x, void* out, const void* residual, int M, int N, int K,
                           int group_size, int kind, cudaStream_t stream) {
  if (M <= 0 || M > 16 || N <= 0 || K <= 0 || K % 64 || group_size < 16 || group_size % 8 || K % group_size) return -1;
  if (kind != 0 && (kind != 1 || group_size != 32)) return -1;  // MXFP4 blocks are 32 wide
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(packed)) % 16) return -3;  // read in vectors, as by the TMA of mfq_w4_gemm
  const mfq::W4GemvParams p{static_cast<const uint8_t*>(packed), static_cast<const uint32_t*>(group), static_cast<const __nv_bfloat16*>(x),
                            static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(residual), M, N, K, K / group_size, group_size / 8};
  if (kind == 1) return M <= 8 ? mfq::launch_w4_gemv<1, 1, true>(p, stream) : mfq::launch_w4_gemv<2, 1, true>(p, stream);
  if (group_size % 32 == 0) return M <= 8 ? mfq::launch_w4_gemv<1, 0, true>(p, stream) : mfq::launch_w4_gemv<2, 0, true>(p, stream);
  return M <= 8 ? mfq::launch_w4_gemv<1, 0, false>(p, stream) : mfq::launch_w4_gemv<2, 0, false>(p, stream);
}
