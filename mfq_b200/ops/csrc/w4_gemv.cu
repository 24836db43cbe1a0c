// 4-bit weight streaming for up to 16 tokens:  out[t, n] = sum_k x[t, k] * w[n, k] (+ residual), weights in the layout of w4_gemm.cu.
//
// A decode step of a few tokens reads every weight once, so the time to beat is 0.625 bytes per weight at the memory's rate.  The
// tcgen05 form decodes into shared memory for the tensor core and is bound there by that hand-over (28672 x 4096: 62 us whatever the
// batch, 1.2 TB/s); here the codes go from memory into registers, through the same decode (w4_decode.cuh) and straight into
// mma.sync.m16n8k16 fragments.
//
// A CTA owns RT blocks of 16 weight rows, its warps take alternate steps of 128 inputs.  In a step a thread holds 32 consecutive codes
// (16 bytes) of rows g and g + 8 of a block; the four threads of a row cover two K blocks of 64 (32 bytes of a row are contiguous, eight
// rows 256).  The MMA's sums do not care which input sits in which k slot as long as both operands agree, so a word of eight codes is the
// thread's share of two MMAs, against the same eight values of x.  128 bytes of codes are in flight per thread, the first of them
// requested before the programmatic-launch wait.  The partial sums of an output meet in shared memory in warp order.
//
// What bounds it, besides the stream: x.  A thread reads 64 bytes of it per step, 16 bytes from each of 16 lines per warp load, and with
// 16 rows per CTA these loads keep L1 busier than the weights do.  Two blocks of rows (RT = 2) use what was read twice; the threads hold
// as many codes in half as many steps.  The sizes that take it are chosen in launch_w4_gemv.
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

// NT: blocks of 8 tokens.  RT: blocks of 16 weight rows.  WARPS: of a CTA.  WHOLE: a thread's 32 codes lie in one group (group size a
// multiple of 32).
template <int NT, int RT, int WARPS, int KIND, bool WHOLE>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS) w4_gemv_kernel(const W4GemvParams p) {
  pdl_trigger();
  constexpr int kRing = 4 / RT;
  __shared__ float red[WARPS][16 * RT][8 * NT + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int n0 = blockIdx.x * 16 * RT, blocks = p.K / 64, steps = (blocks + 1) / 2;
  const int block_in_step = t4 >> 1, half = t4 & 1;
  const uint8_t* codes = p.packed + size_t(n0 >> 7) * blocks * 4096 + ((n0 & 127) + g) * 32 + half * 16;
  const uint32_t* params = p.group + size_t(n0 >> 7) * p.groups * 128 + (n0 & 127) + g;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 wt[kRing][2 * RT];     // rows g, g + 8, ..
  uint32_t gp[kRing][2 * RT];  // their group parameters (WHOLE); zero parameters make the codes of a missing block zero weights
  auto fetch = [&](int step, int j) {
    const int block = step * 2 + block_in_step;
    const bool live = block < blocks;
#pragma unroll
    for (int r = 0; r < 2 * RT; ++r) wt[j][r] = live ? __ldcs(reinterpret_cast<const uint4*>(codes + size_t(block) * 4096 + r * 256)) : zero;
    if (WHOLE) {
      const uint32_t* at = params + (block * 8 + half * 4) / p.words_per_group * 128;
#pragma unroll
      for (int r = 0; r < 2 * RT; ++r) gp[j][r] = live ? __ldcs(at + r * 8) : 0u;
    }
  };
#pragma unroll
  for (int j = 0; j < kRing; ++j) fetch(warp + WARPS * j, j);
  pdl_wait();
  const __nv_bfloat16* xr[NT];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) xr[nt] = p.x + size_t(min(nt * 8 + g, p.M - 1)) * p.K + block_in_step * 64 + half * 32;
  // What this thread's first output is added to: requested under the product instead of after it (it is the only one unless a CTA
  // has more outputs than threads).
  const int t_first = threadIdx.x / (16 * RT), n_first = n0 + threadIdx.x % (16 * RT);
  const float early = p.residual && t_first < p.M && t_first < 8 * NT && n_first < p.N ? __bfloat162float(p.residual[size_t(t_first) * p.N + n_first]) : 0.f;
  float acc[NT][RT][4] = {};
  for (int s0 = warp; s0 < steps; s0 += WARPS * kRing) {
#pragma unroll
    for (int j = 0; j < kRing; ++j) {
      const int step = s0 + WARPS * j, block = step * 2 + block_in_step;
      const bool live = block < blocks;
      uint4 xv[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int w = 0; w < 4; ++w)
          xv[nt][w] = live && nt * 8 + g < p.M ? *reinterpret_cast<const uint4*>(xr[nt] + step * 128 + w * 8) : zero;
#pragma unroll
      for (int rt = 0; rt < RT; ++rt) {
        const uint4 va = wt[j][2 * rt], vb = wt[j][2 * rt + 1];
        const uint32_t ca[4] = {va.x, va.y, va.z, va.w}, cb[4] = {vb.x, vb.y, vb.z, vb.w};
        uint32_t sa, ba, sb, bb;
        if (WHOLE) {
          w4_params(gp[j][2 * rt], sa, ba);
          w4_params(gp[j][2 * rt + 1], sb, bb);
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          if (!WHOLE) {
            const uint32_t* at = params + (block * 8 + half * 4 + w) / p.words_per_group * 128 + rt * 16;
            w4_params(live ? __ldg(at) : 0u, sa, ba);
            w4_params(live ? __ldg(at + 8) : 0u, sb, bb);
          }
          uint32_t a[4], b[4];
          w4_decode<KIND>(ca[w], sa, ba, a);
          w4_decode<KIND>(cb[w], sb, bb, b);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            w4_mma(acc[nt][rt], a[0], b[0], a[1], b[1], xv[nt][w].x, xv[nt][w].y);
            w4_mma(acc[nt][rt], a[2], b[2], a[3], b[3], xv[nt][w].z, xv[nt][w].w);
          }
        }
      }
      fetch(step + WARPS * kRing, j);
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    const int c = nt * 8 + t4 * 2;
#pragma unroll
    for (int rt = 0; rt < RT; ++rt) {
      red[warp][rt * 16 + g][c] = acc[nt][rt][0];
      red[warp][rt * 16 + g][c + 1] = acc[nt][rt][1];
      red[warp][rt * 16 + g + 8][c] = acc[nt][rt][2];
      red[warp][rt * 16 + g + 8][c + 1] = acc[nt][rt][3];
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = threadIdx.x; i < 16 * RT * 8 * NT; i += WARPS * 32) {
    const int t = i / (16 * RT), row = i % (16 * RT), n = n0 + row;
    if (t >= p.M || n >= p.N) continue;
    float v = 0.f;
#pragma unroll
    for (int z = 0; z < WARPS; ++z) v += red[z][row][t];
    const size_t at = size_t(t) * p.N + n;
    if (p.residual) v += i == int(threadIdx.x) ? early : __bfloat162float(p.residual[at]);
    p.out[at] = __float2bfloat16(v);
  }
}

template <int NT, int RT, int WARPS, int KIND, bool WHOLE>
static int launch_w4_rows(const W4GemvParams& p, cudaStream_t stream) {
  // the loads in flight live in L1: ask for a small shared-memory carve-out (as dense_gemv does)
  static bool set[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -6;
  if (!set[dev]) {
    if (cudaFuncSetAttribute(w4_gemv_kernel<NT, RT, WARPS, KIND, WHOLE>, cudaFuncAttributePreferredSharedMemoryCarveout, 15 * NT) != cudaSuccess) return -6;
    set[dev] = true;
  }
  launch_kernel(w4_gemv_kernel<NT, RT, WARPS, KIND, WHOLE>, dim3((p.N + 16 * RT - 1) / (16 * RT)), dim3(32 * WARPS), 0, stream, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

template <int NT, int KIND, bool WHOLE>
static int launch_w4_gemv(const W4GemvParams& p, cudaStream_t stream) {
  // Two blocks of rows per CTA halve the reads of x and the number of CTAs.  Up to 8 tokens that pays where two CTAs per SM are left,
  // or, with 16 warps in one CTA per SM, where K is long: 28672 x 4096 28.0 -> 23.8 us (31.2 with 16 warps), 4096 x 14336 16.0 -> 14.5
  // (20.2 with eight); 6144 x 4096 stays at 9.7.  With 16 tokens, twice the reads, always: 48.4 -> 31.2, 23.7 -> 17.8, 14.3 -> 9.9 us.
  // Where there are three times as many CTAs as SMs and more, four warps each and four CTAs per SM: a warp has twice the steps, so its
  // first loads and its CTA's sum are half as much of its time, and they fall under the work of three other CTAs instead of one.
  // 28672 x 4096 24.3 -> 22.5 us, 128256 x 4096 92.4 -> 82.7 (16 tokens 31.5 -> 28.2, 120 -> 104), 14336 x 2048 7.9 -> 7.1.  Below,
  // the last wave costs more: 13824 x 5120 15.9 and 16.1 us, 12288 x 4096 11.4 and 13.1.
  const int rows32 = (p.N + 31) / 32, steps = (p.K + 127) / 128;
  if (rows32 > 3 * 148) return launch_w4_rows<NT, 2, 4, KIND, WHOLE>(p, stream);
  if (rows32 >= 2 * 148 || (NT == 2 && rows32 > 148)) return launch_w4_rows<NT, 2, 8, KIND, WHOLE>(p, stream);
  if (NT == 2 || (rows32 <= 148 && steps >= 64)) return launch_w4_rows<NT, 2, 16, KIND, WHOLE>(p, stream);
  return launch_w4_rows<1, 1, 8, KIND, WHOLE>(p, stream);
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
