// Causal self-attention for prefill chunks on tcgen05 tensor cores (bf16 in, fp32 accumulate, head dim 128, GQA).
//
// One CTA = (128-query block, query head).  Per 128-key block:
//   S = Q K^T      tcgen05.mma kind::f16, A = Q tile, B = K tile (both K-major, TMA 128 B swizzle), S in TMEM
//   P = softmax    8 warps, two threads per query row (64 keys each): two passes over the TMEM row (max, then exp2 + sum), row maxima
//                  exchanged through shared memory; P goes back as bf16 pairs into the columns its own scores came from
//   O_blk = P V    tcgen05.mma with P from TENSOR MEMORY as the A operand and V as an MN-major B operand (the [key][dim] tile exactly
//                  as TMA delivers it)
//   O = (O + O_blk(prev)) * alpha   folded in fp32 registers, so TMEM never needs an in-place rescale
// The chain  softmax -> P V -> fold  is several times as long as the MMAs, so Q K^T of block j + 1 is issued before P V of block j, into
// the other of two S buffers, and all of it but the chain itself is hidden; P never passes through shared memory and its proxy fence.
// What bounds it is the softmax: exponentials, and the two passes over S.
// Grids that fill two CTAs per SM (two_ctas_per_sm) take the pair form: K and V in one stage each, one S buffer (P lies in S, so Q K^T of block j + 1 follows
// P V of block j), a thread per query row with all 128 of its outputs in registers, no exchange of maxima.  Its chain per block is half as long
// again, but two CTAs hide each other's waits.  (The compiler sees 128 registers a thread, of which setmaxnreg makes 200, and spills 124 bytes.)  O alpha + O_blk is formed as a product while P V runs and a sum while the next Q K^T does, by
// two values per instruction in either form.  32 heads on a B200, one CTA per SM one value per instruction | two | pair form, same bits:
//   120 tokens 8.7 | 7.0 | 7.7 us    512 after 4000 (128 CTAs) 61 | 58 | 88    700 (192) 18.9 | 15.9 | 19.3    1000 after 3001 (256) 95 | 90 | 85
//   1500 43.5 | 40.1 | 36.1    2048 65 | 62 | 51    4096 199 | 192 | 161    8192 688 | 665 | 570
// Heaviest (latest) query blocks are scheduled first, over all heads.
//
// The reference's prefill attention is a llama.cpp-derived mma.sync flash-attention (mfq_fattn_mma_f16.cuh) and a
// wmma D=256 kernel (attention.cu:218).
#include "common.cuh"

#include <cfloat>

namespace mfq {

constexpr int kQB = 128, kKB = 128, kHD = 128;
constexpr int kTileBytes = kQB * kHD * 2;       // 32 KB: one [128 x 128] bf16 tile = two 16 KB swizzled halves
constexpr int kHalfBytes = kTileBytes / 2;
constexpr int kPrefillThreads = 128 + 256;  // TMA warp, MMA warp, two idle warps; eight softmax warps
constexpr int kPrefillSmem = kTileBytes /*Q*/ + 2 * 2 * kTileBytes /*K, V x 2 stages*/ + 1024 + 256 + 6 * kQB * 4 /*row max / sum exchange*/;
constexpr int kPairThreads = 128 + 128;     // two CTAs per SM: four softmax warps each
constexpr int kPairSmem = 3 * kTileBytes /*Q, K, V*/ + 1024 + 256;

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_store_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
// D (+)= A B over 64 keys with A [128 x 64] bf16 in tensor memory (two values per column: 8 columns per k-step of 16) and B = 64 keys x
// 128 dims, MN-major, 2 KB per k-step.  Whole warp, one elected lane issues the four steps.
__device__ __forceinline__ void umma_pv(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred q, f, t;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
      "setp.ne.b32 f, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
      "add.s64 b1, %2, 128;\n\tadd.s64 b2, %2, 256;\n\tadd.s64 b3, %2, 384;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, f;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n\t}"
      ::"r"(d), "r"(a_tmem), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <bool kMasked>
struct MaskedBlock {
  static constexpr bool value = kMasked;
};

struct PrefillParams {
  __nv_bfloat16* out;  // [T, Hq, 128]
  int T, Hq, Hk;       // T: query rows
  int Tk, offset;      // keys available; query row i sees keys 0 .. i + offset (offset = Tk - T: tokens before the chunk)
  float scale_log2;
  int* status;
};

__global__ void __launch_bounds__(kPrefillThreads, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const PrefillParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = base;
  uint8_t* sK = base + kTileBytes;                  // two stages
  uint8_t* sV = sK + 2 * kTileBytes;                // two stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * kTileBytes);
  uint64_t* q_full = bars;            // 1
  uint64_t* k_full = bars + 1;        // [2] per stage, like the three below
  uint64_t* k_empty = bars + 3;
  uint64_t* v_full = bars + 5;
  uint64_t* v_empty = bars + 7;
  uint64_t* s_full = bars + 9;        // [2] per S buffer
  uint64_t* p_full = bars + 11;       // 8 arrivals: P is in TMEM, and O has been read
  uint64_t* o_full = bars + 12;       // P V of a block is complete
  uint64_t* x_bar = bars + 13;        // 8 arrivals: row-maximum exchange, one phase per key block
  uint64_t* l_bar = bars + 14;        // 8 arrivals: row-sum exchange, once
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* s_max = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);  // max: [2 buffers][2 halves][128 rows]; sum: [2 halves][128 rows]

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
  const int qb = (p.T + kQB - 1) / kQB - 1 - int(blockIdx.x) / p.Hq;  // heavy blocks first
  const int head = int(blockIdx.x) % p.Hq, kvh = head / (p.Hq / p.Hk);
  // causal with a past: the last query of the block sees keys up to (qb + 1) * kQB - 1 + offset
  const int nblk = min((p.Tk + kKB - 1) / kKB, ((qb + 1) * kQB + p.offset + kKB - 1) / kKB);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); mbar_init(&s_full[i], 1);
    }
    mbar_init(p_full, 8); mbar_init(o_full, 1); mbar_init(x_bar, 8); mbar_init(l_bar, 8);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_trigger();  // TMEM is held by now
  pdl_wait();
  // columns: S of even blocks, S of odd blocks (P of 64 keys in the first half of each 64 columns), O

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
      mbar_expect_tx(q_full, kTileBytes);
      tma_load_2d(sQ, &tmap_q, q_full, head * kHD, qb * kQB);
      tma_load_2d(sQ + kHalfBytes, &tmap_q, q_full, head * kHD + 64, qb * kQB);
      for (int j = 0; j < nblk; ++j) {
        const int s = j & 1;
        const uint32_t parity = ((j >> 1) & 1) ^ 1;
        uint8_t *k = sK + s * kTileBytes, *v = sV + s * kTileBytes;
        if (!mbar_wait(&k_empty[s], parity, abort_flag, p.status, kStatusTimeoutProducer)) break;
        mbar_expect_tx(&k_full[s], kTileBytes);
        tma_load_2d(k, &tmap_k, &k_full[s], kvh * kHD, j * kKB);
        tma_load_2d(k + kHalfBytes, &tmap_k, &k_full[s], kvh * kHD + 64, j * kKB);
        if (!mbar_wait(&v_empty[s], parity, abort_flag, p.status, kStatusTimeoutProducer)) break;
        mbar_expect_tx(&v_full[s], kTileBytes);
        tma_load_2d(v, &tmap_v, &v_full[s], kvh * kHD, j * kKB);
        tma_load_2d(v + kHalfBytes, &tmap_v, &v_full[s], kvh * kHD + 64, j * kKB);
      }
    }
  } else if (warp == 1) {
    // issued by an elected lane of the converged warp (common.cuh: umma_f8f6f4_block says why)
    constexpr uint32_t idesc_qk = umma_idesc(128, 128, 1, 1, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc(128, 128, 1, 1, 0, 1);  // B = V is MN-major
    constexpr uint64_t kTile = kTileBytes >> 4, kHalf = kHalfBytes >> 4;  // dims 64.. of Q and K live in the second swizzled half
    const uint64_t q_desc = umma_desc_k_sw128(smem_u32(sQ)), k_desc0 = umma_desc_k_sw128(smem_u32(sK));
    const uint64_t v_desc0 = umma_desc_mn_sw128(smem_u32(sV), kHalfBytes);
    const uint32_t s_full_addr = smem_u32(s_full);
    auto issue_qk = [&](int j) {  // S takes the place of P of block j - 2, which the MMAs before have read
      const uint64_t k_desc = k_desc0 + uint64_t(j & 1) * kTile;
      const uint32_t d = tmem_base + uint32_t(j & 1) * 128u;
      umma_f16_block(d, q_desc, k_desc, idesc_qk, 0u);
      umma_f16_block(d, q_desc + kHalf, k_desc + kHalf, idesc_qk, 1u, s_full_addr + (j & 1) * 8);
      tc_commit_warp(&k_empty[j & 1]);
    };
    bool ok = mbar_wait_warp(q_full, 0, abort_flag, p.status, kStatusTimeoutMma) &&
              mbar_wait_warp(&k_full[0], 0, abort_flag, p.status, kStatusTimeoutMma);
    if (ok) {
      tc_fence_after();
      issue_qk(0);
    }
    for (int j = 0; ok && j < nblk; ++j) {
      if (j + 1 < nblk) {
        ok = mbar_wait_warp(&k_full[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag, p.status, kStatusTimeoutMma);
        if (!ok) break;
        tc_fence_after();
        issue_qk(j + 1);
      }
      ok = mbar_wait_warp(&v_full[j & 1], (j >> 1) & 1, abort_flag, p.status, kStatusTimeoutMma) &&
           mbar_wait_warp(p_full, j & 1, abort_flag, p.status, kStatusTimeoutMma);
      if (!ok) break;
      tc_fence_after();
      const uint32_t p_addr = tmem_base + uint32_t(j & 1) * 128u;
      const uint64_t v_desc = v_desc0 + uint64_t(j & 1) * kTile;
      umma_pv(tmem_base + 256u, p_addr, v_desc, idesc_pv, 0u);
      umma_pv(tmem_base + 256u, p_addr + 64u, v_desc + 512, idesc_pv, 1u);
      tc_commit_warp(o_full);
      tc_commit_warp(&v_empty[j & 1]);
    }
  } else if (warp >= 4) {
    // ----- softmax warps: two threads per query row (TMEM lane); `half` selects 64 of the 128 keys of a block and 64 of the 128 output
    // dims -----
    const int half = (warp - 4) >> 2, quarter = warp & 3;
    const int row = quarter * 32 + lane, q_idx = qb * kQB + row;
    const uint32_t lane_base = tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(half) * 64u;
    const uint32_t tO = lane_base + 256u;
    float o[64];
#pragma unroll
    for (int d = 0; d < 64; ++d) o[d] = 0.f;
    float m_run = -FLT_MAX, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < nblk; ++j) {
      const int sb = j & 1;
      const uint32_t tS = lane_base + uint32_t(sb) * 128u;
      ok = mbar_wait_warp(&s_full[sb], (j >> 1) & 1, abort_flag, p.status, kStatusTimeoutEpilogue);
      if (!ok) break;
      tc_fence_after();
      const int key0 = j * kKB + half * 64;
      // masking is needed where the block reaches past the FIRST query's horizon or past the last key
      const bool diag = ((j + 1) * kKB - 1 > qb * kQB + p.offset) || ((j + 1) * kKB > p.Tk);
      // pass 1: maximum over this thread's 64 columns, then exchange with the partner thread of the row
      float mx = -FLT_MAX;
      {
        uint32_t r[2][32];
        tmem_ld_32x32(tS, r[0]);
        tmem_ld_32x32(tS + 32, r[1]);
        tmem_wait_ld();
        if (!diag) {
#pragma unroll
          for (int i = 0; i < 64; ++i) mx = fmaxf(mx, __uint_as_float(r[i >> 5][i & 31]));
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            mx = fmaxf(mx, (key0 + i <= q_idx + p.offset && key0 + i < p.Tk) ? __uint_as_float(r[i >> 5][i & 31]) : -FLT_MAX);
        }
      }
      s_max[(sb * 2 + half) * kQB + row] = mx;
      __syncwarp();
      if (lane == 0) mbar_arrive(x_bar);
      ok = mbar_wait_warp(x_bar, j & 1, abort_flag, p.status, kStatusTimeoutEpilogue);
      if (!ok) break;
      mx = fmaxf(mx, s_max[(sb * 2 + (half ^ 1)) * kQB + row]);
      const float m_new = fmaxf(m_run, mx);
      const float alpha = fast_exp2((m_run - m_new) * p.scale_log2);
      // fold the previous block's P V (it was computed against m_run), then move to the new maximum
      if (j > 0) {
        ok = mbar_wait_warp(o_full, (j - 1) & 1, abort_flag, p.status, kStatusTimeoutEpilogue);
        if (!ok) break;
        tc_fence_after();
        uint32_t r[2][32];
        tmem_ld_32x32(tO, r[0]);
        tmem_ld_32x32(tO + 32, r[1]);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          add2(o[i], o[i + 1], r[i >> 5][i & 31], r[i >> 5][(i & 31) + 1]);
          scale2(o[i], o[i + 1], alpha);
        }
      }
      l_run *= alpha;
      m_run = m_new;
      // pass 2: probabilities -> bf16 pairs over the scores that have been read
      const float mb = m_new * p.scale_log2;
      float psum = 0.f;
      auto probabilities = [&](auto masked) {
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(tS + c, r);
          tmem_wait_ld();
          uint32_t packed[16];
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 e = fma_f2(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), both(p.scale_log2), both(-mb));
            float p0 = fast_exp2(e.x), p1 = fast_exp2(e.y);
            if (decltype(masked)::value) {
              const int key = key0 + c + i;
              if (!(key <= q_idx + p.offset && key < p.Tk)) p0 = 0.f;
              if (!(key + 1 <= q_idx + p.offset && key + 1 < p.Tk)) p1 = 0.f;
            }
            psum += p0 + p1;
            const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
            packed[i >> 1] = *reinterpret_cast<const uint32_t*>(&h);
          }
          tmem_store_32x16(tS + c / 2, packed);
        }
      };
      if (diag) probabilities(MaskedBlock<true>());
      else probabilities(MaskedBlock<false>());
      l_run += psum;
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    if (ok) {
      // total row sum = both halves
      s_max[(4 + half) * kQB + row] = l_run;  // own slots: the last block's maxima may still be read
      __syncwarp();
      if (lane == 0) mbar_arrive(l_bar);
      ok = mbar_wait_warp(l_bar, 0, abort_flag, p.status, kStatusTimeoutEpilogue) &&
           mbar_wait_warp(o_full, (nblk - 1) & 1, abort_flag, p.status, kStatusTimeoutEpilogue);
      if (ok) {
        tc_fence_after();
        const float l_tot = l_run + s_max[(4 + (half ^ 1)) * kQB + row];
        const float inv = l_tot > 0.f ? 1.f / l_tot : 0.f;
        __nv_bfloat16* dst = p.out + (size_t(q_idx) * p.Hq + head) * kHD + half * 64;
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32(tO + c, r);
          tmem_wait_ld();
          if (q_idx < p.T) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 v;
              __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
              for (int e = 0; e < 4; ++e)
                h[e] = __floats2bfloat162_rn((o[c + i + 2 * e] + __uint_as_float(r[i + 2 * e])) * inv,
                                             (o[c + i + 2 * e + 1] + __uint_as_float(r[i + 2 * e + 1])) * inv);
              *reinterpret_cast<uint4*>(dst + c + i) = v;
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// The same with two CTAs per SM, for grids that fill them (the head of this file says how).
__global__ void __launch_bounds__(kPairThreads, 2)
attn_prefill_pair_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const PrefillParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = base;
  uint8_t* sK = base + kTileBytes;
  uint8_t* sV = sK + kTileBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kTileBytes);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = bars + 2;
  uint64_t* v_full = bars + 3;
  uint64_t* v_empty = bars + 4;
  uint64_t* s_full = bars + 5;
  uint64_t* p_full = bars + 6;  // 4 arrivals: P is in TMEM, and O of the block before has been read
  uint64_t* o_full = bars + 7;  // P V of a block is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
  const int qb = (p.T + kQB - 1) / kQB - 1 - int(blockIdx.x) / p.Hq;  // heavy blocks first
  const int head = int(blockIdx.x) % p.Hq, kvh = head / (p.Hq / p.Hk);
  // causal with a past: the last query of the block sees keys up to (qb + 1) * kQB - 1 + offset
  const int nblk = min((p.Tk + kKB - 1) / kKB, ((qb + 1) * kQB + p.offset + kKB - 1) / kKB);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 6; ++i) mbar_init(&bars[i], 1);
    mbar_init(p_full, 4);
    mbar_init(o_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);  // columns: S (P of 64 keys in the first half of each 64 columns), O
  pdl_trigger();  // TMEM is held by now
  // a softmax thread holds a row of O: 128 registers of its own
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  pdl_wait();
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
      mbar_expect_tx(q_full, kTileBytes);
      tma_load_2d(sQ, &tmap_q, q_full, head * kHD, qb * kQB);
      tma_load_2d(sQ + kHalfBytes, &tmap_q, q_full, head * kHD + 64, qb * kQB);
      for (int j = 0; j < nblk; ++j) {
        if (!mbar_wait(k_empty, (j & 1) ^ 1, abort_flag, p.status, kStatusTimeoutProducer)) break;
        mbar_expect_tx(k_full, kTileBytes);
        tma_load_2d(sK, &tmap_k, k_full, kvh * kHD, j * kKB);
        tma_load_2d(sK + kHalfBytes, &tmap_k, k_full, kvh * kHD + 64, j * kKB);
        if (!mbar_wait(v_empty, (j & 1) ^ 1, abort_flag, p.status, kStatusTimeoutProducer)) break;
        mbar_expect_tx(v_full, kTileBytes);
        tma_load_2d(sV, &tmap_v, v_full, kvh * kHD, j * kKB);
        tma_load_2d(sV + kHalfBytes, &tmap_v, v_full, kvh * kHD + 64, j * kKB);
      }
    }
  } else if (warp == 1) {
    // issued by an elected lane of the converged warp (common.cuh: umma_f8f6f4_block says why)
    constexpr uint32_t idesc_qk = umma_idesc(128, 128, 1, 1, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc(128, 128, 1, 1, 0, 1);  // B = V is MN-major
    constexpr uint64_t kHalf = kHalfBytes >> 4;  // dims 64.. of Q and K live in the second swizzled half
    const uint64_t q_desc = umma_desc_k_sw128(smem_u32(sQ)), k_desc = umma_desc_k_sw128(smem_u32(sK));
    const uint64_t v_desc = umma_desc_mn_sw128(smem_u32(sV), kHalfBytes);
    auto issue_qk = [&] {  // S takes the place of P of the block before, which the MMAs before have read
      umma_f16_block(tmem_base, q_desc, k_desc, idesc_qk, 0u);
      umma_f16_block(tmem_base, q_desc + kHalf, k_desc + kHalf, idesc_qk, 1u, smem_u32(s_full), smem_u32(k_empty));
    };
    bool ok = mbar_wait_warp(q_full, 0, abort_flag, p.status, kStatusTimeoutMma) &&
              mbar_wait_warp(k_full, 0, abort_flag, p.status, kStatusTimeoutMma);
    if (ok) {
      tc_fence_after();
      issue_qk();
    }
    for (int j = 0; ok && j < nblk; ++j) {
      ok = mbar_wait_warp(v_full, j & 1, abort_flag, p.status, kStatusTimeoutMma) &&
           (j + 1 == nblk || mbar_wait_warp(k_full, (j + 1) & 1, abort_flag, p.status, kStatusTimeoutMma)) &&
           mbar_wait_warp(p_full, j & 1, abort_flag, p.status, kStatusTimeoutMma);
      if (!ok) break;
      tc_fence_after();
      umma_pv(tmem_base + 128u, tmem_base, v_desc, idesc_pv, 0u);
      umma_pv(tmem_base + 128u, tmem_base + 64u, v_desc + 512, idesc_pv, 1u);
      tc_commit_warp(o_full);
      tc_commit_warp(v_empty);
      if (j + 1 < nblk) issue_qk();
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    pdl_wait();
    // ----- softmax warps: a thread per query row (TMEM lane) -----
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane, q_idx = qb * kQB + row;
    const uint32_t tS = tmem_base + (uint32_t(quarter * 32) << 16), tO = tS + 128u;
    float o[128];
#pragma unroll
    for (int d = 0; d < 128; ++d) o[d] = 0.f;
    float m_run = -FLT_MAX, l_run[2] = {0.f, 0.f};  // sums of the first and the second 64 keys of the blocks
    bool ok = true;
    for (int j = 0; j < nblk; ++j) {
      ok = mbar_wait_warp(s_full, j & 1, abort_flag, p.status, kStatusTimeoutEpilogue);
      if (!ok) break;
      tc_fence_after();
      const int key0 = j * kKB;
      // masking is needed where the block reaches past the FIRST query's horizon or past the last key
      const bool diag = ((j + 1) * kKB - 1 > qb * kQB + p.offset) || ((j + 1) * kKB > p.Tk);
      const int last = min(q_idx + p.offset, p.Tk - 1) - key0;  // last key of the block that this query sees
      float mx[2] = {-FLT_MAX, -FLT_MAX};
      {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          tmem_ld_32x32(tS + c * 32, r);
          tmem_wait_ld();
          if (!diag) {
#pragma unroll
            for (int i = 0; i < 32; ++i) mx[i & 1] = fmaxf(mx[i & 1], __uint_as_float(r[i]));
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) mx[i & 1] = fmaxf(mx[i & 1], c * 32 + i <= last ? __uint_as_float(r[i]) : -FLT_MAX);
          }
        }
      }
      const float m_new = fmaxf(m_run, fmaxf(mx[0], mx[1]));
      const float alpha = fast_exp2((m_run - m_new) * p.scale_log2);
      m_run = m_new;
      // probabilities -> bf16 pairs over the scores that have been read
      const float mb = m_new * p.scale_log2;
      auto probabilities = [&](auto masked) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float psum = 0.f;
#pragma unroll
          for (int c = 0; c < 64; c += 32) {
            uint32_t r[32];
            tmem_ld_32x32(tS + half * 64 + c, r);
            tmem_wait_ld();
            uint32_t packed[16];
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float2 e = fma_f2(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), both(p.scale_log2), both(-mb));
              float p0 = fast_exp2(e.x), p1 = fast_exp2(e.y);
              if (decltype(masked)::value) {
                if (half * 64 + c + i > last) p0 = 0.f;
                if (half * 64 + c + i + 1 > last) p1 = 0.f;
              }
              psum += p0 + p1;
              const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
              packed[i >> 1] = *reinterpret_cast<const uint32_t*>(&h);
            }
            tmem_store_32x16(tS + half * 64 + c / 2, packed);
          }
          l_run[half] = __fadd_rn(__fmul_rn(l_run[half], alpha), psum);
        }
      };
      if (diag) probabilities(MaskedBlock<true>());
      else probabilities(MaskedBlock<false>());
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      if (j > 0) {
#pragma unroll
        for (int d = 0; d < 128; d += 2) scale2(o[d], o[d + 1], alpha);
      }
      ok = mbar_wait_warp(o_full, j & 1, abort_flag, p.status, kStatusTimeoutEpilogue);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 128; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tO + c, r);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 32; i += 2) add2(o[c + i], o[c + i + 1], r[i], r[i + 1]);
      }
    }
    if (ok && q_idx < p.T) {
      const float l_tot = l_run[0] + l_run[1];
      const float inv = l_tot > 0.f ? 1.f / l_tot : 0.f;
      __nv_bfloat16* dst = p.out + (size_t(q_idx) * p.Hq + head) * kHD;
#pragma unroll
      for (int c = 0; c < 128; c += 8) {
        uint4 v;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
        for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(o[c + 2 * e] * inv, o[c + 2 * e + 1] * inv);
        *reinterpret_cast<uint4*>(dst + c) = v;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 256);
}

}  // namespace mfq

namespace mfq {
// Which form a grid takes.  Two CTAs per SM share its rate and hide each other's waits (7 to 20 %), but a CTA alone is half as slow again, so the
// pair form needs company for the longest tiles: enough key blocks in all against those of the first tile, and, in a grid of two
// or three rounds of one CTA per SM, none of those rounds nearly full of tiles alike, which one CTA per SM works off without a rest.  (With a
// long past tiles are alike, and then up to two rounds are the other way about: all of them at once by twos.)  One | pair, on a B200:
//   16 heads: 2028 tokens (256 CTAs) 32.1 | 44.9 us, 2540 (320) 47 | 51, 3052 (384) 62.8 | 61.4, 4076 (512) 94 | 82
//   32 heads: 1004 tokens (256) 20.9 | 24.9, 1260 (320) 31.0 | 29.3, after 3000 (320) 128 | 127; 1004 after 300 30.7 | 33.1, after 1000 43.6 | 45.3,
//   after 3000 85.8 | 84.3, after 8000 188 | 178; 1516 after 8000 (384, three rounds nearly full) 289 | 321
// Over 540 grids of 148 to 1024 CTAs and pasts to 8000 the slower form is taken in 4 by more than 2 % (8 %), and choosing costs 0.7 % on average.
constexpr int kSms = 148;
static bool two_ctas_per_sm(int T, int Tk, int Hq) {
  const long blocks = (T + kQB - 1) / kQB, past = (Tk - T + kKB - 1) / kKB, ctas = blocks * Hq;
  if (ctas < 250) return false;
  const auto keys = [&](long cta) { return min((Tk + kKB - 1L) / kKB, blocks - cta / Hq + past); };  // key blocks of the tile of a CTA; heavy ones first
  const long most = keys(0), all = Hq * (blocks * (blocks + 1) / 2 + blocks * past);
  if (ctas <= 2 * kSms) return 100 * keys(kSms) >= 87 * most;
  return 4 * all >= 5 * kSms * most && (ctas > 3 * kSms || 100 * 3 * keys(2 * kSms) * kSms <= 93 * all);
}
}  // namespace mfq

// 1: the pair form
extern "C" int mfq_attn_prefill_form(int T, int Tk, int Hq) { return T > 0 && Tk >= T && Hq > 0 && mfq::two_ctas_per_sm(T, Tk, Hq); }

// q: [T, Hq, 128] bf16, k/v: [Tk, Hk, 128] bf16 (contiguous), out: [T, Hq, 128] bf16.  Tk >= T: the first Tk - T keys
// are the sequence's past (earlier chunks / a restored prefix); query i attends to keys 0 .. i + (Tk - T).
extern "C" int mfq_attn_prefill_past(const void* q, const void* k, const void* v, void* out, int T, int Tk, int Hq, int Hk,
                                     int D, float sm_scale, int* status, cudaStream_t stream) {
  using namespace mfq;
  if (D != 128 || T <= 0 || Tk < T || Hq % Hk) return -1;
  CUtensorMap tq, tk, tv;
  if (make_tmap_2d(&tq, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, T, uint64_t(Hq) * D, uint64_t(Hq) * D * 2, kQB, 64)) return -2;
  if (make_tmap_2d(&tk, k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, Tk, uint64_t(Hk) * D, uint64_t(Hk) * D * 2, kKB, 64)) return -3;
  if (make_tmap_2d(&tv, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, Tk, uint64_t(Hk) * D, uint64_t(Hk) * D * 2, kKB, 64)) return -4;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(attn_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrefillSmem) != cudaSuccess ||
        cudaFuncSetAttribute(attn_prefill_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem) != cudaSuccess)
      return -6;
    attr = true;
  }
  const PrefillParams p{static_cast<__nv_bfloat16*>(out), T, Hq, Hk, Tk, Tk - T, sm_scale * 1.4426950408889634f, status};
  const int ctas = (T + kQB - 1) / kQB * Hq;
  if (two_ctas_per_sm(T, Tk, Hq)) launch_kernel(attn_prefill_pair_kernel, dim3(ctas), dim3(kPairThreads), kPairSmem, stream, tq, tk, tv, p);
  else launch_kernel(attn_prefill_kernel, dim3(ctas), dim3(kPrefillThreads), kPrefillSmem, stream, tq, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

// Self-contained chunk (no past): Tk = T.
extern "C" int mfq_attn_prefill_bf16(const void* q, const void* k, const void* v, void* out, int T, int Hq, int Hk,
                                     int D, float sm_scale, int* status, cudaStream_t stream) {
  return mfq_attn_prefill_past(q, k, v, out, T, T, Hq, Hk, D, sm_scale, status, stream);
}
