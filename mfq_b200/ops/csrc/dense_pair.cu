// Unquantized linears for wide batches on pairs of SMs:  out[t, n] = epilogue(sum_k x[t, k] w[n, k]),  bf16 -> fp32 accumulate.
//
// Prompt-sized products are a matter of keeping the tensor cores fed.  The one-SM kernel (dense_gemm.cu) launches one CTA per tile:
// of a 4096-deep tile's 29 us (256 tokens) some 7 are its own ramp and store, and it reads every operand byte twice as often from
// L2.  Here a pair of CTAs works on 256 weight rows x BT tokens with `tcgen05.mma.cta_group::2` (each CTA stages its 128 weight
// rows and half of the tokens), pairs walk the tiles without leaving, and the accumulators of TMEM are used in turn, so that a
// tile's output stage runs under the next tile's main loop.
//
// Roles per CTA: warp 0 = TMA, warp 1 = TMEM owner and, in the leader, MMA issuer, warps 4..11 = output stage (TMEM lane quarter =
// warp % 4, two warps per quarter split the tokens).  Barriers as in fp8_gemm_2cta.cu, except that an accumulator is complete once per
// tile.  A warp of the output stage turns 32 rows x 16 tokens through its own 2 KB of shared memory, so that a lane holds 8
// consecutive rows of a token: 16-byte stores, and the pairs of 8 gate and 8 up rows of a gated unit in one thread.
// A product that the one-SM kernel would split along K is summed in the same parts (kParts): each gets an accumulator of its own, and the
// output stage adds them up in order, so that the sums and their rounding are the split form's.  In one accumulator 200 x 6144 x 4096 was
// twice as far from 64 bits (4.4e-6 instead of 2.1e-6 of the result).
// 1508 tokens on a B200, one-SM kernel -> this one: 28672 x 4096 gated 462 -> 252 us (1.40 PFLOP/s), 6144 x 4096 73 -> 53, 4096 x 4096
// 64 -> 50, 4096 x 14336 211 -> 170; 4096 tokens of the first 1225 -> 687.
#include "dense_common.cuh"
#include "pair.cuh"

namespace mfq {
namespace {

constexpr int kRows = 128, kBK = 64;  // weight rows per CTA; bf16 values per K block

template <int BT>
struct DensePairCfg {
  static constexpr int kStages = 6;
  static constexpr int kAcc = 512 / BT;
  static constexpr int kStageBytes = (kRows + BT / 2) * kBK * 2;
  static constexpr int kEpiWarps = 8, kThreads = 128 + 32 * kEpiWarps;
  static constexpr int kTurnBytes = kEpiWarps * 16 * 32 * 4;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256 + kTurnBytes;
};

struct DensePairParams {
  DenseEpilogue epi;
  int* status;
  int M, N, K;
  int kb_per_part;  // kParts: K blocks of a part
};

template <int BT, bool kParts>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(DensePairCfg<BT>::kThreads, 1)
dense_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const DensePairParams p) {
  using Cfg = DensePairCfg<BT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(tiles + Cfg::kStages * Cfg::kStageBytes);  // used in the leader only
  uint64_t* empty = full + Cfg::kStages;                                                  // one set per CTA
  uint64_t* acc_full = empty + Cfg::kStages;                                              // one set per CTA
  uint64_t* acc_empty = acc_full + Cfg::kAcc;                                             // used in the leader only
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + Cfg::kAcc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* turn_all = reinterpret_cast<float*>(tiles + Cfg::kStages * Cfg::kStageBytes + 256);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();  // 0 = leader
  const bool leader = rank == 0;
  const int nkb = (p.K + kBK - 1) / kBK, per_part = kParts ? p.kb_per_part : nkb, parts = kParts ? (nkb + per_part - 1) / per_part : 1;
  const int clusters = int(gridDim.x) / 2, cluster = int(blockIdx.x) / 2;
  // token tiles innermost: pairs at work at the same time share the weight rows in L2
  const int t_tiles = (p.M + BT - 1) / BT, tiles_total = t_tiles * ((p.N + 2 * kRows - 1) / (2 * kRows));
  auto tile_n0 = [&](int tile) { return (tile / t_tiles) * 2 * kRows + int(rank) * kRows; };
  auto tile_t0 = [&](int tile) { return (tile % t_tiles) * BT; };

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < Cfg::kAcc; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 2 * Cfg::kEpiWarps); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anybody signals across
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_trigger();  // TMEM is held by now: a successor that wants some waits for it, not the other way round
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_w);
      tma_prefetch_desc(&tmap_x);
    }
    __syncwarp();
    const uint32_t tiles_addr = smem_u32(tiles), full_local = smem_u32(full), full_leader = map_to_cta(full, 0);
    const uint32_t bytes = leader ? 2u * Cfg::kStageBytes : 0u;  // the bytes of both CTAs land on the leader's barrier
    int s = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = cluster; ok && tile < tiles_total; tile += clusters) {
      const int n0 = tile_n0(tile), t0 = tile_t0(tile) + int(rank) * (BT / 2);
      for (int i = 0; i < nkb; ++i) {
        ok = mbar_wait_warp(&empty[s], phase ^ 1u, abort_flag, p.status, kStatusTimeoutProducer);
        if (!ok) break;
        const uint32_t a = tiles_addr + s * Cfg::kStageBytes;
        tma_load_stage_pair(a, a + kRows * kBK * 2, &tmap_w, &tmap_x, full_leader + s * 8, full_local + s * 8, bytes, i * kBK, n0, t0);
        if (++s == Cfg::kStages) { s = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1 && leader) {
    constexpr uint32_t idesc = umma_idesc(2 * kRows, BT, 1, 1);
    constexpr uint64_t kStageStep = uint64_t(Cfg::kStageBytes >> 4);
    const uint64_t a_desc0 = umma_desc_k_sw128(smem_u32(tiles)), b_desc0 = umma_desc_k_sw128(smem_u32(tiles) + kRows * kBK * 2);
    const uint32_t empty_addr = smem_u32(empty), acc_full_addr = smem_u32(acc_full);
    int s = 0;
    uint32_t phase = 0, buf = 0, acc_phase = 1;  // the first pass over the accumulators finds them free
    bool ok = true;
    for (int tile = cluster; ok && tile < tiles_total; tile += clusters) {
      for (int first = 0; ok && first < nkb; first += per_part) {
        const int end = min(nkb, first + per_part);
        ok = mbar_wait_warp(&acc_empty[buf], acc_phase, abort_flag, p.status, kStatusTimeoutMma);
        for (int i = first; ok && i < end; ++i) {
          ok = mbar_wait_warp(&full[s], phase, abort_flag, p.status, kStatusTimeoutMma);
          if (!ok) break;
          tc_fence_after();
          umma_f16_block_pair(tmem_base + buf * BT, a_desc0 + uint64_t(s) * kStageStep, b_desc0 + uint64_t(s) * kStageStep, idesc,
                              i > first ? 1u : 0u, empty_addr + s * 8, i + 1 == end ? acc_full_addr + buf * 8 : 0u);
          if (++s == Cfg::kStages) { s = 0; phase ^= 1u; }
        }
        if (++buf == Cfg::kAcc) { buf = 0; acc_phase ^= 1u; }
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3, half = (warp - 4) >> 2;
    float* turn = turn_all + (warp - 4) * (16 * 32);
    const uint32_t acc_empty_leader = map_to_cta(acc_empty, 0);
    const int width = dense_is_glu(p.epi.kind) ? 16 : 8, per = 32 / width, items = 16 * per;  // items of a 16-token chunk
    uint32_t buf = 0, phase = 0;
    bool ok = true;
    for (int tile = cluster; ok && tile < tiles_total; tile += clusters) {
      const int n0 = tile_n0(tile) + q * 32, t0 = tile_t0(tile) + half * (BT / 2);
      uint32_t after = buf, after_phase = phase;  // past the parts of this tile, at most kAcc of them
      for (int z = 0; ok && z < parts; ++z) {
        ok = mbar_wait_warp(&acc_full[after], after_phase, abort_flag, p.status, kStatusTimeoutEpilogue);
        if (++after == Cfg::kAcc) { after = 0; after_phase ^= 1u; }
      }
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + half * (BT / 2);
      for (int c = 0; c < BT / 2; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(taddr + buf * BT + c, r);
        tmem_wait_ld();
        if constexpr (kParts) {
          float sum[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) sum[j] = 0.f + __uint_as_float(r[j]);
          for (int z = 1; z < parts; ++z) {
            tmem_ld_32x16(taddr + (buf + z) % Cfg::kAcc * BT + c, r);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) sum[j] += __uint_as_float(r[j]);
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(sum[j]);
        }
        __syncwarp();  // the chunk before has been read
#pragma unroll
        for (int j = 0; j < 16; ++j) turn[j * 32 + lane] = __uint_as_float(r[j]);
        __syncwarp();
        for (int i = lane; i < items; i += 32) {
          const int j = i / per, n = (i - j * per) * width, t = t0 + c + j;
          if (t < p.M && n0 + n < p.N)
            dense_store_item<__nv_bfloat16>(p.epi, t, n0 + n, [&](int row, float(&v)[8]) { load8<float>(turn + j * 32 + row - n0, v); });
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0)
        for (int z = 0; z < parts; ++z) mbar_arrive_cluster(acc_empty_leader + (buf + z) % Cfg::kAcc * 8);
      buf = after;
      phase = after_phase;
    }
  }

  // ----- teardown: every thread of both CTAs arrives here, also after an aborted wait; nobody leaves (and frees
  //       memory the peer's tensor core may still read) before the other has finished -----
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

template <int BT, bool kParts>
int launch_dense_pair(const DensePairParams& p, const void* w, const void* x, int ldx, cudaStream_t stream) {
  using Cfg = DensePairCfg<BT>;
  CUtensorMap tw, tx;
  if (make_tmap_2d(&tw, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.N, p.K, uint64_t(p.K) * 2, kRows, kBK)) return -2;
  if (make_tmap_2d(&tx, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.M, p.K, uint64_t(ldx) * 2, BT / 2, kBK)) return -3;
  static bool attr_set[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -6;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(dense_pair_kernel<BT, kParts>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess) return -6;
    attr_set[dev] = true;
  }
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (p.N + 2 * kRows - 1) / (2 * kRows) * ((p.M + BT - 1) / BT);
  launch_kernel(dense_pair_kernel<BT, kParts>, dim3(2 * (tiles < sms / 2 ? tiles : sms / 2)), dim3(Cfg::kThreads), Cfg::kSmemBytes, stream, tw, tx, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

}  // namespace
}  // namespace mfq

// The plain form of mfq_dense_linear (one matrix, bf16, checked there) on CTA pairs; token_tile 128 or 256.  parts: sums along K, as
// many as there are accumulators (2 with the tile of 256, 4 with 128).
extern "C" int mfq_dense_pair(const void* w, const void* x, int ldx, void* out, int ldo, const float* bias, int M, int N, int K, int epilogue,
                              float alpha, float limit, const void* table, const int* ids, int token_tile, int parts, int* status, cudaStream_t stream) {
  using namespace mfq;
  if ((token_tile != 128 && token_tile != 256) || parts < 1 || parts > 512 / token_tile) return -1;
  const int nkb = (K + kBK - 1) / kBK, per_part = (nkb + parts - 1) / parts;
  const DensePairParams p{DenseEpilogue{epilogue, bias, alpha, limit, table, ids, out, ldo}, status, M, N, K, per_part};
  if (per_part < nkb) return token_tile == 128 ? launch_dense_pair<128, true>(p, w, x, ldx, stream) : launch_dense_pair<256, true>(p, w, x, ldx, stream);
  return token_tile == 128 ? launch_dense_pair<128, false>(p, w, x, ldx, stream) : launch_dense_pair<256, false>(p, w, x, ldx, stream);
}
