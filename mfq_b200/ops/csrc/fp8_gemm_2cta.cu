// Block-scaled FP8 GEMM for wide batches on PAIRS of SMs:  out[M, N] = X[M, K] * W[N, K]^T  (prefill shapes)
//
// The one-CTA kernel (fp8_gemm.cu) streams 32 KB of operands from L2 per 128 x 128 x 128 block of products.  Here two CTAs of a
// cluster work on one 256 x BT tile with `tcgen05.mma.cta_group::2`: each CTA stages ITS 128 weight rows (UMMA A operand, M = 256
// over the pair) and only HALF of the BT token rows (B operand, N = BT: the tensor core reads the other half from the peer CTA's
// shared memory), so a CTA loads 16 KB + BT/2 * 128 B per K block for 128 x BT x 128 products: 1.33x (BT = 128) and 2x (BT = 256)
// the products per byte of the one-CTA kernel.
//
// Roles per CTA: warp 0 = TMA producer, warp 1 = TMEM owner (and, in the leader CTA only, the MMA issuer), warps 2, 3
// idle (they complete the control warp group, which gives its registers away with `setmaxnreg`), warps 4..11 =
// epilogue (TMEM lane quarter = warp % 4, two warps per quarter split the token columns).  As in the one-CTA kernel
// every 128-wide K block lands in a fresh TMEM accumulator and the epilogue folds it, times the block's fp32
// multiplier, into registers while the tensor cores run the next block.  Cross-CTA signalling:
//   full[s]      lives in the leader; both CTAs' TMA loads complete their bytes on it (`.cta_group::2` loads may
//                signal the peer's barrier), the leader's producer arms it with the bytes of BOTH CTAs;
//   empty[s]     one per CTA; one commit of the leader arrives on both after the MMAs of the stage;
//   acc_full[b]  one per CTA, same; acc_empty[b] lives in the leader and counts the epilogue warps of both CTAs (the
//                peer's arrive through the cluster address of the leader's barrier).
// What bounds it: a K block is 512 cycles of tensor-core work (BT = 256) and the loop  issue -> complete -> fold -> hand back ->
// issue  has to fit twice that, TMEM holding two accumulators.  So the issuing and loading warps run converged with one elected
// lane (common.cuh: umma_f8f6f4_block says why), the fold keeps the TMEM load of one 32-column chunk in flight under the
// multiply-adds (two per instruction) of the chunk before, an accumulator is handed back as soon as its last column is in
// registers, and the epilogue looks at its next barrier one step ahead.  Measured on a B200 (operands rotated over more than the
// L2, before: this kernel as it was with one issuing lane and cluster-scope releases | the one-SM kernel | now):
//   4096 x 28672 x 4096   1084 (BT = 256) | 1096 | 593 us (1.62 PFLOP/s)     4096 x 4096 x 14336   550 | 420 | 252 us (1.91 PFLOP/s)
//   357 x 28672 x 4096     115 (one-SM)          | 62 us                     357 x 4096 x 14336     89 (one-SM) | 39 us
// Without the fold the same loads and MMAs run at 2.3 to 3.1 PFLOP/s, without the loads the fold and its hand-shakes at 2.1.
// The kernel is persistent: one pair per two SMs walks the tiles, all roles with continuing barrier phases, so a tile's
// prologue (first loads) and epilogue (store) hide under its neighbours' main loops; with one tile per launched CTA
// the fixed cost per tile was ~9 us of a 23 us tile at K = 4096.
// No load is multicast; the pair shares the token tile through the tensor core's own peer read.
// All waits are bounded; a cluster barrier before the TMEM release keeps a CTA alive while its peer may still read it.
//
// The reference has no FP8 tensor-core path (mfq/kernels/cuda/fp8_sq.cu:564-592 decodes to fp16 for wmma / cuBLAS).
#include "pair.cuh"

namespace mfq {
namespace {

constexpr int kRows = 128;    // weight rows per CTA
constexpr int kBK = 128;      // fp8 elements per K block

template <int BT>
struct PairCfg {
  static constexpr int kStages = 6;
  static constexpr int kAcc = 512 / BT;  // accumulators of BT columns: all of TMEM
  static constexpr int kStageBytes = kRows * kBK + (BT / 2) * kBK;
  static constexpr int kEpiWarps = 8;
  static constexpr int kCols = BT / 2;   // token columns per epilogue thread
  static constexpr int kThreads = 128 + 32 * kEpiWarps;  // warp group 0: TMA, MMA and two idle warps; groups 1, 2: epilogue
  static constexpr int kWsMax = 256;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256 + kEpiWarps * kCols * 4 + kEpiWarps * kWsMax * 4;
  static constexpr int kSumBytes = kCols * kEpiWarps * 32 * 4;  // running totals of split sums
};

struct PairParams {
  const float* w_scale;
  const float* x_scale;
  __nv_bfloat16* out;
  const __nv_bfloat16* residual;
  int* status;
  int M, N, K;
  int kb_per_split;  // split sums: K blocks of a partial sum
};

// kSplitSums: every kb_per_split K blocks are summed on their own and the partial sums added in order -- what the one-SM kernel's split-K
// form does, so that a product gives the same bits on either kernel.
template <int BT, bool kSplitSums>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<BT>::kThreads, 1)
fp8_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                     const PairParams p) {
  using Cfg = PairCfg<BT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + Cfg::kStages * Cfg::kStageBytes);
  uint64_t* full = bars;                       // used in the leader only
  uint64_t* empty = bars + Cfg::kStages;       // one set per CTA
  uint64_t* acc_full = bars + 2 * Cfg::kStages;
  uint64_t* acc_empty = acc_full + Cfg::kAcc;  // used in the leader only
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + Cfg::kAcc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* xs_smem = reinterpret_cast<float*>(tiles + Cfg::kStages * Cfg::kStageBytes + 256);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();  // 0 = leader
  const bool leader = rank == 0;
  const int nkb = p.K / kBK;
  // Persistent: the pair walks the tiles  cluster, cluster + #clusters, ...; a tile = (pair of weight-row blocks,
  // token tile), token tiles innermost so that pairs running at the same time share the weight rows in L2.  Every
  // role runs the same tile loop with barrier phases that simply continue, so the loads and MMAs of the next tile
  // start while the epilogue warps still store the previous one.
  const int clusters = int(gridDim.x) / 2, cluster = int(blockIdx.x) / 2;
  const int t_tiles = (p.M + BT - 1) / BT, n_pairs = p.N / (2 * kRows);
  const int tiles_total = t_tiles * n_pairs;
  auto tile_n0 = [&](int tile) { return (tile / t_tiles) * 2 * kRows + int(rank) * kRows; };  // this CTA's weight rows
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
  // The register file is the scarce resource of the fold: the control warp group hands its registers to the epilogue
  // groups, which then hold a thread's accumulators plus two chunks of raw columns.
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
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
        tma_load_stage_pair(a, a + kRows * kBK, &tmap_w, &tmap_x, full_leader + s * 8, full_local + s * 8, bytes, i * kBK, n0, t0);
        if (++s == Cfg::kStages) { s = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1 && leader) {
    constexpr uint32_t idesc = umma_idesc(2 * kRows, BT, 0, 0);
    constexpr uint64_t kStageStep = uint64_t(Cfg::kStageBytes >> 4);
    const uint64_t a_desc0 = umma_desc_k_sw128(smem_u32(tiles)), b_desc0 = umma_desc_k_sw128(smem_u32(tiles) + kRows * kBK);
    const uint32_t empty_addr = smem_u32(empty), acc_full_addr = smem_u32(acc_full);
    int s = 0;
    uint32_t phase = 0, buf = 0, acc_phase = 1;  // the first pass over the accumulators finds them free
    bool ok = true;
    for (int tile = cluster; ok && tile < tiles_total; tile += clusters) {
      for (int i = 0; i < nkb; ++i) {
        ok = mbar_wait_warp(&acc_empty[buf], acc_phase, abort_flag, p.status, kStatusTimeoutMma) &&
             mbar_wait_warp(&full[s], phase, abort_flag, p.status, kStatusTimeoutMma);
        if (!ok) break;
        tc_fence_after();
        umma_f8f6f4_block_pair(tmem_base + buf * BT, a_desc0 + uint64_t(s) * kStageStep, b_desc0 + uint64_t(s) * kStageStep, idesc, 0u,
                               empty_addr + s * 8, acc_full_addr + buf * 8);
        if (++s == Cfg::kStages) { s = 0; phase ^= 1u; }
        if (++buf == Cfg::kAcc) { buf = 0; acc_phase ^= 1u; }
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    pdl_wait();
    // ----- epilogue warps: thread owns weight row n0 + q*32 + lane and CW token columns from col0 -----
    constexpr int CW = Cfg::kCols;
    constexpr int kChunks = CW / 32;
    const int q = warp & 3;
    const int col0 = ((warp - 4) >> 2) * CW;
    const int row = q * 32 + lane;
    float* xs_w = xs_smem + (warp - 4) * CW;
    float* ws_w = xs_smem + Cfg::kEpiWarps * CW + (warp - 4) * Cfg::kWsMax;
    const bool ws_cached = nkb <= Cfg::kWsMax;
    float* totals = xs_smem + Cfg::kEpiWarps * (CW + Cfg::kWsMax) + (threadIdx.x - 128);  // kSplitSums only: this thread's column of the totals
    const uint32_t acc_empty_leader0 = map_to_cta(&acc_empty[0], 0);
    const uint32_t lane_base = tmem_base + (uint32_t(q * 32) << 16) + col0;
    bool ok = true, ready = false;
    uint32_t buf = 0, phase = 0;
    for (int tile = cluster; ok && tile < tiles_total; tile += clusters) {
      const int n0 = tile_n0(tile), t0 = tile_t0(tile);
      const int n = n0 + row;
      float acc[CW];
#pragma unroll
      for (int tt = 0; tt < CW; ++tt) acc[tt] = 0.f;
      const float* wsc = p.w_scale + size_t(n0 / kRows) * nkb;
      __syncwarp();  // the previous tile's reads of this warp's slices are done
      for (int j = lane; j < CW; j += 32) xs_w[j] = (t0 + col0 + j < p.M) ? p.x_scale[t0 + col0 + j] : 0.f;  // no __ldg: written since this grid began
      if (ws_cached)
        for (int j = lane; j < nkb; j += 32) ws_w[j] = __ldg(wsc + j);
      __syncwarp();
      // Split sums: the total of the splits done so far waits in shared memory, [column][thread].  It is touched once per split; held in
      // registers beside the running sum it takes half of what a thread has (357 x 4096 x 4096: 19.8 us, from here 16.6).
      int left = p.kb_per_split;
      bool started = false;
      auto add_total = [&](int tt) { return started ? totals[tt * (Cfg::kEpiWarps * 32)] + acc[tt] : 0.f + acc[tt]; };
      for (int i = 0; i < nkb; ++i) {
        if constexpr (kSplitSums) {
          if (left == 0) {
#pragma unroll
            for (int tt = 0; tt < CW; ++tt) {
              totals[tt * (Cfg::kEpiWarps * 32)] = add_total(tt);
              acc[tt] = 0.f;
            }
            started = true;
            left = p.kb_per_split;
          }
          --left;
        }
        if (!ready) ok = mbar_wait_warp(&acc_full[buf], phase, abort_flag, p.status, kStatusTimeoutEpilogue);
        if (!ok) break;
        tc_fence_after();
        const float s = ws_cached ? ws_w[i] : __ldg(wsc + i);
        const uint32_t taddr = lane_base + buf * BT;
        uint32_t r[2][32];
        tmem_ld_32x32(taddr, r[0]);
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          tmem_wait_ld();
          if (c + 1 < kChunks) {
            tmem_ld_32x32(taddr + (c + 1) * 32, r[(c + 1) & 1]);
          } else {  // all columns of this block are in registers: hand the accumulator back, look at the next one
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(acc_empty_leader0 + buf * 8);
            if (++buf == Cfg::kAcc) { buf = 0; phase ^= 1u; }
            ready = mbar_test_warp(&acc_full[buf], phase);
          }
#pragma unroll
          for (int j = 0; j < 32; j += 2) fma2(acc[c * 32 + j], acc[c * 32 + j + 1], r[c & 1][j], r[c & 1][j + 1], s);
        }
      }
      if constexpr (kSplitSums) {
#pragma unroll
        for (int tt = 0; tt < CW; ++tt) acc[tt] = add_total(tt);
      }
      if (ok && n < p.N) {
        const int tl = min(BT, p.M - t0);
        // residual and output may be one buffer: all loads first, or every load would wait behind the store before it
        if (p.residual) {
          unsigned short res[CW];
          const unsigned short* rp = reinterpret_cast<const unsigned short*>(p.residual);
#pragma unroll
          for (int tt = 0; tt < CW; ++tt)
            res[tt] = (col0 + tt < tl) ? __ldcg(rp + size_t(t0 + col0 + tt) * p.N + n) : (unsigned short)0;
// the roundings of the one-SM kernel: product and sum in one where its splits meet in a cluster (up to 8), else one by one
          const bool fused = kSplitSums && (nkb + p.kb_per_split - 1) / p.kb_per_split <= 8;
#pragma unroll
          for (int tt = 0; tt < CW; ++tt) {
            const float add = __uint_as_float(uint32_t(res[tt]) << 16);
            acc[tt] = fused ? __fmaf_rn(acc[tt], xs_w[tt], add) : __fadd_rn(__fmul_rn(acc[tt], xs_w[tt]), add);
          }
        } else {
#pragma unroll
          for (int tt = 0; tt < CW; ++tt) acc[tt] *= xs_w[tt];
        }
#pragma unroll
        for (int tt = 0; tt < CW; ++tt) {
          if (col0 + tt < tl) p.out[size_t(t0 + col0 + tt) * p.N + n] = __float2bfloat16(acc[tt]);
        }
      }
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

template <int BT, bool kSplitSums>
int launch_pair(const void* w, const float* w_scale, const void* x, const float* x_scale, void* out, const void* residual,
                int* status, int M, int N, int K, int kb_per_split, cudaStream_t stream) {
  using Cfg = PairCfg<BT>;
  CUtensorMap tw, tx;
  if (make_tmap_2d(&tw, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K, K, kRows, kBK)) return -2;
  if (make_tmap_2d(&tx, x, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, M, K, K, BT / 2, kBK)) return -3;
  constexpr int smem = Cfg::kSmemBytes + (kSplitSums ? Cfg::kSumBytes : 0);
  static bool attr_set[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -6;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(fp8_gemm_pair_kernel<BT, kSplitSums>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return -6;
    attr_set[dev] = true;
  }
  PairParams p{w_scale, x_scale, static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(residual), status, M, N, K, kb_per_split};
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (N / (2 * kRows)) * ((M + BT - 1) / BT);
  const int clusters = tiles < sms / 2 ? tiles : sms / 2;
  launch_kernel(fp8_gemm_pair_kernel<BT, kSplitSums>, dim3(2 * clusters), dim3(Cfg::kThreads), smem, stream, tw, tx, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

}  // namespace
}  // namespace mfq

// Two-SM form of mfq_fp8_gemm for wide batches.  N % 256 == 0, K % 128 == 0, token_tile in {128, 256}; no split-K.  kb_per_split > 0
// (tile 128): the sums are formed as by mfq_fp8_gemm with that many K blocks per split, bit for bit.
extern "C" int mfq_fp8_gemm_pair(const void* w, const float* w_scale, const void* x, const float* x_scale, void* out,
                                 const void* residual, int* status, int M, int N, int K, int token_tile, int kb_per_split,
                                 cudaStream_t stream) {
  if (K % 128 != 0 || N % 256 != 0 || M <= 0 || kb_per_split < 0 || (kb_per_split && token_tile != 128)) return -1;
  if (kb_per_split) return mfq::launch_pair<128, true>(w, w_scale, x, x_scale, out, residual, status, M, N, K, kb_per_split, stream);
  if (token_tile == 128) return mfq::launch_pair<128, false>(w, w_scale, x, x_scale, out, residual, status, M, N, K, 0, stream);
  if (token_tile == 256) return mfq::launch_pair<256, false>(w, w_scale, x, x_scale, out, residual, status, M, N, K, 0, stream);
  return -1;
}
