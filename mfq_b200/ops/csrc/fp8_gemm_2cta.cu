// Block-scaled FP8 GEMM for wide batches on PAIRS of SMs:  out[M, N] = X[M, K] * W[N, K]^T  (prefill shapes)
//
// The one-CTA kernel (fp8_gemm.cu) streams 32 KB of operands from L2 per 128 x 128 x 128 block of products.  Here two CTAs of a
// cluster work on one 256 x BT tile with `tcgen05.mma.cta_group::2`: each CTA stages ITS 128 rows of the A operand (M = 256
// over the pair) and only HALF of the BT rows of B (N = BT: the tensor core reads the other half from the peer CTA's
// shared memory), so a CTA loads 16 KB + BT/2 * 128 B per K block for 128 x BT x 128 products: 1.33x (BT = 128) and 2x (BT = 256)
// the products per byte of the one-CTA kernel.  With BT = 256 the tokens are A, so that a thread of the epilogue holds 128 weight rows
// of one token; with BT = 128 the weights are, so that tokens come in tiles of 128 and fewer are padding.
//
// Roles per CTA: warp 0 = TMA producer, warp 1 = TMEM owner and, in the leader CTA only, MMA issuer, warp 2 = residual and output copies,
// warp 3 = multipliers of the next tile, warps 4..11 = epilogue (TMEM lane quarter = warp % 4, two warps per quarter split the columns).
// The control warp group gives its registers away with `setmaxnreg`.  As in the one-CTA kernel
// every 128-wide K block lands in a fresh TMEM accumulator and the epilogue folds it, times the block's fp32
// multiplier, into registers while the tensor cores run the next block.  Cross-CTA signalling:
//   full[s]      lives in the leader; both CTAs' TMA loads complete their bytes on it (`.cta_group::2` loads may
//                signal the peer's barrier), the leader's producer arms it with the bytes of BOTH CTAs;
//   empty[s]     one per CTA; one commit of the leader arrives on both after the MMAs of the stage;
//   acc_full[b]  one per CTA, same; acc_empty[b] lives in the leader and counts the epilogue warps of both CTAs (the
//                peer's arrive through the cluster address of the leader's barrier).
// What bounds it: a K block is 512 cycles of tensor-core work (BT = 256) and, TMEM holding two accumulators, the way from the end of an
// MMA over the fold to the next MMA on the same accumulator has to fit into that.  So the epilogue warps do nothing but fold: a residual
// arrives by TMA under the main loop and the results leave by TMA under the next tile's, both at warp 2's hand, through a swizzled place
// in shared memory; multipliers are laid there by warp 3; tiles are walked without divisions; the split sums have a loop of their own
// around the fold.  Every condition inside the loop costs: asking there once per tile for the residual took 4 % (BT = 256) and 8 %
// (BT = 128).  Sixteen epilogue warps of 64 columns were 12 % slower than eight of 128, loads of the next block ahead of the last
// multiply-adds of this one 8 % slower.  Measured on a B200 (operands rotated over more than the L2; before: loads, roundings and 2-byte
// stores of a tile by the epilogue warps between two tiles):
//   4096 x 28672 x 4096 531 -> 402 us (2.39 PFLOP/s)     4096 x 4096 x 14336 with residual 311 -> 220     4096 x 4096 x 4096 with residual
//   173 -> 75     1000 x 28672 x 4096 167 -> 114     357 x 28672 x 4096 (BT = 128) 68 -> 59     357 x 4096 x 14336 in three sums 40 -> 32
// A K block takes 750 cycles there at 1.7 GHz (power), a tile 2700 between its last block and the next one's first.
// The kernel is persistent: one pair per two SMs walks the tiles, all roles with continuing barrier phases.
// No load is multicast; the pair shares operand B through the tensor core's own peer read.
// All waits are bounded; a cluster barrier before the TMEM release keeps a CTA alive while its peer may still read it.
//
// The reference has no FP8 tensor-core path (mfq/kernels/cuda/fp8_sq.cu:564-592 decodes to fp16 for wmma / cuBLAS).
#include <type_traits>

#include "pair.cuh"

namespace mfq {
namespace {

constexpr int kRows = 128;  // rows of the A operand per CTA
constexpr int kBK = 128;    // fp8 elements per K block

template <int BT, bool kSplitSums>
struct PairCfg {
  static constexpr bool kTokenRows = BT == 256;  // A = tokens, B = weights; else A = weights, B = tokens
  static constexpr int kStages = BT == 128 ? 6 : 4;
  static constexpr int kAcc = 512 / BT;  // accumulators of BT columns: all of TMEM
  static constexpr int kStageBytes = kRows * kBK + (BT / 2) * kBK;
  static constexpr int kEpiWarps = 8;
  static constexpr int kCols = BT / 2;   // accumulator columns per epilogue thread
  static constexpr int kThreads = 128 + 32 * kEpiWarps;  // warp group 0: TMA, MMA, output places, multipliers; groups 1, 2: epilogue
  static constexpr int kWsMax = 256;
  // Output places: 32 tokens x 128 weight rows of one warp (kTokenRows), else 64 tokens x 64 weight rows of two.
  static constexpr int kPlaces = kTokenRows ? kEpiWarps : kEpiWarps / 2, kPlaceWarps = kEpiWarps / kPlaces, kPlaceBytes = 8192;
  static constexpr int kBoxRows = kTokenRows ? 32 : 64;  // tokens of a bulk copy, 64 weight rows wide
  static constexpr int kXsCols = kTokenRows ? 0 : BT;
  static constexpr int kMulFloats = kXsCols + (kTokenRows ? 2 : 1) * kWsMax;  // multipliers of a tile: of its tokens, of its blocks of rows
  // Running totals of split sums, [column][lane] per warp.  The first kPlaceCols columns lie in the warp's share of the output place, which
  // residual and results then enter only after both warps have read the last of them.
  static constexpr int kPlaceCols = kPlaceBytes / kPlaceWarps / 128, kSumBytes = kSplitSums ? (kCols - kPlaceCols) * kEpiWarps * 32 * 4 : 0;
  static constexpr int kTurnAt = kStages * kStageBytes, kBarsAt = kTurnAt + kPlaces * kPlaceBytes, kMulAt = kBarsAt + 512;
  static constexpr int kSumAt = kMulAt + 2 * kMulFloats * 4;
  static constexpr int kSmemBytes = kSumAt + kSumBytes;
};

struct PairParams {
  const float* w_scale;
  const float* x_scale;
  __nv_bfloat16* out;
  const __nv_bfloat16* residual;
  int* status;
  int M, N, K;
  int kb_per_split;  // split sums: K blocks of a partial sum
  int direct;        // output or residual off a 16-byte boundary: plain loads and stores
};

// kSplitSums: every kb_per_split K blocks are summed on their own and the partial sums added in order -- what the one-SM kernel's split-K
// form does, so that a product gives the same bits on either kernel.
template <int BT, bool kSplitSums>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<BT, kSplitSums>::kThreads, 1)
fp8_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ CUtensorMap tmap_res, const PairParams p) {
  using Cfg = PairCfg<BT, kSplitSums>;
  constexpr bool kTok = Cfg::kTokenRows;
  extern __shared__ __align__(1024) uint8_t tiles[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + Cfg::kBarsAt);
  uint64_t* full = bars;                       // used in the leader only
  uint64_t* empty = bars + Cfg::kStages;       // one set per CTA
  uint64_t* acc_full = bars + 2 * Cfg::kStages;
  uint64_t* acc_empty = acc_full + Cfg::kAcc;  // used in the leader only
  uint64_t* turn_ready = acc_empty + Cfg::kAcc;           // one per output place: it holds the residual, or is free
  uint64_t* turn_done = turn_ready + Cfg::kPlaces;        // ... and holds the results
  uint64_t* mul_full = turn_done + Cfg::kPlaces;          // multipliers, two tiles of them
  uint64_t* mul_empty = mul_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mul_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  float* mul = reinterpret_cast<float*>(tiles + Cfg::kMulAt);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();  // 0 = leader
  const bool leader = rank == 0;
  const int nkb = p.K / kBK;
  // Persistent: the pair walks the tiles  cluster, cluster + #clusters, ...; a tile = (pair of weight-row blocks,
  // token tile), token tiles innermost so that pairs running at the same time share the weight rows in L2.  Every
  // role runs the same tile loop with barrier phases that simply continue, so the loads and MMAs of the next tile
  // start while the epilogue warps still store the previous one.
  const int clusters = int(gridDim.x) / 2, cluster = int(blockIdx.x) / 2;
  const int t_tiles = (p.M + BT - 1) / BT, tiles_total = t_tiles * (p.N / (2 * kRows));
  struct Place {  // of a tile, carried along: a division per tile and role costs as much as half a K block
    int tile, n, t;
  };
  const int step_n = clusters / t_tiles, step_t = clusters % t_tiles;
  auto next_place = [&](Place at) {
    at = Place{at.tile + clusters, at.n + step_n, at.t + step_t};
    if (at.t >= t_tiles) at.t -= t_tiles, ++at.n;
    return at;
  };
  const Place first = {cluster, cluster / t_tiles, cluster % t_tiles};
  // first weight row and token of an output place
  constexpr int CW = Cfg::kCols;
  auto place_n0 = [&](const Place& at, int u) { return at.n * (2 * kRows) + (kTok ? (u >> 2) * kRows : int(rank) * kRows + (u & 1) * 64); };
  auto place_t0 = [&](const Place& at, int u) { return at.t * BT + (kTok ? int(rank) * kRows + (u & 3) * 32 : (u >> 1) * 64); };
  const bool with_res = p.residual && !p.direct;
  const bool ws_cached = nkb <= Cfg::kWsMax;

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < Cfg::kAcc; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 2 * Cfg::kEpiWarps); }
    for (int i = 0; i < Cfg::kPlaces; ++i) { mbar_init(&turn_ready[i], 1); mbar_init(&turn_done[i], Cfg::kPlaceWarps); }
    for (int i = 0; i < 2; ++i) { mbar_init(&mul_full[i], 32); mbar_init(&mul_empty[i], Cfg::kEpiWarps); }
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
  // groups, which then hold a thread's accumulators plus two chunks of raw columns (with 256 tokens all but 44 bytes of it).
  if (warp < 4) {
  if constexpr (kTok) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  else asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
  if (warp != 0) pdl_wait();
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_a);
      tma_prefetch_desc(&tmap_b);
    }
    __syncwarp();
    const uint32_t tiles_addr = smem_u32(tiles), full_local = smem_u32(full), full_leader = map_to_cta(full, 0);
    const uint32_t bytes = leader ? 2u * Cfg::kStageBytes : 0u;  // the bytes of both CTAs land on the leader's barrier
    const CUtensorMap* map_w = kTok ? &tmap_b : &tmap_a;
    const CUtensorMap* map_x = kTok ? &tmap_a : &tmap_b;
    constexpr int kWRows = kTok ? BT / 2 : kRows, kXRows = kTok ? kRows : BT / 2, kWAt = kTok ? kRows * kBK : 0, kXAt = kTok ? 0 : kRows * kBK;
    // Weights are never written by a kernel of the same stream: those of the first ring pass leave before the wait for the kernel before.
    const int ahead = min(nkb, Cfg::kStages);
    for (int i = 0; i < ahead; ++i)
      tma_load_pair(tiles_addr + i * Cfg::kStageBytes + kWAt, map_w, full_leader + i * 8, full_local + i * 8, bytes, i * kBK, first.n * (2 * kRows) + int(rank) * kWRows);
    pdl_wait();
    for (int i = 0; i < ahead; ++i)
      tma_load_pair(tiles_addr + i * Cfg::kStageBytes + kXAt, map_x, full_leader + i * 8, full_local + i * 8, 0u, i * kBK, first.t * BT + int(rank) * kXRows);
    int s = ahead % Cfg::kStages, i0 = ahead;
    uint32_t phase = ahead == Cfg::kStages ? 1u : 0u;
    bool ok = true;
    for (Place at = first; ok && at.tile < tiles_total; at = next_place(at), i0 = 0) {
      const int w0 = at.n * (2 * kRows) + int(rank) * kWRows, x0 = at.t * BT + int(rank) * kXRows;
      for (int i = i0; i < nkb; ++i) {
        ok = mbar_wait_warp(&empty[s], phase ^ 1u, abort_flag, p.status, kStatusTimeoutProducer);
        if (!ok) break;
        const uint32_t a = tiles_addr + s * Cfg::kStageBytes;
        tma_load_stage_pair(a + kWAt, a + kXAt, map_w, map_x, full_leader + s * 8, full_local + s * 8, bytes, i * kBK, w0, x0);
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
        // the operands first: they are there long before the accumulator, and looking at a barrier takes over a hundred cycles
        ok = mbar_wait_warp(&full[s], phase, abort_flag, p.status, kStatusTimeoutMma) &&
             mbar_wait_warp(&acc_empty[buf], acc_phase, abort_flag, p.status, kStatusTimeoutMma);
        if (!ok) break;
        tc_fence_after();
        umma_f8f6f4_block_pair(tmem_base + buf * BT, a_desc0 + uint64_t(s) * kStageStep, b_desc0 + uint64_t(s) * kStageStep, idesc, 0u,
                               empty_addr + s * 8, acc_full_addr + buf * 8);
        if (++s == Cfg::kStages) { s = 0; phase ^= 1u; }
        if (++buf == Cfg::kAcc) { buf = 0; acc_phase ^= 1u; }
      }
    }
  } else if (warp == 2 && !p.direct && lane < Cfg::kPlaces) {
    // a lane per output place: the residual to it, the results from there
    uint8_t* place = tiles + Cfg::kTurnAt + lane * Cfg::kPlaceBytes;
    constexpr int kSlabBytes = Cfg::kBoxRows * 128;
    uint32_t phase = 0;
    bool ok = true;
    for (Place at = first; ok && at.tile < tiles_total; at = next_place(at)) {
      const int n0 = place_n0(at, lane), t0 = place_t0(at, lane);
      if (t0 >= p.M) continue;
      if constexpr (kSplitSums) {
        mbar_arrive(&turn_ready[lane]);  // the store before has read its source: sums may be put there
        ok = mbar_wait(&turn_done[lane], phase, abort_flag, p.status, kStatusTimeoutEpilogue);  // ... and have been read, by both warps
        phase ^= 1u;
        if (!ok) break;
      }
      if (with_res) {
        mbar_expect_tx(&turn_ready[lane], Cfg::kPlaceBytes);
        for (int c = 0; c < Cfg::kPlaceBytes / kSlabBytes; ++c) tma_load_2d(place + c * kSlabBytes, &tmap_res, &turn_ready[lane], n0 + c * 64, t0);
      } else {
        mbar_arrive(&turn_ready[lane]);
      }
      ok = mbar_wait(&turn_done[lane], phase, abort_flag, p.status, kStatusTimeoutEpilogue);
      phase ^= 1u;
      if (ok) {
        for (int c = 0; c < Cfg::kPlaceBytes / kSlabBytes; ++c) tma_store_2d(&tmap_out, smem_u32(place) + c * kSlabBytes, n0 + c * 64, t0);
        bulk_commit();
        bulk_wait_read();
      }
    }
    bulk_wait();
  } else if (warp == 3) {
    // multipliers of the next tile to shared memory while this one is folded
    uint32_t side = 0, phase = 1;
    bool ok = true;
    for (Place at = first; ok && at.tile < tiles_total; at = next_place(at)) {
      ok = mbar_wait_warp(&mul_empty[side], phase, abort_flag, p.status, kStatusTimeoutEpilogue);
      if (!ok) break;
      float* to = mul + side * Cfg::kMulFloats;
      if constexpr (!kTok)
        for (int j = lane; j < BT; j += 32) to[j] = at.t * BT + j < p.M ? p.x_scale[at.t * BT + j] : 0.f;  // no __ldg: written since this grid began
      if (ws_cached) {
        const float* wsc = p.w_scale + size_t(2 * at.n + (kTok ? 0 : int(rank))) * nkb;
        for (int j = lane; j < nkb; j += 32) {
          to[Cfg::kXsCols + j] = __ldg(wsc + j);
          if constexpr (kTok) to[Cfg::kWsMax + j] = __ldg(wsc + nkb + j);
        }
      }
      mbar_arrive(&mul_full[side]);
      side ^= 1u;
      if (side == 0) phase ^= 1u;
    }
  }
  } else {
    if constexpr (kTok) asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    pdl_wait();
    // ----- epilogue warps: a thread owns row q*32 + lane of A (kTok: a token, else a weight row) and CW columns from col0 -----
    constexpr int kChunks = CW / 32;
    const int e = warp - 4, q = warp & 3;
    const int col0 = (e >> 2) * CW;
    const int unit = e / Cfg::kPlaceWarps;
    const uint32_t turn = smem_u32(tiles) + Cfg::kTurnAt + unit * Cfg::kPlaceBytes;
    auto total = [&](int tt) -> float& {  // kSplitSums
      uint8_t* at = tt < Cfg::kPlaceCols ? tiles + Cfg::kTurnAt + e * (Cfg::kPlaceBytes / Cfg::kPlaceWarps) + tt * 128
                                         : tiles + Cfg::kSumAt + (e * (CW - Cfg::kPlaceCols) + tt - Cfg::kPlaceCols) * 128;
      return reinterpret_cast<float*>(at)[lane];
    };
    const uint32_t acc_empty_leader0 = map_to_cta(&acc_empty[0], 0);
    const uint32_t lane_base = tmem_base + (uint32_t(q * 32) << 16) + col0;
    bool ok = true, ready = false;
    uint32_t buf = 0, phase = 0, side = 0, mul_phase = 0, turn_phase = 0;
    for (Place at = first; ok && at.tile < tiles_total; at = next_place(at)) {
      const int t0 = place_t0(at, unit);  // this thread's token (kTok: the one of lane 0), or the first of them
      const bool live = t0 < p.M && !p.direct;
      float acc[CW];
#pragma unroll
      for (int tt = 0; tt < CW; ++tt) acc[tt] = 0.f;
      float xs = 0.f;
      if constexpr (kTok) xs = t0 + lane < p.M ? p.x_scale[t0 + lane] : 0.f;  // no __ldg: written since this grid began
      ok = mbar_wait_warp(&mul_full[side], mul_phase, abort_flag, p.status, kStatusTimeoutEpilogue);
      if (!ok) break;
      const float* xs_w = mul + side * Cfg::kMulFloats + col0;  // !kTok
      // the multipliers of this thread's block of rows, wherever they are
      const float* ws_w = ws_cached ? mul + side * Cfg::kMulFloats + Cfg::kXsCols + (kTok ? (e >> 2) * Cfg::kWsMax : 0)
                                    : p.w_scale + size_t(2 * at.n + (kTok ? e >> 2 : int(rank))) * nkb;
      float s_next = ws_w[0];
      // Split sums: the total of the splits done so far waits in shared memory.  It is touched once per split; held in
      // registers beside the running sum it takes half of what a thread has (357 x 4096 x 4096: 19.8 us, from here 16.6).
      bool started = false;
      auto add_total = [&](int tt) { return started ? total(tt) + acc[tt] : 0.f + acc[tt]; };
      for (int i = 0, end = kSplitSums ? p.kb_per_split : nkb;;) {
        for (; i < end; ++i) {
          if (!ready) ok = mbar_wait_warp(&acc_full[buf], phase, abort_flag, p.status, kStatusTimeoutEpilogue);
          if (!ok) break;
          tc_fence_after();
          const float s = s_next;
          const uint32_t taddr = lane_base + buf * BT;
          uint32_t r[2][32];
          tmem_ld_32x32(taddr, r[0]);
          if (i + 1 < nkb) s_next = ws_w[i + 1];
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            tmem_wait_ld();
            if (c + 1 < kChunks) {
              tmem_ld_32x32(taddr + (c + 1) * 32, r[(c + 1) & 1]);
            } else {  // all columns of this block are in registers: hand the accumulator back, look at the next one
              tc_fence_before();
              __syncwarp();
              mbar_arrive_cluster_warp(acc_empty_leader0 + buf * 8);
              if (++buf == Cfg::kAcc) { buf = 0; phase ^= 1u; }
              ready = mbar_test_warp(&acc_full[buf], phase);
            }
#pragma unroll
            for (int j = 0; j < 32; j += 2) fma2(acc[c * 32 + j], acc[c * 32 + j + 1], r[c & 1][j], r[c & 1][j + 1], s);
          }
        }
        if (!ok || !kSplitSums || i == nkb) break;
        if (!started && live) {
          ok = mbar_wait_warp(&turn_ready[unit], turn_phase, abort_flag, p.status, kStatusTimeoutEpilogue);
          turn_phase ^= 1u;
          if (!ok) break;
        }
        if (live || p.direct) {  // else no result is asked for, and the store of the tile before may still read the place
#pragma unroll
          for (int tt = 0; tt < CW; ++tt) total(tt) = add_total(tt);
        }
#pragma unroll
        for (int tt = 0; tt < CW; ++tt) acc[tt] = 0.f;
        started = true;
        end = min(nkb, end + p.kb_per_split);
      }
      if constexpr (kSplitSums) {
#pragma unroll
        for (int tt = 0; tt < CW; ++tt) acc[tt] = add_total(tt);
        if (live && ok) {  // the place is the residual's and the results'; a row of them covers sums of both warps
          fence_proxy_async_smem();  // the residual comes by TMA where these sums were read and written by plain accesses
          __syncwarp();
          if (lane == 0) mbar_arrive(&turn_done[unit]);
        }
      }
      if (!ok) break;
      // the roundings of the one-SM kernel: product and sum in one where its splits meet in a cluster (up to 8), else one by one
      const bool fused = kSplitSums && (nkb + p.kb_per_split - 1) / p.kb_per_split <= 8;
      auto finish = [&](int tt, bool with, float add) {
        const float m = kTok ? xs : xs_w[tt];
        if (!with) return acc[tt] * m;
        return fused ? __fmaf_rn(acc[tt], m, add) : __fadd_rn(__fmul_rn(acc[tt], m), add);
      };
      if (t0 < p.M && p.direct) {
        const int n0 = place_n0(at, unit) + (kTok ? 0 : (e & 1) * 32 + lane);
#pragma unroll
        for (int tt = 0; tt < CW; ++tt) {
          const int t = t0 + (kTok ? lane : tt), n = n0 + (kTok ? tt : 0);
          if (t < p.M) {
            const size_t to = size_t(t) * p.N + n;
            p.out[to] = __float2bfloat16(finish(tt, p.residual != nullptr, p.residual ? __bfloat162float(p.residual[to]) : 0.f));
          }
        }
      } else if (live) {
        // Through shared memory, 128 swizzled bytes of 64 weight rows per token: the residual came there by TMA under the main loop, the
        // results take its place and leave by TMA under the next tile's.
        ok = mbar_wait_warp(&turn_ready[unit], turn_phase, abort_flag, p.status, kStatusTimeoutEpilogue);
        turn_phase ^= 1u;
        if (!ok) break;
        auto turn_in = [&](auto with) {
          if constexpr (kTok) {
#pragma unroll
            for (int c = 0; c < CW / 8; ++c) {
              const uint32_t place = turn + (c >> 3) * 4096 + lane * 128 + (((c & 7) ^ (lane & 7)) << 4);
              uint32_t v[4] = {0u, 0u, 0u, 0u};
              if constexpr (with) asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(place));
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const __nv_bfloat162 two = __floats2bfloat162_rn(finish(c * 8 + 2 * j, with, __uint_as_float(v[j] << 16)),
                                                                 finish(c * 8 + 2 * j + 1, with, __uint_as_float(v[j] & 0xffff0000u)));
                v[j] = *reinterpret_cast<const uint32_t*>(&two);
              }
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(place), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
            }
          } else {
            // A thread has one weight row of tokens t and t + 4.  Neighbours trade halves: an even lane gets its pair of rows of token t, an
            // odd one of token t + 4, whose four chunks of 16 bytes the swizzle puts beside those of token t: no bank is met twice.
            const bool odd = lane & 1;
            const uint32_t chunk = (e & 1) * 4 + (lane >> 3), within = ((lane >> 1) & 3) * 4;
#pragma unroll
            for (int tt = 0; tt < CW; tt += 8) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const uint32_t row = j + (odd ? 4 : 0);  // of the eight tokens
                const uint32_t place = turn + (tt + row) * 128 + ((chunk ^ row) << 4) + within;
                float add0 = 0.f, add4 = 0.f;
                if constexpr (with) {
                  uint32_t w;
                  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w) : "r"(place));
                  const uint32_t other = __shfl_xor_sync(0xffffffffu, w, 1);
                  add0 = __uint_as_float(odd ? other & 0xffff0000u : w << 16);
                  add4 = __uint_as_float(odd ? w & 0xffff0000u : other << 16);
                }
                const __nv_bfloat162 two = __floats2bfloat162_rn(finish(tt + j, with, add0), finish(tt + j + 4, with, add4));
                const uint32_t own = *reinterpret_cast<const uint32_t*>(&two), other = __shfl_xor_sync(0xffffffffu, own, 1);
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(place), "r"(__byte_perm(own, other, odd ? 0x3276 : 0x5410)) : "memory");
              }
            }
          }
        };
        if (with_res) turn_in(std::true_type{});
        else turn_in(std::false_type{});
        fence_proxy_async_smem();
      }
      __syncwarp();
      if (lane == 0) {
        if (live) mbar_arrive(&turn_done[unit]);
        mbar_arrive(&mul_empty[side]);
      }
      side ^= 1u;
      if (side == 0) mul_phase ^= 1u;
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
  using Cfg = PairCfg<BT, kSplitSums>;
  CUtensorMap ta, tb, to = {}, tr = {};
  const void *a = Cfg::kTokenRows ? x : w, *b = Cfg::kTokenRows ? w : x;
  const int a_rows = Cfg::kTokenRows ? M : N, b_rows = Cfg::kTokenRows ? N : M;
  if (make_tmap_2d(&ta, a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a_rows, K, K, kRows, kBK)) return -2;
  if (make_tmap_2d(&tb, b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, b_rows, K, K, BT / 2, kBK)) return -3;
  const bool direct = ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(residual)) & 15) != 0;
  if (!direct) {
    if (make_tmap_2d(&to, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, M, N, uint64_t(N) * 2, Cfg::kBoxRows, 64)) return -4;
    if (residual && make_tmap_2d(&tr, residual, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, M, N, uint64_t(N) * 2, Cfg::kBoxRows, 64)) return -5;
  }
  static bool attr_set[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -6;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(fp8_gemm_pair_kernel<BT, kSplitSums>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess)
      return -6;
    attr_set[dev] = true;
  }
  PairParams p{w_scale, x_scale, static_cast<__nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(residual), status, M, N, K, kb_per_split, direct};
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int tiles = (N / (2 * kRows)) * ((M + BT - 1) / BT);
  const int clusters = tiles < sms / 2 ? tiles : sms / 2;
  launch_kernel(fp8_gemm_pair_kernel<BT, kSplitSums>, dim3(2 * clusters), dim3(Cfg::kThreads), Cfg::kSmemBytes, stream, ta, tb, to, tr, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

}  // namespace
}  // namespace mfq

// Two-SM form of mfq_fp8_gemm for wide batches.  N % 256 == 0, K % 128 == 0, token_tile in {128, 256}; no split-K.  kb_per_split > 0
// (tile 128): the sums are formed as by mfq_fp8_gemm with that many K blocks per split, bit for bit.
extern "C" int mfq_fp8_gemm_pair(const void* w, const float* w_scale, const void* x, const float* x_scale, void* out,
                                 const void* residual, int* status, int M, int N, int K, int token_tile, int kb_per_split,
                                 cudaStream_t stream) {
  using namespace mfq;
  if (K % 128 != 0 || N % 256 != 0 || M <= 0 || kb_per_split < 0 || (kb_per_split && token_tile != 128)) return -1;
  if (kb_per_split && kb_per_split < K / 128) return launch_pair<128, true>(w, w_scale, x, x_scale, out, residual, status, M, N, K, kb_per_split, stream);
  if (token_tile == 128) return launch_pair<128, false>(w, w_scale, x, x_scale, out, residual, status, M, N, K, 0, stream);
  if (token_tile == 256) return launch_pair<256, false>(w, w_scale, x, x_scale, out, residual, status, M, N, K, 0, stream);
  return -1;
}
