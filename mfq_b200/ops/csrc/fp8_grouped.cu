// Grouped block-scaled FP8 GEMM over expert-sorted token rows:  out[r, :] = X[r, :] * W[e(r), :, :]^T  (formats as in fp8_gemm.cu).
//
// An expert's share of a batch is small -- a prompt of 3000 tokens gives each of 512 experts 59 rows, K may be four blocks -- so the
// weights are streamed once and a tile is over before a CTA of its own has set up barriers and tensor memory.  With a CTA per tile the
// down projection of that layer (2048 x 512) spent 8 us per CTA on four K blocks; here one CTA per SM walks the tiles: the loads of the
// tiles to come fill the ring while the epilogue warps still fold and store, nothing but the first tile pays for set-up, and what a tile
// needs from memory to begin (its place, its weight multipliers) is fetched during the one before.
// What bounds a tile of few K blocks is its end and the next one's beginning: tiles of 32 tokens and more leave through shared memory in
// 16-byte stores (a thread's own columns are 2 bytes every N), and entries, row ranges and multipliers are requested up to two tiles ahead.
// 512 experts of 3 x 2048 x 512, top 10 on a B200, gate/up + down (before: 2-byte stores, entries one tile ahead): 3000 tokens 217 + 193 ->
// 206 + 159 us (what they read and write takes 184 + 104 at the copy rate), 4096 250 + 261 -> 224 + 169, 1500 202 + 178 -> 188 + 144; 200 (tiles
// of 16, which store their columns themselves: 102 through shared memory) 158 + 90 -> 156 + 91, 32 77 + 46 -> 77 + 44.
//
// Roles: warp 0 = TMA, warp 1 = TMEM owner + MMA issuer, warps 2.. = epilogue (TMEM lane quarter = warp % 4; tiles of 64 and 128 tokens
// use two warps per quarter, each taking half of the token columns).  Per 128-wide K block a fresh TMEM accumulator, folded with the
// block's multiplier into fp32 registers, as in fp8_gemm.cu and with its sums.
#include "common.cuh"

namespace mfq {
namespace {

constexpr int kTileN = 128, kBlockK = 128;

template <int BT>
struct GroupedCfg {
  static constexpr int kStageBytes = (kTileN + BT) * kBlockK;
  static constexpr int kStages = BT == 16 ? 10 : BT == 32 ? 9 : BT == 64 ? 8 : 6;
  static constexpr int kAcc = 4;
  static constexpr int kTmemCols = kAcc * BT;
  static constexpr int kEpiWarps = BT >= 64 ? 8 : 4;
  static constexpr int kCols = BT / (kEpiWarps / 4);  // token columns per epilogue thread
  static constexpr int kThreads = 64 + 32 * kEpiWarps;
  static constexpr bool kTurned = BT >= 32;           // whether results leave through shared memory
  static constexpr int kGroups = kEpiWarps / 4;       // of four warps: 128 weight rows x kCols tokens
  static constexpr int kTurnBytes = kCols * kTileN * 2;  // their results on the way out
  static constexpr int kTurnAt = kStages * kStageBytes, kBarsAt = kTurnAt + (kTurned ? kGroups * kTurnBytes : 0);
  static constexpr int kBarBytes = (2 * kStages + 2 * kAcc + 4) * 8 + 8;  // two per stage and accumulator, four of the turned results; TMEM slot, abort flag
  static constexpr int kSmemBytes = kBarsAt + kBarBytes + 1024;           // aligned by hand
};

struct GroupedParams {
  const float* w_scale;   // [experts][N / 128][K / 128]
  const float* x_scale;   // [rows]
  __nv_bfloat16* out;     // [rows][N]
  const int2* tile_map;   // (expert, token tile inside the expert); entries that are not used hold expert -1
  const int* offsets;     // expert e owns rows [offsets[e], offsets[e + 1])
  int* status;
  int N, K, map_len;
  int direct;             // output off a 16-byte boundary: plain stores
};

template <int BT>
__global__ void __launch_bounds__(GroupedCfg<BT>::kThreads, 1)
fp8_grouped_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const GroupedParams p) {
  using Cfg = GroupedCfg<BT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + Cfg::kBarsAt);
  uint64_t* empty = full + Cfg::kStages;
  uint64_t* acc_full = empty + Cfg::kStages;
  uint64_t* acc_empty = acc_full + Cfg::kAcc;
  uint64_t* turn_full = acc_empty + Cfg::kAcc;  // [kGroups] the four warps' results are in shared memory
  uint64_t* turn_free = turn_full + 2;          // ... and have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(turn_free + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < Cfg::kAcc; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], Cfg::kEpiWarps); }
    for (int i = 0; i < Cfg::kGroups; ++i) { mbar_init(&turn_full[i], 4); mbar_init(&turn_free[i], 4); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_trigger();  // TMEM is held by now: a successor that wants some waits for it, not the other way round
  pdl_wait();

  // Tile t = (entry t / n_tiles of the map, weight rows of block t % n_tiles): CTAs at work at the same time share token rows.  Entries
  // are dense: the first unused one ends the list.  The plan and the row multipliers are read by plain loads: under the programmatic
  // launch this grid began before they were written, so they are not constant for its life, as __ldg promises (weights are).
  const int n_tiles = p.N / kTileN, nkb = p.K / kBlockK, tiles = p.map_len * n_tiles, step = int(gridDim.x);
  // What a tile starts from is requested two tiles ahead (its entry) and one (rows of its expert, multipliers), and looked at only then:
  // a tile of four K blocks is 1500 cycles, a load 700.
  auto request = [&](int tile) { return tile < tiles ? p.tile_map[tile / n_tiles] : make_int2(-1, 0); };
  auto same = [&](int2 e) { return make_int2(__shfl_sync(0xffffffffu, e.x, 0), __shfl_sync(0xffffffffu, e.y, 0)); };  // for the whole warp

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_w);
      tma_prefetch_desc(&tmap_x);
    }
    __syncwarp();
    const uint32_t ring_addr = smem_u32(ring), full_addr = smem_u32(full);
    int s = 0;
    uint32_t phase = 0;
    bool ok = true;
    int2 e = same(request(blockIdx.x)), next = same(request(blockIdx.x + step));
    int first = e.x >= 0 ? p.offsets[e.x] : 0;
    for (int tile = blockIdx.x; ok && e.x >= 0; tile += step) {
      const int2 after = request(tile + 2 * step);
      const int next_first = next.x >= 0 ? p.offsets[next.x] : 0;
      const int t0 = __shfl_sync(0xffffffffu, first, 0) + e.y * BT, n0 = tile % n_tiles * kTileN;
      for (int i = 0; i < nkb; ++i) {
        ok = mbar_wait_warp(&empty[s], phase ^ 1u, abort_flag, p.status, kStatusTimeoutProducer);
        if (!ok) break;
        const uint32_t a = ring_addr + s * Cfg::kStageBytes;
        tma_load_stage(a, a + kTileN * kBlockK, &tmap_w, &tmap_x, full_addr + s * 8, Cfg::kStageBytes, true, i * kBlockK, n0, e.x, t0, i * kBlockK);
        if (++s == Cfg::kStages) { s = 0; phase ^= 1u; }
      }
      e = next;
      next = same(after);
      first = next_first;
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc(kTileN, BT, 0, 0);
    constexpr uint64_t kStageStep = uint64_t(Cfg::kStageBytes >> 4);
    const uint64_t a_desc0 = umma_desc_k_sw128(smem_u32(ring)), b_desc0 = umma_desc_k_sw128(smem_u32(ring) + kTileN * kBlockK);
    const uint32_t empty_addr = smem_u32(empty), acc_full_addr = smem_u32(acc_full);
    int s = 0, buf = 0;
    uint32_t phase = 0, acc_phase = 1;  // the first pass over the accumulators finds them free
    bool ok = true;
    int2 e = same(request(blockIdx.x));
    for (int tile = blockIdx.x; ok && e.x >= 0; tile += step) {
      const int2 next = request(tile + step);
      for (int i = 0; i < nkb; ++i) {
        ok = mbar_wait_warp(&acc_empty[buf], acc_phase, abort_flag, p.status, kStatusTimeoutMma) &&
             mbar_wait_warp(&full[s], phase, abort_flag, p.status, kStatusTimeoutMma);
        if (!ok) break;
        tc_fence_after();
        umma_f8f6f4_block(tmem_base + buf * BT, a_desc0 + uint64_t(s) * kStageStep, b_desc0 + uint64_t(s) * kStageStep, idesc, 0u, empty_addr + s * 8,
                          acc_full_addr + buf * 8);
        if (++s == Cfg::kStages) { s = 0; phase ^= 1u; }
        if (++buf == Cfg::kAcc) { buf = 0; acc_phase ^= 1u; }
      }
      e = same(next);
    }
  } else {
    // ----- epilogue warps: thread owns output feature n0 + q*32 + lane and CW token columns from col0 -----
    constexpr int CW = Cfg::kCols, kChunk = CW < 32 ? CW : 32, kChunks = CW / kChunk;
    const int q = warp & 3, group = (warp - 2) >> 2, col0 = group * CW;
    const uint32_t turn = smem_u32(ring) + Cfg::kTurnAt + group * Cfg::kTurnBytes;
    const bool odd = lane & 1;
    const uint32_t chunk = q * 4 + (lane >> 3), within = ((lane >> 1) & 3) * 4;
    const int place = ((warp - 2) & 3) * 32 + lane;  // of the group's 128 threads
    uint32_t turn_phase = 0;
    const uint32_t lane_base = tmem_base + (uint32_t(q * 32) << 16) + col0;
    int buf = 0;
    uint32_t phase = 0;
    bool ok = true, ready = false;
    // row range of a tile's expert, 32 weight multipliers and the row multipliers of this warp's columns, one per lane
    struct Start {
      int lo, hi;
      float ws;
    };
    auto fetch = [&](int tile, int2 at) {
      Start r = {0, 0, 0.f};
      if (at.x < 0) return r;
      r.lo = p.offsets[at.x];
      r.hi = p.offsets[at.x + 1];
      if (lane < nkb) r.ws = __ldg(p.w_scale + (size_t(at.x) * n_tiles + tile % n_tiles) * nkb + lane);
      return r;
    };
    constexpr int kXs = (CW + 31) / 32;
    float xs[kXs];
    auto fetch_rows = [&](int2 at, const Start& r) {
#pragma unroll
      for (int j = 0; j < kXs; ++j) {
        const int row = r.lo + at.y * BT + col0 + j * 32 + lane;
        xs[j] = at.x >= 0 && j * 32 + lane < CW && row < r.hi ? p.x_scale[row] : 0.f;
      }
    };
    int2 e = same(request(blockIdx.x)), next = same(request(blockIdx.x + step));
    Start now = fetch(blockIdx.x, e);
    fetch_rows(e, now);
    for (int tile = blockIdx.x; ok && e.x >= 0; tile += step) {
      const int2 after = request(tile + 2 * step);
      const Start then = fetch(tile + step, next);
      const int t0 = now.lo + e.y * BT, tl = min(BT, now.hi - t0), n = tile % n_tiles * kTileN + q * 32 + lane;
      const float* wsc = p.w_scale + (size_t(e.x) * n_tiles + tile % n_tiles) * nkb;
      float ws = now.ws;
      float acc[CW];
#pragma unroll
      for (int tt = 0; tt < CW; ++tt) acc[tt] = 0.f;
      float ws_after = lane + 32 < nkb ? __ldg(wsc + 32 + lane) : 0.f;
      for (int i = 0; i < nkb; ++i) {
        if (i > 0 && (i & 31) == 0) {
          ws = ws_after;
          ws_after = i + 32 + lane < nkb ? __ldg(wsc + i + 32 + lane) : 0.f;
        }
        if (!ready) ok = mbar_wait_warp(&acc_full[buf], phase, abort_flag, p.status, kStatusTimeoutEpilogue);
        if (!ok) break;
        tc_fence_after();
        const float s = __shfl_sync(0xffffffffu, ws, i & 31);
        const uint32_t taddr = lane_base + buf * BT;
        uint32_t r[2][kChunk];
        auto load_chunk = [&](int c) {
          if constexpr (kChunk == 32) tmem_ld_32x32(taddr + c * 32, r[c & 1]);
          else tmem_ld_32x16(taddr, r[0]);
        };
        load_chunk(0);
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          tmem_wait_ld();
          if (c + 1 < kChunks) {
            load_chunk(c + 1);
          } else {  // all columns are in registers: hand the accumulator back and look at the next one
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
            if (++buf == Cfg::kAcc) { buf = 0; phase ^= 1u; }
            ready = mbar_test_warp(&acc_full[buf], phase);
          }
#pragma unroll
          for (int j = 0; j < kChunk; j += 2) fma2(acc[c * kChunk + j], acc[c * kChunk + j + 1], r[c & 1][j], r[c & 1][j + 1], s);
        }
      }
      if (!ok) break;
#pragma unroll
      for (int tt = 0; tt < CW; ++tt) acc[tt] *= __shfl_sync(0xffffffffu, xs[tt / 32], tt & 31);
      fetch_rows(next, then);
      if (!Cfg::kTurned || p.direct) {
        __nv_bfloat16* dst = p.out + size_t(t0 + col0) * p.N + n;
#pragma unroll
        for (int tt = 0; tt < CW; ++tt)
          if (col0 + tt < tl) dst[size_t(tt) * p.N] = __float2bfloat16(acc[tt]);
      } else {
        // Through shared memory, 256 swizzled bytes of 128 weight rows per token.  A thread has one weight row of tokens t and t + 4; neighbours
        // trade halves, so that an even lane has its pair of rows of token t, an odd one of token t + 4, whose chunks of 16 bytes the swizzle
        // puts beside those of token t.  Out in 16-byte stores, a token's 256 bytes by half a warp.
        ok = mbar_wait_warp(&turn_free[group], turn_phase ^ 1u, abort_flag, p.status, kStatusTimeoutEpilogue);
        if (!ok) break;
#pragma unroll
        for (int tt = 0; tt < CW; tt += 8) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 two = __floats2bfloat162_rn(acc[tt + j], acc[tt + j + 4]);
            const uint32_t own = *reinterpret_cast<const uint32_t*>(&two), other = __shfl_xor_sync(0xffffffffu, own, 1);
            const uint32_t row = j + (odd ? 4 : 0);  // of the eight tokens
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(turn + (tt + row) * 256 + ((chunk ^ row) << 4) + within), "r"(__byte_perm(own, other, odd ? 0x3276 : 0x5410))
                         : "memory");
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&turn_full[group]);
        ok = mbar_wait_warp(&turn_full[group], turn_phase, abort_flag, p.status, kStatusTimeoutEpilogue);
        if (!ok) break;
        __nv_bfloat16* dst = p.out + size_t(t0 + col0) * p.N + tile % n_tiles * kTileN;
#pragma unroll
        for (int i = 0; i < CW * 16 / 128; ++i) {
          const int tt = (i * 128 + place) >> 4, c = place & 15;
          uint4 v;
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(turn + tt * 256 + ((c ^ (tt & 7)) << 4)));
          if (col0 + tt < tl) *reinterpret_cast<uint4*>(dst + size_t(tt) * p.N + c * 8) = v;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&turn_free[group]);
        turn_phase ^= 1u;
      }
      e = next;
      next = same(after);
      now = then;
    }
  }

  // ----- teardown: every thread arrives here, also after an aborted wait -----
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::kTmemCols);
}

template <int BT>
int launch_grouped(const GroupedParams& p, const void* w, const void* x, int rows, int experts, cudaStream_t stream) {
  using Cfg = GroupedCfg<BT>;
  CUtensorMap tw, tx;
  if (make_tmap_3d(&tw, w, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.K, p.N, experts, uint64_t(p.K), uint64_t(p.K) * p.N, kBlockK, kTileN, 1)) return -2;
  if (make_tmap_2d(&tx, x, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, rows, p.K, p.K, BT, kBlockK)) return -3;
  static bool attr_set[64] = {};
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -6;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(fp8_grouped_kernel<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess) return -6;
    attr_set[dev] = true;
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long tiles = long(p.map_len) * (p.N / kTileN);
  launch_kernel(fp8_grouped_kernel<BT>, dim3(unsigned(tiles < sms ? tiles : sms)), dim3(Cfg::kThreads), Cfg::kSmemBytes, stream, tw, tx, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

}  // namespace
}  // namespace mfq

// Grouped GEMM over expert-sorted token rows (mixture of experts): w [E, N, K] E4M3 with w_scale [E, N/128, K/128];
// x / out rows are sorted by expert, expert e owning rows [expert_offsets[e], expert_offsets[e+1]); tile_map holds
// map_len (expert, token-tile) pairs, the unused entries at its end having an expert < 0.  No split-K, no residual.
extern "C" int mfq_fp8_gemm_grouped(const void* w, const float* w_scale, const void* x, const float* x_scale, void* out,
                                    int* status, int rows, int N, int K, int experts, const void* tile_map,
                                    const int* expert_offsets, int map_len, int token_tile, cudaStream_t stream) {
  if (K % 128 != 0 || rows <= 0 || N <= 0 || experts <= 0 || map_len <= 0 || N % 128 != 0) return -1;
  const mfq::GroupedParams p{w_scale, x_scale, static_cast<__nv_bfloat16*>(out), static_cast<const int2*>(tile_map), expert_offsets, status, N, K, map_len, (reinterpret_cast<uintptr_t>(out) & 15) != 0};
  switch (token_tile) {
    case 16: return mfq::launch_grouped<16>(p, w, x, rows, experts, stream);
    case 32: return mfq::launch_grouped<32>(p, w, x, rows, experts, stream);
    case 64: return mfq::launch_grouped<64>(p, w, x, rows, experts, stream);
    case 128: return mfq::launch_grouped<128>(p, w, x, rows, experts, stream);
    default: return -1;
  }
}
