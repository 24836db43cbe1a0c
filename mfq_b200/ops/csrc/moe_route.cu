// Mixture-of-experts routing that does not depend on the element type of the experts (part of both libraries): scoring and top-k
// of given router logits, and the route plan of a batch (per-expert row ranges + tile map of the grouped products).
//
// Reference counterparts: moe.cu (moe_topk_kernel and its specialisations, count_experts / scan_expert_counts /
// fill_tile_experts / scatter_routes).
#include "moe_route.cuh"

#include <cfloat>

namespace mfq {

// Scoring and top-k with one WARP per token (logits precomputed, E <= 32 kPer <= 1024, no group limiting): a lane keeps E / 32
// scores in registers, and nothing synchronises a block.  Few tokens are latency, many are issue slots; both are the selection rounds.  So
// a round is a tree over the lane's scores, as many as there are, two warp reductions of whole numbers (the largest value in an order that
// keeps the floats', then the lowest index that has it), and the weight is that value itself unless a bias took part in the choice.
// Logits and selection over 512 experts, top 10 on a B200 (before: a chain over 32 slots and five shuffles of value, weight and index): 32
// tokens 15.4 -> 8.8 us, 3000 tokens 32.5 -> 23.5.
template <int kPer>
__global__ void __launch_bounds__(128) moe_router_topk_warp_kernel(const RouterParams p) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (t >= p.T) return;
  constexpr int kNone = 0x7fffffff;
  float sc[kPer], sel[kPer];
  float mx = -FLT_MAX;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = i * 32 + lane;
    sc[i] = e < p.E ? p.logits[size_t(t) * p.E + e] : -FLT_MAX;
    mx = fmaxf(mx, sc[i]);
  }
  if (p.sigmoid) {
#pragma unroll
    for (int i = 0; i < kPer; ++i) sc[i] = sc[i] == -FLT_MAX ? -FLT_MAX : 1.f / (1.f + __expf(-sc[i]));
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const float v = sc[i] == -FLT_MAX ? 0.f : __expf(sc[i] - mx);
      sc[i] = v;
      sum += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float inv = 1.f / sum;
#pragma unroll
    for (int i = 0; i < kPer; ++i) sc[i] = (i * 32 + lane < p.E) ? sc[i] * inv : -FLT_MAX;
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = i * 32 + lane;
    const bool live = e < p.E;
    const float v = live ? sc[i] + (p.bias ? p.bias[e] : 0.f) : -FLT_MAX;
    sel[i] = v > -FLT_MAX ? v : -FLT_MAX;  // never chosen: places beyond E, NaN, minus infinity
    if (live && p.scores_out) p.scores_out[size_t(t) * p.E + e] = sc[i];
  }
  float wsum = 0.f, my_w = 0.f;
  int my_id = 0;
  for (int k = 0; k < p.K; ++k) {
    float v[kPer];
    int at[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) { v[i] = sel[i]; at[i] = i; }
#pragma unroll
    for (int w = 1; w < kPer; w *= 2) {
#pragma unroll
      for (int i = 0; i < kPer; i += 2 * w)
        if (v[i + w] > v[i]) { v[i] = v[i + w]; at[i] = at[i + w]; }  // neighbours: the lower index wins ties
    }
    const uint32_t bits = __float_as_uint(v[0]);
    const uint32_t key = bits & 0x80000000u ? ~bits : bits | 0x80000000u;
    const uint32_t top = __reduce_max_sync(0xffffffffu, key);
    const int bi = int(__reduce_min_sync(0xffffffffu, unsigned(key == top && v[0] > -FLT_MAX ? at[0] * 32 + lane : kNone)));
    const int mine = bi != kNone && lane == (bi & 31) ? bi >> 5 : -1;
    float best_w = bi == kNone ? 0.f : __uint_as_float(top & 0x80000000u ? top & 0x7fffffffu : ~top);
    if (p.bias && bi != kNone) {
      float own = 0.f;
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        if (i == mine) own = sc[i];
      best_w = __shfl_sync(0xffffffffu, own, bi & 31);
    }
    if (lane == k) { my_id = bi; my_w = best_w; }
    wsum += best_w;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (i == mine) sel[i] = -FLT_MAX;
  }
  if (lane < p.K) {
    const float mul = (p.norm_topk ? 1.f / fmaxf(wsum, 1e-20f) : 1.f) * p.scale;
    p.topk_ids[size_t(t) * p.K + lane] = my_id;
    p.topk_w[size_t(t) * p.K + lane] = my_w * mul;
  }
}

__device__ __forceinline__ void plan_cluster_barrier() {
  __syncwarp();  // loops or branches of single lanes may come before
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t plan_peer_load(const int* mine, int cta) {  // the same variable of another CTA of the cluster
  uint32_t addr, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(smem_u32(mine)), "r"(cta));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// Route plan for the experts [e_lo, e_hi) owned by this rank, by one CTA or a cluster of them.  Row order inside an expert depends on atomic
// arrival order; results do not, because each row is computed independently and the un-permute sums a token's K
// contributions in slot order.
//   offsets[e - e_lo]   first sorted row of local expert e (offsets[n_local] = total rows)
//   dest[t*K + k]       sorted row of that (token, slot) pair, -1 if its expert lives on another rank
//   src_token[row]      token of the sorted row
//   tile_map[i]         (local expert, token tile inside it) for the grouped GEMM; padded with (-1, -1)
// Bound by the shared-memory additions of one route after the other, so many routes are shared out over a cluster of CTAs (kShare of them):
// each counts its own, looks up in the others' counts where its rows of an expert begin, and writes its share.
template <int kShare>
__global__ void __launch_bounds__(1024) moe_plan_kernel(const int* __restrict__ topk_ids, int entries, int K, int e_lo,
                                                        int e_hi, int token_tile, int* __restrict__ offsets,
                                                        int* __restrict__ dest, int* __restrict__ src_token,
                                                        int2* __restrict__ tile_map, int map_cap,
                                                        int* __restrict__ totals) {
  pdl_trigger();
  pdl_wait();
  __shared__ int cnt[kMaxExperts + 1];
  __shared__ int fill[kMaxExperts];
  __shared__ int tbase[kMaxExperts + 1];
  constexpr int kAtOnce = kShare > 1 ? 4 : 1;  // loads of a thread that are on the way at a time
  const int n_local = e_hi - e_lo, share = kShare > 1 ? int(blockIdx.x) : 0;
  const int per = (entries + kShare - 1) / kShare, first = share * per, end = min(entries, first + per);
  for (int e = threadIdx.x; e <= n_local; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  for (int i0 = first + threadIdx.x; i0 < end; i0 += kAtOnce * blockDim.x) {
    int id[kAtOnce];
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const int i = i0 + u * int(blockDim.x);
      id[u] = i < end ? topk_ids[i] - e_lo : -1;
    }
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u)
      if (id[u] >= 0 && id[u] < n_local) atomicAdd(&cnt[id[u]], 1);
  }
  if constexpr (kShare > 1) plan_cluster_barrier();
  else __syncthreads();
  {
    // exclusive prefix sums of the per-expert row and tile counts: one expert per thread, warp scans, then a scan of
    // the 32 warp totals (the block has 1024 threads and at most 512 experts)
    __shared__ int wrow[32], wtile[32];
    const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
    int c = e < n_local ? cnt[e] : 0, before = 0;  // of all shares, of the shares before this one
    if (kShare > 1 && e < n_local) {
      uint32_t other[kShare];
#pragma unroll
      for (int r = 0; r < kShare; ++r) other[r] = plan_peer_load(&cnt[e], r);
      c = 0;
#pragma unroll
      for (int r = 0; r < kShare; ++r) {
        if (r == share) before = c;
        c += int(other[r]);
      }
    }
    const int tl = (c + token_tile - 1) / token_tile;
    int ir = c, it = tl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ur = __shfl_up_sync(0xffffffffu, ir, o), ut = __shfl_up_sync(0xffffffffu, it, o);
      if (lane >= o) { ir += ur; it += ut; }
    }
    if (lane == 31) { wrow[warp] = ir; wtile[warp] = it; }
    __syncthreads();
    if (warp == 0) {
      int vr = wrow[lane], vt = wtile[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int ur = __shfl_up_sync(0xffffffffu, vr, o), ut = __shfl_up_sync(0xffffffffu, vt, o);
        if (lane >= o) { vr += ur; vt += ut; }
      }
      wrow[lane] = vr;
      wtile[lane] = vt;
    }
    __syncthreads();
    const int base_r = warp ? wrow[warp - 1] : 0, base_t = warp ? wtile[warp - 1] : 0;
    if (e < n_local) {
      if (share == 0) offsets[e] = base_r + ir - c;
      fill[e] = base_r + ir - c + before;
      tbase[e] = base_t + it - tl;
    }
    if (e == n_local) {  // totals: everything before this (empty) slot
      tbase[n_local] = base_t + it;
      if (share == 0) {
        offsets[n_local] = base_r + ir;
        totals[0] = base_r + ir;
        totals[1] = base_t + it;
      }
    }
  }
  __syncthreads();
  for (int i0 = first + threadIdx.x; i0 < end; i0 += kAtOnce * blockDim.x) {
    int id[kAtOnce];
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const int i = i0 + u * int(blockDim.x);
      id[u] = i < end ? topk_ids[i] - e_lo : -1;
    }
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const int i = i0 + u * int(blockDim.x);
      int row = -1;
      if (id[u] >= 0 && id[u] < n_local) {
        row = atomicAdd(&fill[id[u]], 1);
        src_token[row] = i / K;
      }
      if (i < end) dest[i] = row;
    }
  }
  for (int e = share + kShare * int(threadIdx.x); e < n_local; e += kShare * int(blockDim.x)) {
    const int n = tbase[e + 1] - tbase[e];
    for (int j = 0; j < n; ++j)
      if (tbase[e] + j < map_cap) tile_map[tbase[e] + j] = make_int2(e, j);
  }
  for (int i = tbase[n_local] + share * int(blockDim.x) + int(threadIdx.x); i < map_cap; i += kShare * int(blockDim.x)) tile_map[i] = make_int2(-1, -1);
  if constexpr (kShare > 1) plan_cluster_barrier();  // nobody's counts go away while a peer may read them
}

int launch_router_topk_warp(const RouterParams& p, cudaStream_t stream) {
  launch_kernel(p.E <= 128 ? moe_router_topk_warp_kernel<4> : p.E <= 256 ? moe_router_topk_warp_kernel<8> : p.E <= 512 ? moe_router_topk_warp_kernel<16>
                : moe_router_topk_warp_kernel<32>, dim3((p.T + 3) / 4), dim3(128), 0, stream, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

}  // namespace mfq

using namespace mfq;

// Routes from which a cluster of eight CTAs shares the plan.  One CTA | eight on a B200: 640 routes 2.5 | 3.6 us, 2000 3.7 | 3.9, 5120 6.3 | 4.3,
// 30000 24.9 | 6.8.
constexpr int kPlanShared = 2500;

// logits [T, E] fp32; the rest as RouterParams
extern "C" int mfq_moe_topk(const float* logits, const float* bias, int* topk_ids, float* topk_w, int T, int E, int K, int sigmoid,
                            int norm_topk, float scale, cudaStream_t stream) {
  if (T <= 0 || E <= 0 || E > kMaxExperts || K <= 0 || K > kMaxTopK || K > E) return -1;
  return launch_router_topk_warp(RouterParams{nullptr, nullptr, bias, topk_ids, topk_w, nullptr, T, 0, E, K, sigmoid, norm_topk, scale, 1, 1,
                                              logits}, stream);
}

extern "C" int mfq_moe_plan(const int* topk_ids, int T, int K, int e_lo, int e_hi, int token_tile, int* offsets, int* dest,
                            int* src_token, void* tile_map, int map_cap, int* totals, cudaStream_t stream) {
  if (e_hi - e_lo > kMaxExperts || e_hi <= e_lo || T <= 0) return -1;
  const auto launch = [&](auto kernel, int share) {
    const dim3 grid(share), block(1024);
    if (share == 1) return launch_kernel(kernel, grid, block, 0, stream, topk_ids, T * K, K, e_lo, e_hi, token_tile, offsets, dest, src_token,
                                         static_cast<int2*>(tile_map), map_cap, totals);
    return launch_kernel_clustered(kernel, grid, block, grid, 0, stream, topk_ids, T * K, K, e_lo, e_hi, token_tile, offsets, dest, src_token,
                                   static_cast<int2*>(tile_map), map_cap, totals);
  };
  if (T * K > kPlanShared) launch(moe_plan_kernel<8>, 8);
  else launch(moe_plan_kernel<1>, 1);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}
