// Memory-bound building blocks of the decode/prefill step: fused (residual +) RMSNorm + FP8 row
// quantization, SwiGLU + FP8 quantization, RoPE + paged FP8 KV write, paged GQA decode attention with
// split-KV, greedy arg-max, embedding gather and the graph-resident step bookkeeping.
//
// Reference counterparts (all scalar fp16/fp32 kernels without an FP8 path): norm.cu / acc.cu
// (acc_rms_norm_*), activation.cu, qk_rope_kv.cu, paged_kv.cu (paged_attention_decode_*_kernel, split +
// reduce), sampling.cu (greedy arg-max), embedding.cu, acc.cu:465 (decode_graph_commit_kernel).
#include "common.cuh"

#include <cfloat>

namespace mfq {

constexpr float kE4M3Max = 448.f;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Largest of 32 values that are not negative (and not NaN, as results of fmaxf with one that is not): their bits are in the same order.
__device__ __forceinline__ float warp_max_abs(float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v))); }
// Block-wide reductions over <= 1024 threads; `red` is 33 floats of shared memory.
template <bool kMax>
__device__ __forceinline__ float block_reduce(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = kMax ? warp_max(v) : warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float x = lane < nw ? red[lane] : (kMax ? -FLT_MAX : 0.f);
    x = kMax ? warp_max(x) : warp_sum(x);
    if (lane == 0) red[32] = x;
  }
  __syncthreads();
  return red[32];
}

__device__ __forceinline__ uint8_t to_e4m3(float v) {
  return static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
}
// Eight values times `inv`, two per conversion instruction.
__device__ __forceinline__ uint2 to_e4m3x8(const float (&v)[8], float inv) {
  uint32_t h[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    h[j] = __nv_cvt_float2_to_fp8x2(make_float2(v[2 * j] * inv, v[2 * j + 1] * inv), __NV_SATFINITE, __NV_E4M3);
  return make_uint2(h[0] | h[1] << 16, h[2] | h[3] << 16);
}
__device__ __forceinline__ float from_e4m3(uint8_t c) {
  __half_raw h = __nv_cvt_fp8_to_halfraw(c, __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}

// g / (1 + exp(-g)) of two values, rounded as the division rounds it.  A division by itself is most of a gated row's instructions, and for
// these operands, whose quotient neither over- nor underflows, it needs no cases: a reciprocal by a Newton step, the quotient from
// it, and two corrections by the remainder, which a fused multiply-add gives exactly (P. Markstein, IBM J. Res. Dev. 34 (1990) 111), two values
// per instruction.  Others -- large, infinite, NaN, zero and what is nearly that -- divide.
__device__ __forceinline__ float2 silu2(float2 g) {
  const float2 d = make_float2(1.f + __expf(-g.x), 1.f + __expf(-g.y));
  if (!(fabsf(g.x) < 64.f && fabsf(g.y) < 64.f && fabsf(g.x) > 1e-30f && fabsf(g.y) > 1e-30f)) return make_float2(g.x / d.x, g.y / d.y);
  float2 r, minus = make_float2(-d.x, -d.y);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(d.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(d.y));
  r = fma_f2(r, fma_f2(minus, r, both(1.f)), r);
  float2 q = fma_f2(g, r, both(-0.f));
  q = fma_f2(fma_f2(minus, q, g), r, q);
  return fma_f2(fma_f2(minus, q, g), r, q);
}

// ---------------------------------------------------------------------------------------------
// (x [+ residual]) -> RMSNorm * w -> per-row FP8.  One CTA per row.  Values stay in registers
// (up to 8 x 8 elements per thread => H <= 8 * 8 * blockDim), so the row is read once.
// ---------------------------------------------------------------------------------------------
constexpr int kNormVecs = 8;

// Where a thread holds several vectors they wait as the bf16 values that they are, four registers a vector: 4096 rows of 4096 on a B200 with
// eight registers a vector (84 a thread) 18.6 us, so 12.8; 2000 rows 12.8 -> 8.5.
// kAhead: all of the residual and the multipliers are requested before the first of them is used, for 16 to 24 more registers.  That pays where
// the rows are on the SMs at once either way, and without it they wait longer than with fp32 values.  fp32 | bf16 | requested ahead, in a chain
// with another kernel: 200 rows of 8192 with residual 5.9 | 7.2 | 5.5 us, 296 of 16384 7.7 | 10.9 | 7.1, 1100 of 4096 10.9 | 12.0 | 9.3; but 900 of 8192
// 14.1 | 11.4 | 12.6 and 1300 of 8192 21.3 | 13.5 | 14.1.
template <int kNormVecs, bool kAhead = false>
__global__ void rmsnorm_quant_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                                     __nv_bfloat16* __restrict__ residual_out, const __nv_bfloat16* __restrict__ w,
                                     uint8_t* __restrict__ q_out, float* __restrict__ scale_out,
                                     __nv_bfloat16* __restrict__ y_out, int H, float eps) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[33];
  const size_t row = blockIdx.x;
  const int nvec = H / 8;
  uint4 held[kNormVecs];
  auto load8 = [](const uint4& a, float (&v)[8]) {
    const uint32_t u[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = __uint_as_float(u[j] << 16);
      v[2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u);
    }
  };
  auto pack8 = [](const float (&v)[8]) {
    uint4 a;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&a);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    return a;
  };
#pragma unroll
  for (int i = 0; i < kNormVecs; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi < nvec) held[i] = *reinterpret_cast<const uint4*>(x + row * H + vi * 8);
  }
  if (residual) {
    uint4 add[kAhead ? kNormVecs : 1];
    if constexpr (kAhead) {
#pragma unroll
      for (int i = 0; i < kNormVecs; ++i) {
        const int vi = threadIdx.x + i * blockDim.x;
        if (vi < nvec) add[i] = *reinterpret_cast<const uint4*>(residual + row * H + vi * 8);
      }
    }
#pragma unroll
    for (int i = 0; i < kNormVecs; ++i) {
      const int vi = threadIdx.x + i * blockDim.x;
      if (vi < nvec) {
        float a[8], r[8];
        load8(held[i], a);
        if constexpr (kAhead) load8(add[i], r);
        else load8(*reinterpret_cast<const uint4*>(residual + row * H + vi * 8), r);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] += r[j];
        held[i] = pack8(a);
        *reinterpret_cast<uint4*>(residual_out + row * H + vi * 8) = held[i];
      }
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < kNormVecs; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi < nvec) {
      float v[8];
      load8(held[i], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
    }
  }
  uint4 held_w[kAhead ? kNormVecs : 1];
  if constexpr (kAhead) {
#pragma unroll
    for (int i = 0; i < kNormVecs; ++i) {
      const int vi = threadIdx.x + i * blockDim.x;
      if (vi < nvec) held_w[i] = *reinterpret_cast<const uint4*>(w + vi * 8);
    }
  }
  const float rstd = rsqrtf(block_reduce<false>(ss, red) / float(H) + eps);
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < kNormVecs; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi < nvec) {
      float v[8], wv[8];
      load8(held[i], v);
      if constexpr (kAhead) load8(held_w[i], wv);
      else load8(*reinterpret_cast<const uint4*>(w + vi * 8), wv);
      // round through bf16 like an unfused norm would, so fused and unfused paths agree bit for bit
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = v[j] * rstd * wv[j];
      held[i] = pack8(v);
      load8(held[i], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
    }
  }
  amax = block_reduce<true>(amax, red);
  const float scale = fmaxf(amax, 1e-12f) / kE4M3Max;
  const float inv = 1.f / scale;
  if (threadIdx.x == 0 && scale_out) scale_out[row] = scale;
#pragma unroll
  for (int i = 0; i < kNormVecs; ++i) {
    const int vi = threadIdx.x + i * blockDim.x;
    if (vi < nvec) {
      if (q_out) {
        float v[8];
        load8(held[i], v);
        *reinterpret_cast<uint2*>(q_out + row * H + vi * 8) = to_e4m3x8(v, inv);
      }
      if (y_out) *reinterpret_cast<uint4*>(y_out + row * H + vi * 8) = held[i];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Row quantization.  mode 0: y = x[row, :K]; mode 1 (SwiGLU): y = silu(x[row, :K]) * x[row, K:2K];
// mode 2 (attention output gate): y = x[row, :K] * sigmoid(x2[row, :K]) with x2 a second, separately strided tensor.
// Up to kRowVecs vectors per thread stay in registers between the maximum and the encoding (every value is a bf16 by then, so a
// vector is four registers); longer rows are read, and their gates evaluated, a second time.  One pass instead of two, and two
// values per conversion: 4096 rows of 14336 on a B200 went from 129 to 80 us (reading and writing alone: 44; the gates' exponentials and
// divisions kept the issue slots two thirds busy), 1000 rows from 36 to 20.  With the gates by silu2 74 and 19, with all loads of a full row
// requested before the first is used 69 and 18.
// ---------------------------------------------------------------------------------------------
// kFull: gated rows of kRowVecs vectors for every thread.  They need 62 registers, which the others do without: three CTAs per SM, with 40 registers and
// 16 bytes of spills, take 4096 gated rows of 11008 in 54.5 us and 1000 of 18944 in 39.4, two with 47 and none 61.3 and 43.4 (2000 rows of 512: 3.9
// and 3.5).
constexpr int kRowVecs = 4;
template <int kMode, bool kFull = false>
__global__ void __launch_bounds__(512, kFull ? 1 : 3) quant_rows_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q_out,
                                  float* __restrict__ scale_out, int K, int in_stride,
                                  const __nv_bfloat16* __restrict__ x2 = nullptr, int x2_stride = 0) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[33];
  const size_t row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * in_stride;
  const __nv_bfloat16* gr = kMode == 2 ? x2 + row * x2_stride : nullptr;
  const int nvec = K / 8;
  auto value = [&](int vi, float (&y)[8]) {
    uint4 a = *reinterpret_cast<const uint4*>(xr + vi * 8);
    const __nv_bfloat16* ab = reinterpret_cast<const __nv_bfloat16*>(&a);
    if (kMode == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) y[j] = __bfloat162float(ab[j]);
    } else if (kMode == 2) {
      uint4 b = *reinterpret_cast<const uint4*>(gr + vi * 8);
      const __nv_bfloat16* bb = reinterpret_cast<const __nv_bfloat16*>(&b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float h = __bfloat162float(ab[j]) / (1.f + __expf(-__bfloat162float(bb[j])));
        y[j] = __bfloat162float(__float2bfloat16(h));
      }
    } else {
      uint4 b = *reinterpret_cast<const uint4*>(xr + K + vi * 8);
      const __nv_bfloat16* bb = reinterpret_cast<const __nv_bfloat16*>(&b);
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const float2 h = silu2(make_float2(__bfloat162float(ab[j]), __bfloat162float(ab[j + 1])));
        y[j] = __bfloat162float(__float2bfloat16(h.x * __bfloat162float(bb[j])));
        y[j + 1] = __bfloat162float(__float2bfloat16(h.y * __bfloat162float(bb[j + 1])));
      }
    }
  };
  float amax = 0.f;
  if (nvec <= kRowVecs * int(blockDim.x)) {
    uint4 held[kRowVecs];
    if (kMode == 0 && nvec == kRowVecs * int(blockDim.x)) {
      // Nothing but the row, and as many vectors as a thread can hold: bound by its loads in flight, so all of a thread's are requested
      // before the first is used.  4000 rows of 16384: 44.5 us with each load under its condition, 37.5 in two passes of four loads, 30.9 so;
      // of 4096: 7.9, 20.0, 7.0.
#pragma unroll
      for (int i = 0; i < kRowVecs; ++i) held[i] = *reinterpret_cast<const uint4*>(xr + (threadIdx.x + i * blockDim.x) * 8);
#pragma unroll
      for (int i = 0; i < kRowVecs; ++i) {
        const uint32_t w[4] = {held[i].x, held[i].y, held[i].z, held[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(w[j] << 16)), fabsf(__uint_as_float(w[j] & 0xffff0000u))));
      }
    } else if (kFull) {  // likewise, gates and values
      uint4 up[kRowVecs];
#pragma unroll
      for (int i = 0; i < kRowVecs; ++i) {
        held[i] = *reinterpret_cast<const uint4*>(xr + (threadIdx.x + i * blockDim.x) * 8);
        up[i] = *reinterpret_cast<const uint4*>(xr + K + (threadIdx.x + i * blockDim.x) * 8);
      }
#pragma unroll
      for (int i = 0; i < kRowVecs; ++i) {
        const uint32_t a[4] = {held[i].x, held[i].y, held[i].z, held[i].w}, b[4] = {up[i].x, up[i].y, up[i].z, up[i].w};
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&held[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 s = silu2(make_float2(__uint_as_float(a[j] << 16), __uint_as_float(a[j] & 0xffff0000u)));
          h[j] = __floats2bfloat162_rn(s.x * __uint_as_float(b[j] << 16), s.y * __uint_as_float(b[j] & 0xffff0000u));
          const float2 y = __bfloat1622float2(h[j]);
          amax = fmaxf(amax, fmaxf(fabsf(y.x), fabsf(y.y)));
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < kRowVecs; ++i) {
        const int vi = threadIdx.x + i * blockDim.x;
        if (vi < nvec) {
          float y[8];
          value(vi, y);
          __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&held[i]);
#pragma unroll
          for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(y[j]));
#pragma unroll
          for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(y[2 * j], y[2 * j + 1]);
        }
      }
    }
    amax = block_reduce<true>(amax, red);
    const float scale = fmaxf(amax, 1e-12f) / kE4M3Max, inv = 1.f / scale;
    if (threadIdx.x == 0) scale_out[row] = scale;
#pragma unroll
    for (int i = 0; i < kRowVecs; ++i) {
      const int vi = threadIdx.x + i * blockDim.x;
      if (vi < nvec) {
        const uint32_t w[4] = {held[i].x, held[i].y, held[i].z, held[i].w};
        float y[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          y[2 * j] = __uint_as_float(w[j] << 16);
          y[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
        }
        *reinterpret_cast<uint2*>(q_out + row * K + vi * 8) = to_e4m3x8(y, inv);
      }
    }
    return;
  }
  for (int vi = threadIdx.x; vi < nvec; vi += blockDim.x) {
    float y[8];
    value(vi, y);
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(y[j]));
  }
  amax = block_reduce<true>(amax, red);
  const float scale = fmaxf(amax, 1e-12f) / kE4M3Max;
  const float inv = 1.f / scale;
  if (threadIdx.x == 0) scale_out[row] = scale;
  for (int vi = threadIdx.x; vi < nvec; vi += blockDim.x) {
    float y[8];
    value(vi, y);
    *reinterpret_cast<uint2*>(q_out + row * K + vi * 8) = to_e4m3x8(y, inv);
  }
}


// Many short rows (routed experts' halves): a warp per row and no block, all its vectors requested together.  A block | a warp per row on a
// B200: 30000 rows of 512 gated values 31.5 | 17.0 us (reading and writing alone: 12), 10000 10.9 | 6.9, 2000 4.0 | 4.3; gated rows of 1024
// 30000 39.4 | 37.1, 5120 8.5 | 8.8; plain rows of 1024 30000 31.6 | 11.3, 320 2.0 | 1.7, 80 1.5 | 1.6.
template <int kMode, int kVecs>
__global__ void __launch_bounds__(256) quant_short_rows_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q_out,
                                                               float* __restrict__ scale_out, int M, int K, int in_stride) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5), nvec = K / 8;
  if (row >= M) return;
  const __nv_bfloat16* xr = x + size_t(row) * in_stride;
  uint4 a[kVecs], b[kVecs];
#pragma unroll
  for (int i = 0; i < kVecs; ++i)
    if (lane + i * 32 < nvec) {
      a[i] = *reinterpret_cast<const uint4*>(xr + (lane + i * 32) * 8);
      if (kMode == 1) b[i] = *reinterpret_cast<const uint4*>(xr + K + (lane + i * 32) * 8);
    }
  float y[kVecs][8], amax = 0.f;
#pragma unroll
  for (int i = 0; i < kVecs; ++i)
    if (lane + i * 32 < nvec) {
      const uint32_t gate[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, up[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 g = make_float2(__uint_as_float(gate[j] << 16), __uint_as_float(gate[j] & 0xffff0000u));
        const float2 s = kMode == 1 ? silu2(g) : g;
        y[i][2 * j] = kMode == 1 ? __bfloat162float(__float2bfloat16(s.x * __uint_as_float(up[j] << 16))) : s.x;
        y[i][2 * j + 1] = kMode == 1 ? __bfloat162float(__float2bfloat16(s.y * __uint_as_float(up[j] & 0xffff0000u))) : s.y;
        amax = fmaxf(amax, fmaxf(fabsf(y[i][2 * j]), fabsf(y[i][2 * j + 1])));
      }
    }
  amax = warp_max(amax);
  const float scale = fmaxf(amax, 1e-12f) / kE4M3Max, inv = 1.f / scale;
  if (lane == 0) scale_out[row] = scale;
#pragma unroll
  for (int i = 0; i < kVecs; ++i)
    if (lane + i * 32 < nvec) *reinterpret_cast<uint2*>(q_out + size_t(row) * K + (lane + i * 32) * 8) = to_e4m3x8(y[i], inv);
}

// SwiGLU + row quantization for decode-sized batches, one ROW PER CLUSTER of kSplit CTAs: with one CTA per row a batch
// of 64 rows occupies 64 of 148 SMs and every thread walks its slice twice (amax, then encode, the SiLU evaluated both
// times).  Here a CTA owns 1/kSplit of the row, keeps its products in registers, and puts its maximum into every CTA's shared memory: the
// barrier that says that all have is the only one on the way (that all CTAs run, which remote stores need, is asked for before the wait for
// the kernel before).  64 rows of 14336 on a B200, maxima fetched behind one barrier and kept alive by another: 4.9 us, so 4.3.
constexpr int kSwigluSplit = 4;
constexpr int kSwigluVecs = 2;  // 16-byte vectors per thread: covers K <= 8 * 256 * kSwigluVecs * kSwigluSplit
__global__ void __cluster_dims__(kSwigluSplit, 1, 1) __launch_bounds__(256)
silu_mul_quant_split_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q_out, float* __restrict__ scale_out,
                            int K, int in_stride) {
  pdl_trigger();
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
  __shared__ float red[33];
  __shared__ float maxima[kSwigluSplit];
  const size_t row = blockIdx.x / kSwigluSplit;
  const int part = blockIdx.x % kSwigluSplit;
  const __nv_bfloat16* xr = x + row * in_stride;
  const int nvec = K / 8 / kSwigluSplit, v0 = part * nvec;
  pdl_wait();
  uint4 a[kSwigluVecs], b[kSwigluVecs];
#pragma unroll
  for (int i = 0; i < kSwigluVecs; ++i) {
    const int vi = threadIdx.x + i * 256;
    if (vi < nvec) {
      a[i] = *reinterpret_cast<const uint4*>(xr + (v0 + vi) * 8);
      b[i] = *reinterpret_cast<const uint4*>(xr + K + (v0 + vi) * 8);
    }
  }
  float y[kSwigluVecs][8];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < kSwigluVecs; ++i) {
    const int vi = threadIdx.x + i * 256;
    if (vi < nvec) {
      const uint32_t gate[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, up[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 s = silu2(make_float2(__uint_as_float(gate[j] << 16), __uint_as_float(gate[j] & 0xffff0000u)));
        y[i][2 * j] = __bfloat162float(__float2bfloat16(s.x * __uint_as_float(up[j] << 16)));
        y[i][2 * j + 1] = __bfloat162float(__float2bfloat16(s.y * __uint_as_float(up[j] & 0xffff0000u)));
        amax = fmaxf(amax, fmaxf(fabsf(y[i][2 * j]), fabsf(y[i][2 * j + 1])));
      }
    }
  }
  amax = block_reduce<true>(amax, red);
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  if (threadIdx.x < kSwigluSplit) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(&maxima[part])), "r"(threadIdx.x));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(amax) : "memory");
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  float row_max = maxima[0];
#pragma unroll
  for (int r = 1; r < kSwigluSplit; ++r) row_max = fmaxf(row_max, maxima[r]);
  const float scale = fmaxf(row_max, 1e-12f) / kE4M3Max, inv = 1.f / scale;
  if (part == 0 && threadIdx.x == 0) scale_out[row] = scale;
#pragma unroll
  for (int i = 0; i < kSwigluVecs; ++i) {
    const int vi = threadIdx.x + i * 256;
    if (vi < nvec) {
      *reinterpret_cast<uint2*>(q_out + row * K + (v0 + vi) * 8) = to_e4m3x8(y[i], inv);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// RoPE (rotate-half pairing i <-> i + rot/2 over the first `rot` dims) on Q and K, then K/V -> FP8 pages.
// qkv: [T, (Hq + 2 Hk) * D] bf16.  One warp per (token, head).  Cache page layout [page][Hk][page_size][D]
// with one fp32 multiplier per (page, head, slot).  slots[t] = physical page * page_size + offset (< 0: skip).
// ---------------------------------------------------------------------------------------------
// YaRN context extension: rotary pair `fi` keeps its frequency below `low`, is slowed down by `factor` above `high`,
// blended linearly in between; cos / sin carry `mscale`.  factor == 1 leaves the frequencies bit-identical.
struct RopeScale {
  float factor, low, high, mscale;
};

__device__ __forceinline__ float rope_inv_freq(float log2_theta, int fi, int rot, const RopeScale& y) {
  float f = exp2f(-log2_theta * (2.f * fi) / float(rot));
  if (y.factor != 1.f) {
    const float ramp = fminf(fmaxf((float(fi) - y.low) / (y.high - y.low), 0.f), 1.f);
    f *= (1.f - ramp) + ramp / y.factor;
  }
  return f;
}

// Where a head's rows go.
struct RopeOut {
  __nv_bfloat16* q;  // [T, Hq, D]
  uint8_t *k_cache, *v_cache;
  float *k_scale, *v_scale;
  __nv_bfloat16 *kd, *vd;  // [T, Hk, D], optional
  int Hq, Hk, page_size;
};

// One head of a token by a warp: `lo`, `hi` are the lane's D / 64 values of either half of `src`.  `angle(j, s, c)`: sine and cosine of
// the lane's j-th pair (full rotary).  kWide: what a lane writes to q, kd and vd goes out in one store.
template <int D, bool kWide, typename Angle, typename Slot>
__device__ __forceinline__ void rope_head(const __nv_bfloat16* __restrict__ src, float (&lo)[D / 64], float (&hi)[D / 64], int t, int h,
                                          int lane, const int* __restrict__ positions, int rot, float log2_theta, const RopeScale& ys,
                                          const float* __restrict__ q_norm_w, const float* __restrict__ k_norm_w, float norm_eps,
                                          const RopeOut& to, const Angle& angle, const Slot& slot_of) {
  constexpr int HP = D / 64;
  auto store_half = [&](__nv_bfloat16* ptr, const float (&v)[HP]) {
    if constexpr (kWide && HP % 2 == 0) {
      uint32_t packed[HP / 2];
#pragma unroll
      for (int j = 0; j < HP / 2; ++j) {
        const __nv_bfloat162 two = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        packed[j] = *reinterpret_cast<const uint32_t*>(&two);
      }
      if constexpr (HP == 4) *reinterpret_cast<uint2*>(ptr) = make_uint2(packed[0], packed[1]);
      else *reinterpret_cast<uint32_t*>(ptr) = packed[0];
    } else {
#pragma unroll
      for (int j = 0; j < HP; ++j) ptr[j] = __float2bfloat16(v[j]);
    }
  };
  const int Hq = to.Hq, Hk = to.Hk, page_size = to.page_size;
  const bool is_v = h >= Hq + Hk;
  // optional per-head RMSNorm of q and k before the rotation (QK-norm); nw_scale folds 1/rms into the partner reads
  const float* nw = is_v ? nullptr : (h < Hq ? q_norm_w : k_norm_w);
  float inv_rms = 1.f;
  if (nw) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < HP; ++j) ss += lo[j] * lo[j] + hi[j] * hi[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    inv_rms = rsqrtf(ss / float(D) + norm_eps);
#pragma unroll
    for (int j = 0; j < HP; ++j) {
      lo[j] *= inv_rms * nw[lane * HP + j];
      hi[j] *= inv_rms * nw[D / 2 + lane * HP + j];
    }
  }
  if (!is_v) {
    const int half_rot = rot / 2;
    if (rot == D) {
#pragma unroll
      for (int j = 0; j < HP; ++j) {
        float s, c;
        angle(j, s, c);
        const float a = lo[j], b = hi[j];
        lo[j] = __fmaf_rn(a, c, -__fmul_rn(b, s));
        hi[j] = __fmaf_rn(b, c, __fmul_rn(a, s));
      }
    } else {
      // partial rotary: pairs (i, i + rot/2) live inside the first `rot` dims.  Handle through shared
      // exchange-free recomputation: each lane re-reads its partner element.
      const float pos = float(positions[t]);
#pragma unroll
      for (int j = 0; j < HP; ++j) {
        for (int part = 0; part < 2; ++part) {
          const int idx = (part ? D / 2 : 0) + lane * HP + j;
          if (idx < rot) {
            const int fi = idx % half_rot;
            const float inv_freq = rope_inv_freq(log2_theta, fi, rot, ys);
            float s, c;
            sincosf(pos * inv_freq, &s, &c);
            s *= ys.mscale;
            c *= ys.mscale;
            const float self = part ? hi[j] : lo[j];
            const int pidx = idx < half_rot ? idx + half_rot : idx - half_rot;
            const float other = __bfloat162float(src[pidx]) * (nw ? inv_rms * nw[pidx] : 1.f);
            const float r = idx < half_rot ? self * c - other * s : self * c + other * s;
            if (part) hi[j] = r; else lo[j] = r;
          }
        }
      }
    }
  }
  if (h < Hq) {
    __nv_bfloat16* dst = to.q + size_t(t) * Hq * D + size_t(h) * D;
    store_half(dst + lane * HP, lo);
    store_half(dst + D / 2 + lane * HP, hi);
    return;
  }
  const int slot = slot_of();
  if (slot < 0) return;
  const int kvh = is_v ? h - Hq - Hk : h - Hq;
  const int page = slot / page_size, off = slot % page_size;
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < HP; ++j) {
    lo[j] = __bfloat162float(__float2bfloat16(lo[j]));
    hi[j] = __bfloat162float(__float2bfloat16(hi[j]));
    amax = fmaxf(amax, fmaxf(fabsf(lo[j]), fabsf(hi[j])));
  }
  amax = warp_max_abs(amax);
  const float scale = fmaxf(amax, 1e-12f) / kE4M3Max;
  const float inv = 1.f / scale;
  const size_t base = ((size_t(page) * Hk + kvh) * page_size + off);
  const size_t ph = size_t(page) * Hk + kvh;
  if (!is_v) {
    // K page: [D/64 chunks][page_size tokens][64 dims]
    uint8_t* dst = to.k_cache + ph * (size_t(page_size) * D);
    if constexpr (HP == 2) {  // neighbouring dims of a chunk: one store of two
      const int d0 = lane * HP, d1 = D / 2 + lane * HP;
      *reinterpret_cast<__nv_fp8x2_storage_t*>(dst + (d0 >> 6) * (page_size * 64) + off * 64 + (d0 & 63)) =
          __nv_cvt_float2_to_fp8x2(make_float2(lo[0] * inv, lo[1] * inv), __NV_SATFINITE, __NV_E4M3);
      *reinterpret_cast<__nv_fp8x2_storage_t*>(dst + (d1 >> 6) * (page_size * 64) + off * 64 + (d1 & 63)) =
          __nv_cvt_float2_to_fp8x2(make_float2(hi[0] * inv, hi[1] * inv), __NV_SATFINITE, __NV_E4M3);
    } else {
#pragma unroll
      for (int j = 0; j < HP; ++j) {
        const int d0 = lane * HP + j, d1 = D / 2 + lane * HP + j;
        dst[(d0 >> 6) * (page_size * 64) + off * 64 + (d0 & 63)] = to_e4m3(lo[j] * inv);
        dst[(d1 >> 6) * (page_size * 64) + off * 64 + (d1 & 63)] = to_e4m3(hi[j] * inv);
      }
    }
  } else {
    // V page: [D dims][page_size tokens in the order 0,1,8,9,2,3,10,11,4,5,12,13,6,7,14,15]
    uint8_t* dst = to.v_cache + ph * (size_t(page_size) * D);
    const int pos = 4 * ((off & 7) >> 1) + 2 * (off >> 3) + (off & 1);
#pragma unroll
    for (int j = 0; j < HP; ++j) {
      dst[(lane * HP + j) * page_size + pos] = to_e4m3(lo[j] * inv);
      dst[(D / 2 + lane * HP + j) * page_size + pos] = to_e4m3(hi[j] * inv);
    }
  }
  // Optional contiguous copy of what the pages now hold (code * multiplier), [T, Hk, D] bf16: the prefill attention
  // of this chunk reads it, so prefill and later decode steps see the same FP8-rounded K/V.
  __nv_bfloat16* dq = is_v ? to.vd : to.kd;
  if (dq) {
    dq += (size_t(t) * Hk + kvh) * D;
#pragma unroll
    for (int j = 0; j < HP; ++j) {
      lo[j] = from_e4m3(to_e4m3(lo[j] * inv)) * scale;
      hi[j] = from_e4m3(to_e4m3(hi[j] * inv)) * scale;
    }
    store_half(dq + lane * HP, lo);
    store_half(dq + D / 2 + lane * HP, hi);
  }
  if (lane == 0) (is_v ? to.v_scale : to.k_scale)[base] = scale;
}

// The values of sixteen tokens and one head, the tokens of one page where a prompt fills whole ones: a page holds a dim's sixteen tokens side
// by side, so token by token every byte goes to a sector of its own.  A lane has D / 32 neighbouring dims of all sixteen tokens: the bytes
// of a dim come together in its registers and leave as one store.  The tokens of other groups (a page's part, slots in another order, none)
// are left to the warps that go token by token.
constexpr int kGroupTokens = 16;
// First token of the whole page that begins within sixteen tokens from `from` on, and its slot; -1: none does.  Two cannot: the second would lie
// inside the first.  So prompts packed one after the other have their pages found wherever they begin.
__device__ __forceinline__ int whole_page_from(const int* __restrict__ slots, int from, int T, int lane, int& slot0) {
  const int slot = from + lane < T ? slots[from + lane] : -1;
  const int next = __shfl_down_sync(0xffffffffu, slot, 1);
  const uint32_t runs = __ballot_sync(0xffffffffu, lane < 31 && slot >= 0 && next == slot + 1);
  const uint32_t begins = __ballot_sync(0xffffffffu, lane < 16 && slot >= 0 && (slot & 15) == 0 && (runs >> lane & 0x7fffu) == 0x7fffu);
  const int at = __ffs(begins) - 1;
  slot0 = __shfl_sync(0xffffffffu, slot, at & 31);
  return at < 0 ? -1 : from + at;
}
// Whether token t, which goes to `slot`, belongs to such a page.
__device__ __forceinline__ bool in_whole_page(const int* __restrict__ slots, int t, int slot, int T, int lane) {
  const int t0 = t - (slot & 15);
  return slot >= 0 && t0 >= 0 && t0 + kGroupTokens <= T && __all_sync(0xffffffffu, slots[t0 + (lane & 15)] == (slot & ~15) + (lane & 15));
}
template <int D>
__device__ __forceinline__ void value_group(const __nv_bfloat16* __restrict__ qkv, const int* __restrict__ slots, const RopeOut& to, int T, int row_stride,
                                            int block) {
  constexpr int VPL = D / 32, W = VPL / 4;  // dims of a lane, words of their codes
  const int lane = threadIdx.x & 31, head_blocks = (to.Hk + 7) / 8;
  const int h = block % head_blocks * 8 + (threadIdx.x >> 5);
  if (h >= to.Hk) return;
  int slot0;
  const int t0 = whole_page_from(slots, block / head_blocks * kGroupTokens, T, lane, slot0);
  if (t0 < 0) return;
  const __nv_bfloat16* src = qkv + size_t(to.Hq + to.Hk + h) * D + lane * VPL;
  uint2 raw[kGroupTokens][W];
#pragma unroll
  for (int i = 0; i < kGroupTokens; ++i) {
    const int t = t0 + i;
#pragma unroll
    for (int w = 0; w < W; ++w) raw[i][w] = *reinterpret_cast<const uint2*>(src + size_t(t) * row_stride + w * 4);
  }
  uint32_t code[kGroupTokens][W];
  float my_scale = 0.f;
#pragma unroll
  for (int i = 0; i < kGroupTokens; ++i) {
    float v[VPL], amax = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      v[4 * w] = __uint_as_float(raw[i][w].x << 16);
      v[4 * w + 1] = __uint_as_float(raw[i][w].x & 0xffff0000u);
      v[4 * w + 2] = __uint_as_float(raw[i][w].y << 16);
      v[4 * w + 3] = __uint_as_float(raw[i][w].y & 0xffff0000u);
    }
#pragma unroll
    for (int j = 0; j < VPL; ++j) amax = fmaxf(amax, fabsf(v[j]));
    amax = warp_max_abs(amax);
    const float scale = fmaxf(amax, 1e-12f) / kE4M3Max, inv = 1.f / scale;
    if (lane == i) my_scale = scale;
    const int t = t0 + i;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * w] * inv, v[4 * w + 1] * inv), __NV_SATFINITE, __NV_E4M3);
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * w + 2] * inv, v[4 * w + 3] * inv), __NV_SATFINITE, __NV_E4M3);
      code[i][w] = lo | hi << 16;
    }
    if (to.vd) {
      __nv_bfloat16* dst = to.vd + (size_t(t) * to.Hk + h) * D + lane * VPL;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        float d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) d[j] = from_e4m3(uint8_t(code[i][w] >> (8 * j))) * scale;
        const __nv_bfloat162 a = __floats2bfloat162_rn(d[0], d[1]), b = __floats2bfloat162_rn(d[2], d[3]);
        *reinterpret_cast<uint2*>(dst + w * 4) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
      }
    }
  }
  if (lane < kGroupTokens) to.v_scale[(size_t(slot0 >> 4) * to.Hk + h) * 16 + lane] = my_scale;
  uint4* dst = reinterpret_cast<uint4*>(to.v_cache + (size_t(slot0 >> 4) * to.Hk + h) * (size_t(16) * D) + lane * VPL * 16);
#pragma unroll
  for (int w = 0; w < W; ++w) {
    uint32_t out[4][4];  // [dim][word]: word g of a page's row holds tokens 2g, 2g + 1, 2g + 8, 2g + 9
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const uint32_t a = code[2 * g][w], b = code[2 * g + 1][w], c = code[2 * g + 8][w], d = code[2 * g + 9][w];
      const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362), cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
      out[0][g] = __byte_perm(ab0, cd0, 0x5410);
      out[1][g] = __byte_perm(ab0, cd0, 0x7632);
      out[2][g] = __byte_perm(ab1, cd1, 0x5410);
      out[3][g] = __byte_perm(ab1, cd1, 0x7632);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[w * 4 + j] = make_uint4(out[j][0], out[j][1], out[j][2], out[j][3]);
  }
}

// kHeads: heads of a token that a warp takes.  Several (full rotary only): their angles are evaluated once.
template <int D, int kHeads>
__device__ __forceinline__ void rope_rows(const __nv_bfloat16* __restrict__ qkv, const int* __restrict__ positions,
                                          const int* __restrict__ slots, __nv_bfloat16* __restrict__ q_out,
                                          uint8_t* __restrict__ k_cache, uint8_t* __restrict__ v_cache,
                                          float* __restrict__ k_scale, float* __restrict__ v_scale, int T, int Hq, int Hk,
                                          int page_size, int rot, float log2_theta, __nv_bfloat16* __restrict__ kd_out,
                                          __nv_bfloat16* __restrict__ vd_out, const float* __restrict__ q_norm_w,
                                          const float* __restrict__ k_norm_w, float norm_eps, int row_stride,
                                          const RopeScale ys, int value_blocks) {
  pdl_trigger();
  pdl_wait();
  const RopeOut to{q_out, k_cache, v_cache, k_scale, v_scale, kd_out, vd_out, Hq, Hk, page_size};
  if constexpr (kHeads > 1 && D >= 128) {
    if (int(blockIdx.x) < value_blocks) {
      value_group<D>(qkv, slots, to, T, row_stride, blockIdx.x);
      return;
    }
  }
  constexpr int EPL = D / 32;  // elements per lane
  const int warps_per_block = blockDim.x >> 5;
  const int gw = (int(blockIdx.x) - value_blocks) * warps_per_block + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int heads = Hq + 2 * Hk, groups = (heads + kHeads - 1) / kHeads;
  if (gw >= T * groups) return;
  const int t = gw / groups, h_first = gw % groups * kHeads;
  const __nv_bfloat16* src = qkv + size_t(t) * row_stride + size_t(h_first) * D;  // rows may carry extra trailing columns
  // lane owns EPL/2 rotation pairs: indices j and j + rot/2 for j = lane*EPL/2 .. (only when below rot/2),
  // plus pass-through of non-rotated dims; simplest uniform scheme: lane handles dims
  // [lane*EPL/2, lane*EPL/2 + EPL/2) of each half of the head vector.
  constexpr int HP = EPL / 2;
  float lo[HP], hi[HP];
  // explicit vector loads: with a run-time row stride the compiler can no longer prove the alignment itself
  // (the host entry checks that the stride is a multiple of 8 elements)
  auto load_half = [&](const __nv_bfloat16* ptr, float (&dst)[HP]) {
    if constexpr (HP == 2) {
      const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(ptr);
      dst[0] = __bfloat162float(v.x);
      dst[1] = __bfloat162float(v.y);
    } else if constexpr (HP == 4) {
      const uint2 raw = *reinterpret_cast<const uint2*>(ptr);
      const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[j] = __bfloat162float(e[j]);
    } else {
#pragma unroll
      for (int j = 0; j < HP; ++j) dst[j] = __bfloat162float(ptr[j]);
    }
  };
  constexpr bool kAhead = kHeads > 1 && HP <= 2;  // all heads of the warp requested before the first is used
  const int h_end = min(h_first + kHeads, heads);
  uint32_t raw[kAhead ? kHeads : 1][2];
  if constexpr (kAhead) {
#pragma unroll
    for (int i = 0; i < kHeads; ++i) {
      const __nv_bfloat16* at = src + (h_first + i < h_end ? i * D : 0) + lane * HP;
      if constexpr (HP == 2) {
        raw[i][0] = *reinterpret_cast<const uint32_t*>(at);
        raw[i][1] = *reinterpret_cast<const uint32_t*>(at + D / 2);
      } else {
        raw[i][0] = *reinterpret_cast<const unsigned short*>(at);
        raw[i][1] = *reinterpret_cast<const unsigned short*>(at + D / 2);
      }
    }
  } else {
    load_half(src + lane * HP, lo);
    load_half(src + D / 2 + lane * HP, hi);
  }
  auto evaluate = [&](int j, float& s, float& c) {
    sincosf(float(positions[t]) * rope_inv_freq(log2_theta, lane * HP + j, rot, ys), &s, &c);
    s *= ys.mscale;
    c *= ys.mscale;
  };
  // The slot is requested with the position, not after the rotation (0.4 us of a decode step's launch), but for one head of 64, where it
  // costs a block per SM (36 registers instead of 32: 500 tokens of 36 heads 4.6 -> 4.8 us).
  constexpr bool kEarlySlot = kHeads > 1 || D > 64;
  const int slot_early = kEarlySlot && h_first + kHeads > Hq ? slots[t] : -1;
  const auto slot = [&] { return kEarlySlot ? slot_early : slots[t]; };
  if constexpr (kHeads == 1) {
    rope_head<D, false>(src, lo, hi, t, h_first, lane, positions, rot, log2_theta, ys, q_norm_w, k_norm_w, norm_eps, to, evaluate, slot);
  } else {
    float cs[HP], sn[HP];
    if (h_first < Hq + Hk) {  // values are not rotated; the first head is on its way from memory
#pragma unroll
      for (int j = 0; j < HP; ++j) evaluate(j, sn[j], cs[j]);
    }
    // by the warps that take whole pages
    const bool values_done = value_blocks && h_end > Hq + Hk && in_whole_page(slots, t, slot_early, T, lane);
    const auto shared_angle = [&](int j, float& s, float& c) { s = sn[j]; c = cs[j]; };
    if constexpr (kAhead) {
#pragma unroll
      for (int i = 0; i < kHeads; ++i) {
        if (h_first + i >= h_end || (values_done && h_first + i >= Hq + Hk)) break;
#pragma unroll
        for (int j = 0; j < HP; ++j) {
          lo[j] = __uint_as_float(j ? raw[i][0] & 0xffff0000u : raw[i][0] << 16);
          hi[j] = __uint_as_float(j ? raw[i][1] & 0xffff0000u : raw[i][1] << 16);
        }
        rope_head<D, true>(src + i * D, lo, hi, t, h_first + i, lane, positions, D, log2_theta, ys, q_norm_w, k_norm_w, norm_eps, to, shared_angle, slot);
      }
    } else {
      for (int h = h_first; h < h_end; ++h, src += D) {
        if (values_done && h >= Hq + Hk) break;
        if (h != h_first) {
          load_half(src + lane * HP, lo);
          load_half(src + D / 2 + lane * HP, hi);
        }
        rope_head<D, true>(src, lo, hi, t, h, lane, positions, D, log2_theta, ys, q_norm_w, k_norm_w, norm_eps, to, shared_angle, slot);
      }
    }
  }
}

template <int D>
__global__ void rope_kv_write_kernel(const __nv_bfloat16* __restrict__ qkv, const int* __restrict__ positions,
                                     const int* __restrict__ slots, __nv_bfloat16* __restrict__ q_out,
                                     uint8_t* __restrict__ k_cache, uint8_t* __restrict__ v_cache,
                                     float* __restrict__ k_scale, float* __restrict__ v_scale, int T, int Hq, int Hk,
                                     int page_size, int rot, float log2_theta, __nv_bfloat16* __restrict__ kd_out,
                                     __nv_bfloat16* __restrict__ vd_out, const float* __restrict__ q_norm_w,
                                     const float* __restrict__ k_norm_w, float norm_eps, int row_stride,
                                     const RopeScale ys, int value_blocks) {
  rope_rows<D, 1>(qkv, positions, slots, q_out, k_cache, v_cache, k_scale, v_scale, T, Hq, Hk, page_size, rot, log2_theta, kd_out, vd_out, q_norm_w, k_norm_w,
                  norm_eps, row_stride, ys, value_blocks);
}

constexpr int kRopeHeads = 8;
template <int D, int kPerSm>  // CTAs per SM
__global__ void __launch_bounds__(256, kPerSm) rope_kv_write_heads_kernel(const __nv_bfloat16* __restrict__ qkv, const int* __restrict__ positions,
                                     const int* __restrict__ slots, __nv_bfloat16* __restrict__ q_out,
                                     uint8_t* __restrict__ k_cache, uint8_t* __restrict__ v_cache,
                                     float* __restrict__ k_scale, float* __restrict__ v_scale, int T, int Hq, int Hk,
                                     int page_size, int rot, float log2_theta, __nv_bfloat16* __restrict__ kd_out,
                                     __nv_bfloat16* __restrict__ vd_out, const float* __restrict__ q_norm_w,
                                     const float* __restrict__ k_norm_w, float norm_eps, int row_stride,
                                     const RopeScale ys, int value_blocks) {
  rope_rows<D, kRopeHeads>(qkv, positions, slots, q_out, k_cache, v_cache, k_scale, v_scale, T, Hq, Hk, page_size, rot, log2_theta, kd_out, vd_out, q_norm_w, k_norm_w,
                       norm_eps, row_stride, ys, value_blocks);
}

// ---------------------------------------------------------------------------------------------
// Greedy sampling: arg-max over the vocabulary, one CTA per row (lowest index wins ties).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float logit_value(__nv_bfloat16 v) { return __bfloat162float(v); }
__device__ __forceinline__ float logit_value(float v) { return v; }

template <typename T>
__global__ void argmax_kernel(const T* __restrict__ logits, int* __restrict__ out, int V, int stride) {
  pdl_trigger();
  pdl_wait();
  __shared__ float sv[32];
  __shared__ int si[32];
  const T* row = logits + size_t(blockIdx.x) * stride;
  float best = -FLT_MAX;
  int bi = 0x7fffffff;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    const float v = logit_value(row[i]);
    if (v > best) { best = v; bi = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { sv[warp] = best; si[warp] = bi; }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    best = lane < nw ? sv[lane] : -FLT_MAX;
    bi = lane < nw ? si[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) out[blockIdx.x] = bi;
  }
}

// Wide vocabularies, few rows: the row is split over several CTAs.  Each folds its best (value, index) into a 64-bit
// key -- order-preserving value bits above the inverted index, so the larger value and then the lower index win an
// atomicMax -- and the last CTA of the row to arrive writes the result and clears the row's scratch for the next
// launch.  The scratch is static device memory: nothing to allocate, safe under graph capture; launches that share
// it must be ordered on one stream.
constexpr int kArgmaxRows = 8192;
__device__ unsigned long long g_argmax_key[kArgmaxRows];
__device__ unsigned int g_argmax_count[kArgmaxRows];

template <typename T>
__global__ void argmax_split_kernel(const T* __restrict__ logits, int* __restrict__ out, int V, int stride) {
  pdl_trigger();
  pdl_wait();
  __shared__ unsigned long long sk[8];
  const int b = blockIdx.x, seg = blockIdx.y, nseg = gridDim.y;
  const int per = (V + nseg - 1) / nseg;
  const int lo = seg * per, hi = min(V, lo + per);
  const T* row = logits + size_t(b) * stride;
  unsigned long long key = 0ull;
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const uint32_t u = __float_as_uint(logit_value(row[i]));
    const uint32_t ord = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    const unsigned long long k = (static_cast<unsigned long long>(ord) << 32) | (0xffffffffu - uint32_t(i));
    key = k > key ? k : key;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, o);
    key = other > key ? other : key;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sk[warp] = key;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (blockDim.x >> 5); ++w) key = sk[w] > key ? sk[w] : key;
    atomicMax(&g_argmax_key[b], key);
    __threadfence();
    if (atomicAdd(&g_argmax_count[b], 1u) == uint32_t(nseg - 1)) {
      __threadfence();
      const unsigned long long best = atomicExch(&g_argmax_key[b], 0ull);
      out[b] = int(0xffffffffu - uint32_t(best & 0xffffffffull));
      g_argmax_count[b] = 0u;
    }
  }
}

__global__ void embed_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                             __nv_bfloat16* __restrict__ out, int H) {
  pdl_trigger();
  pdl_wait();
  const size_t row = blockIdx.x;
  const size_t src = size_t(ids[row]);
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x)
    reinterpret_cast<uint4*>(out + row * H)[i] = reinterpret_cast<const uint4*>(table + src * H)[i];
}

// Per-step bookkeeping that lives inside the captured decode graph: the sampled token becomes the next
// input, the position advances, the KV slot of the new token is looked up in the page table.
__global__ void decode_advance_kernel(const int* __restrict__ sampled, int* __restrict__ input_ids,
                                      int* __restrict__ positions, int* __restrict__ seq_lens,
                                      int* __restrict__ slots, const int* __restrict__ block_table, int B,
                                      int max_pages, int page_size, const int* __restrict__ active) {
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  if (active && !active[b]) { slots[b] = -1; return; }
  if (sampled) input_ids[b] = sampled[b];
  const int pos = seq_lens[b];  // position of the token about to be written
  positions[b] = pos;
  const int page = block_table[size_t(b) * max_pages + pos / page_size];
  slots[b] = page * page_size + pos % page_size;
  seq_lens[b] = pos + 1;
}

}  // namespace mfq

using namespace mfq;

extern "C" int mfq_rmsnorm_quant(const void* x, const void* residual, void* residual_out, const void* w, void* q_out,
                                 float* scale_out, void* y_out, int M, int H, float eps, cudaStream_t stream) {
  if (H % 8 || M <= 0) return -1;
  int threads = ((H / 8 + kNormVecs - 1) / kNormVecs + 31) / 32 * 32;
  if (threads < 32) threads = 32;
  if (threads > 1024) return -1;
  // few rows (decode): the kernel is pure latency, so spread a row over as many threads as it has 16-byte vectors
  if (M <= 1024) threads = max(threads, min(512, (H / 8 + 31) / 32 * 32));  // 512: the register file allows no more
  const auto launch = [&](auto kernel) {
    launch_kernel(kernel, dim3(M), dim3(threads), 0, stream, static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(residual),
                  static_cast<__nv_bfloat16*>(residual_out), static_cast<const __nv_bfloat16*>(w), static_cast<uint8_t*>(q_out), scale_out,
                  static_cast<__nv_bfloat16*>(y_out), H, eps);
  };
  // vectors a thread has to hold: registers for no more than that leave room for more rows on an SM
  if (H / 8 <= threads) launch(rmsnorm_quant_kernel<1>);
  else if (H / 8 <= 4 * threads) launch(M <= 2 * 148 ? rmsnorm_quant_kernel<4, true> : rmsnorm_quant_kernel<4>);
  else launch(M <= 1600 && H <= 4096 ? rmsnorm_quant_kernel<kNormVecs, true> : rmsnorm_quant_kernel<kNormVecs>);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

// Threads per row: with few rows the kernel is latency, so a row is spread over many threads; with many, a thread takes as many
// vectors as it can hold, and an SM more rows.
static int quant_row_threads(int M, int K) {
  if (M < 512) return K >= 4096 ? 512 : 256;
  const int t = (K / 8 + kRowVecs - 1) / kRowVecs;
  return t < 64 ? 64 : t > 512 ? 512 : (t + 31) / 32 * 32;
}

extern "C" int mfq_quant_rows(const void* x, void* q_out, float* scale_out, int M, int K, int in_stride, int swiglu,
                              cudaStream_t stream) {
  if (K % 8 || in_stride % 8 || M <= 0) return -1;
  const int threads = quant_row_threads(M, K);
  if (swiglu ? M >= 5000 && K <= 512 : M >= 256 && K <= 1024) {
    const auto kernel = swiglu ? quant_short_rows_kernel<1, 2> : K <= 512 ? quant_short_rows_kernel<0, 2> : quant_short_rows_kernel<0, 4>;
    launch_kernel(kernel, dim3((M + 7) / 8), dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q_out), scale_out, M, K,
                  in_stride);
    return cudaGetLastError() == cudaSuccess ? 0 : -7;
  }
  if (swiglu && M <= 256 && K % (8 * kSwigluSplit) == 0 && K / 8 / kSwigluSplit <= 256 * kSwigluVecs && K >= 4096) {
    launch_kernel(silu_mul_quant_split_kernel, dim3(M * kSwigluSplit), dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(x),
                  static_cast<uint8_t*>(q_out), scale_out, K, in_stride);
    return cudaGetLastError() == cudaSuccess ? 0 : -7;
  }
  if (swiglu)
    launch_kernel(K == 8 * kRowVecs * threads ? quant_rows_kernel<1, true> : quant_rows_kernel<1>, dim3(M), dim3(threads), 0, stream, static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q_out), scale_out, K, in_stride, static_cast<const __nv_bfloat16*>(nullptr), 0);
  else
    launch_kernel(quant_rows_kernel<0>, dim3(M), dim3(threads), 0, stream, static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q_out), scale_out, K, in_stride, static_cast<const __nv_bfloat16*>(nullptr), 0);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

// fp8 rows of x * sigmoid(gate): the output gate of gated attention, fused with the quantization that feeds o_proj.
extern "C" int mfq_gate_quant_rows(const void* x, const void* gate, void* q_out, float* scale_out, int M, int K,
                                   int in_stride, int gate_stride, cudaStream_t stream) {
  if (K % 8 || in_stride % 8 || gate_stride % 8 || M <= 0) return -1;
  launch_kernel(quant_rows_kernel<2>, dim3(M), dim3(quant_row_threads(M, K)), 0, stream, static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q_out),
                                                                scale_out, K, in_stride, static_cast<const __nv_bfloat16*>(gate),
                                                                gate_stride);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

// q_norm_w / k_norm_w ([D] fp32, may be null): per-head RMSNorm of q / k before the rotation; row_stride: elements
// between token rows of qkv (>= (Hq + 2 Hk) * D; an attention output gate may follow the v heads).
// yarn_*: context extension (see RopeScale); factor 1 and mscale 1 are the plain rotation.
extern "C" int mfq_rope_kv_write_yarn(const void* qkv, const int* positions, const int* slots, void* q_out, void* k_cache,
                                      void* v_cache, float* k_scale, float* v_scale, int T, int Hq, int Hk, int D,
                                      int page_size, int rot, float theta, void* kd_out, void* vd_out,
                                      const float* q_norm_w, const float* k_norm_w, float norm_eps, int row_stride,
                                      float yarn_factor, float yarn_low, float yarn_high, float yarn_mscale,
                                      cudaStream_t stream) {
  if (T <= 0 || row_stride < (Hq + 2 * Hk) * D || row_stride % 8) return -1;
  if (!(yarn_factor >= 1.f) || !(yarn_high > yarn_low) || !(yarn_mscale > 0.f)) return -1;
  // A warp per head, or one per kRopeHeads heads of a token, whose angles (sine, cosine and the frequency's power, a good part of a head's
  // work) it evaluates once.  That needs full rotary, enough heads that the fewer and longer warps still fill the GPU, and groups that are
  // three quarters full; and its stores are up to 8 bytes wide, where a warp per head writes values one by one.  Up to 128 wide the eight heads
  // of a warp are requested together, and from 128 on a prompt's values of whole pages go by themselves (value_group).
  // On a B200, a warp per head | eight heads | and values by pages, one prompt | prompts of 40 to 200 tokens packed:
  //   48 heads of 128, 378 tokens 8.1 | 8.3 | 8.1 | 8.2 us, 605 11.5 | 10.0 | 9.2 | 9.6, 834 14.9 | 13.5 | 11.9 | 12.3, 2084 32 | 22 | 20.3 | 20.6
  //   16 of 128, 1132 tokens 6.5 | 7.6 | 5.6 | 6.3, 1813 9.3 | 8.5 | 6.3 | 6.6    16 of 256, 1132 15.4 | 22.8 | 12.3 | 13.6, 2063 24.9 | 26.6 | 17.8 | 17.9
  // so the line is 18000 heads of work with values by pages, and 36000 without (rows of a decode batch, other pages).
  // Heads of 64 have no such values: 48 of them, 459 tokens 5.9 | 7.3 us, 605 7.3 | 7.3, 688 8.0 | 7.4.  Their warps are alike in length, so waves
  // of CTAs are what counts: four CTAs per SM take 7.3 us a wave, 11.8 two, 17.2 three, and six, with 28 bytes of spills, 10.4 and 15.0.
  const int heads = Hq + 2 * Hk, full_groups = (heads + kRopeHeads - 1) / kRopeHeads;
  const bool aligned = (reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(kd_out) | reinterpret_cast<uintptr_t>(vd_out)) % 8 == 0;
  const bool by_pages = D >= 128 && page_size == 16 && reinterpret_cast<uintptr_t>(qkv) % 8 == 0 && row_stride % 4 == 0 && reinterpret_cast<uintptr_t>(v_cache) % 16 == 0;
  const long shared_from = by_pages && kd_out ? 18000 : D == 64 ? 30000 : 36000;
  const bool shared = rot == D && long(T) * heads >= shared_from && 4 * heads >= 3 * kRopeHeads * full_groups && aligned;
  // values of whole pages sixteen tokens at a time
  const int value_blocks = shared && by_pages ? (T + kGroupTokens - 1) / kGroupTokens * ((Hk + 7) / 8) : 0;
  const int blocks = value_blocks + int((long(T) * (shared ? full_groups : heads) + 7) / 8);
  const bool six = D == 64 && (blocks > 8 * 148 || (blocks > 4 * 148 && blocks <= 6 * 148));
  const float l2t = log2f(theta);
  const RopeScale ys{yarn_factor, yarn_low, yarn_high, yarn_mscale};
#define MFQ_ROPE(DD)                                                                                             \
  launch_kernel(!shared ? rope_kv_write_kernel<DD> : six ? rope_kv_write_heads_kernel<DD, DD == 64 ? 6 : 4> : rope_kv_write_heads_kernel<DD, 4>, dim3(blocks), dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(qkv), positions, slots, \
      static_cast<__nv_bfloat16*>(q_out), static_cast<uint8_t*>(k_cache), static_cast<uint8_t*>(v_cache),      \
      k_scale, v_scale, T, Hq, Hk, page_size, rot, l2t, static_cast<__nv_bfloat16*>(kd_out),                   \
      static_cast<__nv_bfloat16*>(vd_out), q_norm_w, k_norm_w, norm_eps, row_stride, ys, value_blocks)
  if (D == 128) MFQ_ROPE(128);
  else if (D == 64) MFQ_ROPE(64);
  else if (D == 256) MFQ_ROPE(256);
  else return -1;
#undef MFQ_ROPE
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

extern "C" int mfq_rope_kv_write_ex(const void* qkv, const int* positions, const int* slots, void* q_out, void* k_cache,
                                    void* v_cache, float* k_scale, float* v_scale, int T, int Hq, int Hk, int D,
                                    int page_size, int rot, float theta, void* kd_out, void* vd_out,
                                    const float* q_norm_w, const float* k_norm_w, float norm_eps, int row_stride,
                                    cudaStream_t stream) {
  return mfq_rope_kv_write_yarn(qkv, positions, slots, q_out, k_cache, v_cache, k_scale, v_scale, T, Hq, Hk, D, page_size,
                                rot, theta, kd_out, vd_out, q_norm_w, k_norm_w, norm_eps, row_stride, 1.f, 0.f, 1.f, 1.f,
                                stream);
}

extern "C" int mfq_rope_kv_write(const void* qkv, const int* positions, const int* slots, void* q_out, void* k_cache,
                                 void* v_cache, float* k_scale, float* v_scale, int T, int Hq, int Hk, int D,
                                 int page_size, int rot, float theta, void* kd_out, void* vd_out,
                                 cudaStream_t stream) {
  return mfq_rope_kv_write_ex(qkv, positions, slots, q_out, k_cache, v_cache, k_scale, v_scale, T, Hq, Hk, D, page_size, rot,
                              theta, kd_out, vd_out, nullptr, nullptr, 0.f, (Hq + 2 * Hk) * D, stream);
}

template <typename T>
static int launch_argmax(const void* logits, int* out, int B, int V, int stride, cudaStream_t stream) {
  const int segs = V / 4096 > 32 ? 32 : V / 4096;
  if (segs >= 2 && B <= kArgmaxRows && B * segs <= 4096)
    launch_kernel(argmax_split_kernel<T>, dim3(B, segs), dim3(256), 0, stream, static_cast<const T*>(logits), out, V, stride);
  else
    launch_kernel(argmax_kernel<T>, dim3(B), dim3(1024), 0, stream, static_cast<const T*>(logits), out, V, stride);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

extern "C" int mfq_argmax(const void* logits, int* out, int B, int V, int stride, cudaStream_t stream) {
  return launch_argmax<__nv_bfloat16>(logits, out, B, V, stride, stream);
}

// fp32 logits (models that run in full precision)
extern "C" int mfq_argmax_f32(const void* logits, int* out, int B, int V, int stride, cudaStream_t stream) {
  return launch_argmax<float>(logits, out, B, V, stride, stream);
}

extern "C" int mfq_embed(const int* ids, const void* table, void* out, int T, int H, cudaStream_t stream) {
  if (H % 8) return -1;
  launch_kernel(embed_kernel, dim3(T), dim3(128), 0, stream, ids, static_cast<const __nv_bfloat16*>(table), static_cast<__nv_bfloat16*>(out), H);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

extern "C" int mfq_decode_advance(const int* sampled, int* input_ids, int* positions, int* seq_lens, int* slots,
                                  const int* block_table, int B, int max_pages, int page_size, const int* active,
                                  cudaStream_t stream) {
  launch_kernel(decode_advance_kernel, dim3((B + 127) / 128), dim3(128), 0, stream, sampled, input_ids, positions, seq_lens, slots,
                                                             block_table, B, max_pages, page_size, active);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

// ---------------------------------------------------------------------------------------------
// SwiGLU without quantization: out[row, :I] = silu(x[row, :I]) * x[row, I:2I] in bf16 (input of bf16-activation GEMMs).
// ---------------------------------------------------------------------------------------------
namespace mfq {
__global__ void silu_mul_bf16_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ out, int I, int in_stride) {
  pdl_trigger();
  pdl_wait();
  const size_t row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * in_stride;
  for (int v = blockIdx.y * blockDim.x + threadIdx.x; v < I / 8; v += gridDim.y * blockDim.x) {
    const uint4 a = *reinterpret_cast<const uint4*>(xr + v * 8);
    const uint4 b = *reinterpret_cast<const uint4*>(xr + I + v * 8);
    const __nv_bfloat16* ab = reinterpret_cast<const __nv_bfloat16*>(&a);
    const __nv_bfloat16* bb = reinterpret_cast<const __nv_bfloat16*>(&b);
    uint4 o;
    __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float g = __bfloat162float(ab[j]);
      ob[j] = __float2bfloat16(g / (1.f + __expf(-g)) * __bfloat162float(bb[j]));
    }
    *reinterpret_cast<uint4*>(out + row * I + v * 8) = o;
  }
}
}  // namespace mfq

extern "C" int mfq_silu_mul_bf16(const void* x, void* out, int M, int I, int in_stride, cudaStream_t stream) {
  if (M <= 0 || I % 8 || in_stride % 8) return -1;
  // Fewer rows than two waves of CTAs: a row over several of them, a vector per thread, instead of up to seven vectors one after the
  // other (6 rows of 14336 took 6.8 us with a CTA each).  Rows of no width keep one: a grid has no empty dimension.
  const int parts = M >= 296 ? 1 : max(1, (I / 8 + 255) / 256);
  mfq::launch_kernel(mfq::silu_mul_bf16_kernel, dim3(M, parts), dim3(256), 0, stream, static_cast<const __nv_bfloat16*>(x),
                     static_cast<__nv_bfloat16*>(out), I, in_stride);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

namespace mfq {
__global__ void __launch_bounds__(256) silu_check_kernel(const float2* __restrict__ g, float2* __restrict__ paired, float2* __restrict__ divided, int pairs) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= pairs) return;
  const float2 v = g[i];
  paired[i] = silu2(v);
  divided[i] = make_float2(v.x / (1.f + __expf(-v.x)), v.y / (1.f + __expf(-v.y)));
}
}  // namespace mfq

// silu2 and what it stands for, in fp32: a gated row's bf16 and 8 bits would hide a quotient that is off in its last places.
extern "C" int mfq_silu_check(const float* gates, float* paired, float* divided, int pairs, cudaStream_t stream) {
  if (pairs <= 0 || (reinterpret_cast<uintptr_t>(gates) | reinterpret_cast<uintptr_t>(paired) | reinterpret_cast<uintptr_t>(divided)) & 7) return -1;
  mfq::silu_check_kernel<<<(pairs + 255) / 256, 256, 0, stream>>>(reinterpret_cast<const float2*>(gates), reinterpret_cast<float2*>(paired),
                                                                  reinterpret_cast<float2*>(divided), pairs);
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}

// ---------------------------------------------------------------------------------------------
// Past K/V of one sequence out of the FP8 pages into contiguous bf16 [T, Hk, D] (code * multiplier): the keys /
// values a later prefill chunk attends to (chunked prefill, restored prefix).  A warp takes one head's page: its rows by 16 bytes, and of the
// values, which lie dim by dim, the four dims of a lane, turned in registers.  8 heads of 128 on a B200, before a warp per token and head
// that reads byte by byte (4001 tokens 10.3 us, 357 2.9), so 7.8 and 3.1.
// ---------------------------------------------------------------------------------------------
namespace mfq {
// kVectors: pages and rows on 16-byte boundaries; else bytes and single values, as a caller's own buffers may need.
template <bool kVectors>
__device__ __forceinline__ uint4 load_codes(const uint8_t* from) {
  if constexpr (kVectors) return *reinterpret_cast<const uint4*>(from);
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = from[4 * i] | uint32_t(from[4 * i + 1]) << 8 | uint32_t(from[4 * i + 2]) << 16 | uint32_t(from[4 * i + 3]) << 24;
  return make_uint4(w[0], w[1], w[2], w[3]);
}
template <bool kVectors, int N>
__device__ __forceinline__ void store_pairs(__nv_bfloat16* to, const uint32_t (&pairs)[N]) {
  if constexpr (!kVectors) {
#pragma unroll
    for (int i = 0; i < 2 * N; ++i) reinterpret_cast<unsigned short*>(to)[i] = static_cast<unsigned short>(pairs[i / 2] >> (16 * (i & 1)));
  } else if constexpr (N == 1) {
    *reinterpret_cast<uint32_t*>(to) = pairs[0];
  } else if constexpr (N == 2) {
    *reinterpret_cast<uint2*>(to) = make_uint2(pairs[0], pairs[1]);
  } else {
    static_assert(N % 4 == 0, "whole vectors");
#pragma unroll
    for (int i = 0; i < N; i += 4) reinterpret_cast<uint4*>(to)[i / 4] = make_uint4(pairs[i], pairs[i + 1], pairs[i + 2], pairs[i + 3]);
  }
}
template <int D, bool kVectors>
__global__ void __launch_bounds__(256) kv_gather_dequant_kernel(const uint8_t* __restrict__ k_cache, const uint8_t* __restrict__ v_cache,
                                         const float* __restrict__ k_scale, const float* __restrict__ v_scale,
                                         const int* __restrict__ block_row, __nv_bfloat16* __restrict__ kd,
                                         __nv_bfloat16* __restrict__ vd, int T, int Hk) {
  pdl_trigger();
  pdl_wait();
  constexpr int P = 16;  // tokens of a page
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int pages = (T + P - 1) / P, side = gw / (pages * Hk), at = gw - side * (pages * Hk);  // keys, then values
  if (side > 1) return;
  const int pi = at / Hk, h = at - pi * Hk, t0 = pi * P, rows = min(P, T - t0);
  const size_t ph = size_t(block_row[pi]) * Hk + h;
  const float my_scale = (side ? v_scale : k_scale)[ph * P + (lane & 15)];
  auto two = [](uint32_t codes, int j, float s) {  // codes j and j + 1 of a word
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(__nv_fp8x2_storage_t(codes >> (8 * j)), __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    const __nv_bfloat162 r = __floats2bfloat162_rn(f.x * s, f.y * s);
    return *reinterpret_cast<const uint32_t*>(&r);
  };
  if (side == 0) {  // [D / 64 chunks][16 tokens][64 dims]
    const uint8_t* src = k_cache + ph * (size_t(P) * D);
#pragma unroll
    for (int i = 0; i < D / 32; ++i) {
      const int v = i * 32 + lane, chunk = v >> 6, t = (v >> 2) & 15, dim = chunk * 64 + (v & 3) * 16;
      const uint4 c = load_codes<kVectors>(src + v * 16);
      const float s = __shfl_sync(0xffffffffu, my_scale, t);
      if (t < rows) {
        const uint32_t row[8] = {two(c.x, 0, s), two(c.x, 2, s), two(c.y, 0, s), two(c.y, 2, s), two(c.z, 0, s), two(c.z, 2, s), two(c.w, 0, s), two(c.w, 2, s)};
        store_pairs<kVectors>(kd + (size_t(t0 + t) * Hk + h) * D + dim, row);
      }
    }
    return;
  }
  constexpr int VPL = D / 32;  // dims of a lane
  const uint8_t* src = v_cache + ph * (size_t(P) * D) + lane * VPL * P;
  uint4 c[VPL];
#pragma unroll
  for (int j = 0; j < VPL; ++j) c[j] = load_codes<kVectors>(src + j * P);
#pragma unroll
  for (int t = 0; t < P; ++t) {
    const float s = __shfl_sync(0xffffffffu, my_scale, t);
    const int word = (t & 7) >> 1, byte = 8 * (2 * (t >> 3) + (t & 1));  // word g of a dim holds tokens 2g, 2g + 1, 2g + 8, 2g + 9
    uint32_t out[VPL / 2];
#pragma unroll
    for (int j = 0; j < VPL; j += 2) {
      const uint32_t a = word == 0 ? c[j].x : word == 1 ? c[j].y : word == 2 ? c[j].z : c[j].w;
      const uint32_t b = word == 0 ? c[j + 1].x : word == 1 ? c[j + 1].y : word == 2 ? c[j + 1].z : c[j + 1].w;
      out[j / 2] = two(__byte_perm(a, b, (byte >> 3) | (4 + (byte >> 3)) << 4), 0, s);
    }
    if (t < rows) store_pairs<kVectors>(vd + (size_t(t0 + t) * Hk + h) * D + lane * VPL, out);
  }
}
}  // namespace mfq

// block_row: the sequence's page ids ([ceil(T / page_size)] int32, device); kd / vd: [T, Hk, D] bf16.
extern "C" int mfq_kv_gather_dequant(const void* k_cache, const void* v_cache, const float* k_scale, const float* v_scale,
                                     const int* block_row, void* kd, void* vd, int T, int Hk, int D, int page_size,
                                     cudaStream_t stream) {
  if (T <= 0 || Hk <= 0 || page_size != 16) return -1;
  const bool vectors = ((reinterpret_cast<uintptr_t>(kd) | reinterpret_cast<uintptr_t>(vd) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) == 0;
  const int blocks = (2 * ((T + 15) / 16) * Hk + 7) / 8;
#define MFQ_GATHER(DD)                                                                                              \
  mfq::launch_kernel(vectors ? mfq::kv_gather_dequant_kernel<DD, true> : mfq::kv_gather_dequant_kernel<DD, false>, dim3(blocks), dim3(256), 0, stream,                        \
                     static_cast<const uint8_t*>(k_cache), static_cast<const uint8_t*>(v_cache), k_scale, v_scale,  \
                     block_row, static_cast<__nv_bfloat16*>(kd), static_cast<__nv_bfloat16*>(vd), T, Hk)
  if (D == 128) MFQ_GATHER(128);
  else if (D == 64) MFQ_GATHER(64);
  else if (D == 256) MFQ_GATHER(256);
  else return -1;
#undef MFQ_GATHER
  return cudaGetLastError() == cudaSuccess ? 0 : -7;
}
