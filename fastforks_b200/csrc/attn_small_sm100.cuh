// Attention forward without bias for calls too small to fill the GPU with 128-row query tiles: one image's heads of a
// classifier are 24 such tiles, and a CTA of the persistent kernel then spends its time on one chain of tensor-memory
// set-up, descriptor loads, two dependent softmax steps and the store.
//
// Bound by that chain of latencies, so the work is cut as finely as it goes: a CTA takes 32 queries of one (batch, head)
// and all its keys, a warp 16 of the queries and a quarter of the keys. The quarters need no running maximum (a warp sees
// all of its logits at once) and meet in shared memory at the end. Products are mma.sync: operands of 16 rows, no tensor
// memory to allocate, results where the softmax needs them. us per launch in CUDA graphs, before (the persistent kernel) and
// now: [1,12,197] 5.9 and 3.7, [1,12,50] 4.6 and 2.2, [1,12,256] 5.9 and 3.7, [1,12,320] 7.3 and 4.2, [1,6,512] 8.0 and 5.6.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "attn_fwd_sm100.cuh"
#include "sm100_ptx.cuh"

namespace b200 {

constexpr int kSmallThreads = 256;  // 2 row groups x 4 key quarters
constexpr int kSmallRows = 32;
constexpr int kSmallMaxSteps = 8;   // 16-key steps per quarter: up to 512 keys
constexpr int kSmallPartStride = 72;  // floats per row of a partial result: 64 and padding against bank conflicts
constexpr int kSmallPartBytes = 4 * kSmallRows * kSmallPartStride * 4;

struct SmallAttnParams {
  const void* q;
  const void* k;
  const void* v;
  void* o;
  int64_t q_stride[3], k_stride[3], v_stride[3], o_stride[3];  // batch, token, head; elements
  int heads, q_tokens, kv_tokens;
  float scale_log2;
};

// Shared memory: V, then Q and K, over which the partial results are laid once every warp has its logits.
constexpr int small_attn_smem(int steps) {
  const int kv = steps * 64 * 128, qk = kSmallRows * 128 + kv;
  return kv + (qk > kSmallPartBytes ? qk : kSmallPartBytes);
}

template <typename T>
__device__ __forceinline__ void small_load(uint32_t smem, const T* rows, int64_t stride, int first, int end, int count) {
  for (int i = threadIdx.x; i < count * 8; i += kSmallThreads) {
    const int row = i >> 3, chunk = i & 7;
    const bool valid = first + row < end;
    cp_async_16(swizzled_chunk(smem, row, chunk), rows + (valid ? first + row : 0) * stride + chunk * 8, valid);
  }
}

// Grid: (ceil(q_tokens / 32), batch * heads). STEPS = ceil(kv_tokens / 64).
template <typename T, int STEPS>
__global__ void __launch_bounds__(kSmallThreads) attn_small_kernel(const SmallAttnParams p) {
  extern __shared__ __align__(128) uint8_t small_smem[];
  __shared__ float2 stats[4][kSmallRows];  // a quarter's maximum (log2 units; -inf without keys) and sum, per row
  const uint32_t sv = smem_u32(small_smem);
  const uint32_t sq = sv + STEPS * 64 * 128, sk = sq + kSmallRows * 128;
  float* part = reinterpret_cast<float*>(small_smem + STEPS * 64 * 128);

  const int b = blockIdx.y / p.heads, h = blockIdx.y - b * p.heads;
  const int row0 = blockIdx.x * kSmallRows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = warp & 1, quarter = warp >> 1;
  const int g = lane >> 2, t = lane & 3;
  const int key0 = quarter * STEPS * 16;  // of this warp

  grid_dependency_wait();
  grid_launch_dependents();
  small_load(sq, static_cast<const T*>(p.q) + b * p.q_stride[0] + h * p.q_stride[2], p.q_stride[1], row0, p.q_tokens, kSmallRows);
  small_load(sk, static_cast<const T*>(p.k) + b * p.k_stride[0] + h * p.k_stride[2], p.k_stride[1], 0, p.kv_tokens, STEPS * 64);
  cp_async_commit();
  small_load(sv, static_cast<const T*>(p.v) + b * p.v_stride[0] + h * p.v_stride[2], p.v_stride[1], 0, p.kv_tokens, STEPS * 64);
  cp_async_commit();
  cp_async_wait<1>();
  __syncthreads();

  float s[2 * STEPS][4];  // rows g and g + 8 of the group, keys key0 + 8 j + 2 t and + 1
#pragma unroll
  for (int j = 0; j < 2 * STEPS; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    uint32_t a[4];
    ldmatrix_x4(a, swizzled_chunk(sq, group * 16 + (lane & 15), 2 * d + (lane >> 4)));
#pragma unroll
    for (int i = 0; i < STEPS; ++i) {
      uint32_t kk[4];
      ldmatrix_x4(kk, swizzled_chunk(sk, key0 + i * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * d + ((lane >> 3) & 1)));
      mma_16816<T>(s[2 * i], a, kk[0], kk[1]);
      mma_16816<T>(s[2 * i + 1], a, kk[2], kk[3]);
    }
  }

  constexpr float kNone = -__builtin_huge_valf();
  float top[2] = {kNone, kNone}, sum[2] = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 2 * STEPS; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (key0 + 8 * j + 2 * t + (e & 1) >= p.kv_tokens) s[j][e] = kNone;
      top[e >> 1] = fmaxf(top[e >> 1], s[j][e]);
    }
  float shift[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    top[r] = fmaxf(top[r], __shfl_xor_sync(~0u, top[r], 1));
    top[r] = fmaxf(top[r], __shfl_xor_sync(~0u, top[r], 2)) * p.scale_log2;
    shift[r] = top[r] == kNone ? 0.f : -top[r];
  }
  uint32_t probs[2 * STEPS][2];
#pragma unroll
  for (int j = 0; j < 2 * STEPS; ++j) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float x = fast_exp2(fmaf(s[j][2 * r], p.scale_log2, shift[r])), y = fast_exp2(fmaf(s[j][2 * r + 1], p.scale_log2, shift[r]));
      sum[r] += x + y;
      probs[j][r] = pack2<T>(x, y);
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    sum[r] += __shfl_xor_sync(~0u, sum[r], 1);
    sum[r] += __shfl_xor_sync(~0u, sum[r], 2);
    if (t == 0) stats[quarter][group * 16 + 8 * r + g] = make_float2(top[r], sum[r]);
  }
  cp_async_wait<0>();
  __syncthreads();  // V is there, and nobody reads Q or K any more

  float acc[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
  for (int i = 0; i < STEPS; ++i) {
    const uint32_t a[4] = {probs[2 * i][0], probs[2 * i][1], probs[2 * i + 1][0], probs[2 * i + 1][1]};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t vv[4];
      ldmatrix_x4_trans(vv, swizzled_chunk(sv, key0 + i * 16 + (lane & 15), 2 * j + (lane >> 4)));
      mma_16816<T>(acc[2 * j], a, vv[0], vv[1]);
      mma_16816<T>(acc[2 * j + 1], a, vv[2], vv[3]);
    }
  }
  float* mine = part + (quarter * kSmallRows + group * 16 + g) * kSmallPartStride + 2 * t;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    *reinterpret_cast<float2*>(mine + 8 * j) = make_float2(acc[j][0], acc[j][1]);
    *reinterpret_cast<float2*>(mine + 8 * kSmallPartStride + 8 * j) = make_float2(acc[j][2], acc[j][3]);
  }
  __syncthreads();

  const int row = threadIdx.x >> 3, chunk = threadIdx.x & 7;  // eight values of one row per thread
  float2 st[4];
  float most = kNone, total = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    st[i] = stats[i][row];
    most = fmaxf(most, st[i].x);
  }
  float out[8] = {};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float weight = fast_exp2(st[i].x - most);
    total = fmaf(weight, st[i].y, total);
    const float4* from = reinterpret_cast<const float4*>(part + (i * kSmallRows + row) * kSmallPartStride + chunk * 8);
    const float4 lo = from[0], hi = from[1];
    out[0] = fmaf(weight, lo.x, out[0]); out[1] = fmaf(weight, lo.y, out[1]); out[2] = fmaf(weight, lo.z, out[2]); out[3] = fmaf(weight, lo.w, out[3]);
    out[4] = fmaf(weight, hi.x, out[4]); out[5] = fmaf(weight, hi.y, out[5]); out[6] = fmaf(weight, hi.z, out[6]); out[7] = fmaf(weight, hi.w, out[7]);
  }
  if (row0 + row >= p.q_tokens) return;
  const float inv = 1.f / total;
  uint4 packed;
  packed.x = pack2<T>(out[0] * inv, out[1] * inv);
  packed.y = pack2<T>(out[2] * inv, out[3] * inv);
  packed.z = pack2<T>(out[4] * inv, out[5] * inv);
  packed.w = pack2<T>(out[6] * inv, out[7] * inv);
  *reinterpret_cast<uint4*>(static_cast<T*>(p.o) + b * p.o_stride[0] + (row0 + row) * p.o_stride[1] + h * p.o_stride[2] + chunk * 8) = packed;
}

}  // namespace b200
