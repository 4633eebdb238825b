// Attention forward for up to 128 keys: windows of 7 x 7 or 8 x 8 tokens with their own bias, short sequences.
//
// A 128 x 128 tile of the persistent kernel (attn_fwd_sm100.cuh) holds 49 x 49 logits in a seventh of its area, and a CTA walks
// such tiles one after another through a chain of tensor-memory waits. Here a CTA of four warps takes 64 queries of one head and
// all its keys, a warp 16 of the queries: mma.sync on operands of 16 rows, the whole row of logits in registers, no running maximum.
// Bound by latency: load, two short products, store. Nothing is overlapped inside a CTA; the CTAs of an SM (window_ctas) cover each
// other. (Persistent CTAs with K and V in a TMA ring and 32 queries per warp held too few warps for that: [8,192,49] 20 us.)
// us per launch in CUDA graphs, persistent kernel and this one: [8,192,49] with a dense bias 25.0 and 10.5, without 18.1 and 8.8,
// [64,16,64] with a dense bias 17.0 and 8.3, [64,12,64] 10.4 and 5.7, [100,12,36] with 6 x 6 tables 24.4 and 8.0.
// Issue slots count next: 870 instructions a warp took 4.6 of [8,192,49]'s 11.5 us. The bias comes in pairs of columns as the logits lie
// (11.5 -> 10.9; in rows of 16 bytes turned by shuffles before), the block number is taken apart by multiplies (-> 10.5). Outputs in pairs
// instead of 16 bytes turned by shuffles: 12.1. Prefetching the next round's rows into L2: 11.0.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "attn_fwd_sm100.cuh"
#include "sm100_ptx.cuh"

namespace b200 {

enum : int { kWindowPlain = 0, kWindowDense = 1, kWindowRel = 2 };  // bias forms
constexpr int kWindowMaxKeys = 128;
constexpr int kWindowMaxRel = 32;  // values of a decomposed bias per row (rel_kh + rel_kw)
constexpr int kWindowRows = 64;    // queries per CTA
constexpr int kWindowThreads = 128;
// CTAs per SM, by registers: 72 a thread hold 64 logits of two rows but for one to four words (spilled, with a bias; without one three at 80), 128
// hold 128. us at 6 and 7: [8,192,49] / [64,192,49] with a bias
// 10.5 / 76.6 and 10.5 / 74.8, [8,64,64] 7.1 and 5.8, [100,12,36] with tables 8.4 and 8.0, but [64,12,64] without either 5.7 and 6.3.
constexpr int window_ctas(int eights, int bias) { return eights > 8 ? 4 : bias == kWindowPlain ? 6 : 7; }
// 7 x 7 windows and the 50 tokens of a 224 px image in patches of 32 need no eighth group of eight. us with it and without: [64,192,49] with a
// bias 74.5 and 72.5, [8,192,49] 10.6 and 10.5, [64,12,50] 5.85 and 5.55. (At 64 registers and eight CTAs an SM: 77.1, 10.6, 6.5.)
// Other counts with an odd number of groups, 17 to 24 and so on, have less from it, and six more forms for every type and bias have not been
// taken for that. us with the last group and without, dense bias: [64,48,24] 9.1 and 8.8, [64,48,40] 12.5 and 12.2, [64,48,72] 45.3 and 45.3,
// [8,64,104] 11.1 and 11.0, [64,48,120] 52.5 and 53.0; plain 8.0 and 7.8, 11.5 and 11.4, 37.3 and 37.2, 9.2 and 9.0, 45.4 and 45.5.
constexpr int window_eights(int keys) { return keys > 48 && keys <= 56 ? 7 : (keys + 15) / 16 * 2; }

struct WindowParams {
  const void* q;
  const void* k;
  const void* v;
  void* o;
  int64_t q_stride[3], k_stride[3], v_stride[3], o_stride[3];  // batch, token, head; elements
  int batch, heads, q_tokens, kv_tokens;
  int q_blocks;        // ceil(q_tokens / 64)
  uint64_t magic_blocks, magic_inner;  // fast_div constants of q_blocks and of the index that runs fastest
  float scale_log2, scale;
  int batch_fastest;   // heads are numbered with the batch index running fastest (a bias every image shares is then read side by side)
  const void* bias;    // dense form
  int64_t bias_stride[3];  // batch, head, query row
  int bias_half;       // its type: fp16, else bf16
  const uint16_t* rel_h;   // decomposed form, tables of the type of q
  const uint16_t* rel_w;
  int64_t rel_h_stride[3], rel_w_stride[3];
  int rel_kh, rel_kw;
  int rel_pairs;       // rows begin on four bytes and both counts are even: values are read two at a time
  uint32_t rel_one;    // 1 / scale, 16 bits
};

// Four lanes of a quad hold four words each: afterwards word j is what lane j of the quad had as word (lane & 3).
__device__ __forceinline__ void quad_transpose(uint32_t (&w)[4], int lane) {
  const bool odd = lane & 1, upper = lane & 2;
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const uint32_t r = __shfl_xor_sync(0xffffffffu, odd ? w[i] : w[i + 1], 1);
    if (odd) w[i] = r;
    else w[i + 1] = r;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t r = __shfl_xor_sync(0xffffffffu, upper ? w[i] : w[i + 2], 2);
    if (upper) w[i] = r;
    else w[i + 2] = r;
  }
}

// Rows of 64 bytes (the one-hot operand), permuted likewise: see swizzled_chunk.
__device__ __forceinline__ uint32_t onehot_chunk(uint32_t base, int row, int chunk) { return base + row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4); }

// Loads through L2 only (the kernel in front may have written the data while this one was already on the SM), nothing where !valid.
// Written as predicated instructions, so that a row's loads are all in flight before the first is used.
__device__ __forceinline__ uint32_t load_u32_if(const uint16_t* src, bool valid) {
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.cg.u32 %0, [%1];\n\t}\n" : "=&r"(v) : "l"(src), "r"(valid ? 1 : 0));
  return v;
}
__device__ __forceinline__ uint32_t load_u16_if(const uint16_t* src, bool valid) {
  uint32_t v;
  asm volatile("{\n\t.reg .pred p;\n\t.reg .u16 h;\n\tsetp.ne.s32 p, %2, 0;\n\tmov.u16 h, 0;\n\t@p ld.global.cg.u16 h, [%1];\n\tcvt.u32.u16 %0, h;\n\t}\n"
               : "=r"(v) : "l"(src), "r"(valid ? 1 : 0));
  return v;
}

template <typename T, int ROWS>
__device__ __forceinline__ void window_load(uint32_t smem, const T* rows, int64_t stride, int count) {
#pragma unroll
  for (int i = 0; i < ROWS * 8 / kWindowThreads; ++i) {
    const int row = (threadIdx.x >> 3) + i * (kWindowThreads / 8), chunk = threadIdx.x & 7;
    cp_async_16(swizzled_chunk(smem, row, chunk), rows + (row < count ? row : 0) * stride + chunk * 8, row < count);
  }
}

// EIGHTS = ceil(kv_tokens / 8), of which an odd number is only told from the next even one where window_eights() says so. Grid: q_blocks *
// batch * heads.
template <typename T, int BIAS, int EIGHTS>
__global__ void __launch_bounds__(kWindowThreads, window_ctas(EIGHTS, BIAS)) attn_window_kernel(const WindowParams p) {
  constexpr int GROUPS = (EIGHTS + 1) / 2;  // of 16 keys: what a step of the second product takes
  __shared__ __align__(128) uint8_t smem_q[kWindowRows * 128];
  __shared__ __align__(128) uint8_t smem_k[GROUPS * 16 * 128];
  __shared__ __align__(128) uint8_t smem_v[GROUPS * 16 * 128];
  __shared__ __align__(128) uint8_t smem_e[BIAS == kWindowRel ? GROUPS * 16 * 64 : 16];
  const uint32_t sq = smem_u32(smem_q), sk = smem_u32(smem_k), sv = smem_u32(smem_v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  constexpr float kNone = -__builtin_huge_valf();

  const int item = fast_div(static_cast<int>(blockIdx.x), p.magic_blocks), row0 = (static_cast<int>(blockIdx.x) - item * p.q_blocks) * kWindowRows;
  const int inner = p.batch_fastest ? p.batch : p.heads, outer = fast_div(item, p.magic_inner), rest = item - outer * inner;
  const int b = p.batch_fastest ? rest : outer, h = p.batch_fastest ? outer : rest;
  const int my_row0 = row0 + warp * 16;
  auto row_of = [&](int r) { return my_row0 + 8 * r + g; };

  if constexpr (BIAS == kWindowRel) {
    // Key (y, x): 1 / scale at value y and at value rel_kh + x of its row.
    const uint32_t se = smem_u32(smem_e);
    for (int i = threadIdx.x; i < GROUPS * 16 * 4; i += kWindowThreads) {
      const int key = i >> 2, c = i & 3;
      const int y = key / p.rel_kw, x = p.rel_kh + key - y * p.rel_kw;
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int lo = 8 * c + 2 * e;
        w[e] = (lo == y || lo == x ? p.rel_one : 0u) | (lo + 1 == y || lo + 1 == x ? p.rel_one << 16 : 0u);
      }
      st_shared_v4(onehot_chunk(se, key, c), make_uint4(w[0], w[1], w[2], w[3]));
    }
  }
  grid_dependency_wait();
  grid_launch_dependents();
  window_load<T, kWindowRows>(sq, static_cast<const T*>(p.q) + b * p.q_stride[0] + h * p.q_stride[2] + row0 * p.q_stride[1], p.q_stride[1], p.q_tokens - row0);
  window_load<T, GROUPS * 16>(sk, static_cast<const T*>(p.k) + b * p.k_stride[0] + h * p.k_stride[2], p.k_stride[1], p.kv_tokens);
  window_load<T, GROUPS * 16>(sv, static_cast<const T*>(p.v) + b * p.v_stride[0] + h * p.v_stride[2], p.v_stride[1], p.kv_tokens);
  cp_async_commit();

  // The rows' bias, in flight with the operands: a lane loads the pairs of columns whose logits it will hold. A pair never reaches behind
  // the row's end.
  [[maybe_unused]] uint32_t bw[2][EIGHTS];
  if constexpr (BIAS == kWindowDense) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const bool valid = row_of(r) < p.q_tokens;
      const uint16_t* src = static_cast<const uint16_t*>(p.bias) + b * p.bias_stride[0] + h * p.bias_stride[1] + (valid ? row_of(r) : 0) * p.bias_stride[2] + 2 * t;
#pragma unroll
      for (int j = 0; j < EIGHTS; ++j) bw[r][j] = load_u32_if(src + 8 * j, valid && 8 * j + 2 * t + 1 < p.kv_tokens);
      if ((p.kv_tokens & 1) != 0) {  // the last key's half of its pair
#pragma unroll
        for (int j = EIGHTS - 2 < 0 ? 0 : EIGHTS - 2; j < EIGHTS; ++j) bw[r][j] |= load_u16_if(src + 8 * j, valid && 8 * j + 2 * t + 1 == p.kv_tokens);
      }
    }
  }
  // Decomposed: a row's values are an operand like its query, against the one-hot grid coordinates of the keys.
  float sum[2] = {0.f, 0.f};  // this thread's share
  [[maybe_unused]] uint32_t ra[2][4];
  if constexpr (BIAS == kWindowRel) {
    constexpr uint32_t inf = std::is_same<T, __half>::value ? 0x7c00u : 0x7f80u;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const bool valid = row_of(r) < p.q_tokens;
      const int row = valid ? row_of(r) : 0;
      const uint16_t* rh = p.rel_h + b * p.rel_h_stride[0] + h * p.rel_h_stride[1] + row * p.rel_h_stride[2];
      const uint16_t* rw = p.rel_w + b * p.rel_w_stride[0] + h * p.rel_w_stride[1] + row * p.rel_w_stride[2];
      uint32_t v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int at = 8 * c + 2 * t;
        if (p.rel_pairs) {
          v[c] = load_u32_if(at < p.rel_kh ? rh + at : rw + (at - p.rel_kh), valid && at < p.rel_kh + p.rel_kw);
        } else {
          v[c] = load_u16_if(at < p.rel_kh ? rh + at : rw + (at - p.rel_kh), valid && at < p.rel_kh + p.rel_kw);
          v[c] |= load_u16_if(at + 1 < p.rel_kh ? rh + at + 1 : rw + (at + 1 - p.rel_kh), valid && at + 1 < p.rel_kh + p.rel_kw) << 16;
        }
      }
      bool any_inf = false;  // an infinity would meet zeros: it goes in as the largest finite value (see kBiasDecomposedMma)
#pragma unroll
      for (int c = 0; c < 4; ++c) ra[c >> 1][(c & 1) * 2 + r] = clamp_finite2(v[c], inf, &any_inf);
      if (__any_sync(0xffffffffu, any_inf)) sum[r] = t == 0 && valid ? infinite_row(rh, p.rel_kh, rw, p.rel_kw, inf) : 0.f;  // a NaN stays in the sum
    }
  }

  cp_async_wait<0>();
  __syncthreads();
  if (my_row0 < p.q_tokens) {
    const int k_row = (lane & 7) + ((lane >> 4) << 3), k_chunk = (lane >> 3) & 1;  // ldmatrix addresses: 16 keys x 16 of the head dim
    float s[EIGHTS][4];  // rows g and g + 8, keys 8 j + 2 t and + 1
#pragma unroll
    for (int j = 0; j < EIGHTS; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      uint32_t a[4];
      ldmatrix_x4(a, swizzled_chunk(sq, warp * 16 + (lane & 15), 2 * d + (lane >> 4)));
#pragma unroll
      for (int i = 0; i < GROUPS; ++i) {
        uint32_t kk[4];
        ldmatrix_x4(kk, swizzled_chunk(sk, i * 16 + k_row, 2 * d + k_chunk));
        mma_16816<T>(s[2 * i], a, kk[0], kk[1]);
        if (2 * i + 1 < EIGHTS) mma_16816<T>(s[2 * i + 1], a, kk[2], kk[3]);
      }
    }
    if constexpr (BIAS == kWindowRel) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (16 * c >= p.rel_kh + p.rel_kw) break;
#pragma unroll
        for (int i = 0; i < GROUPS; ++i) {
          uint32_t kk[4];
          ldmatrix_x4(kk, onehot_chunk(smem_u32(smem_e), i * 16 + k_row, 2 * c + k_chunk));
          mma_16816<T>(s[2 * i], ra[c], kk[0], kk[1]);
          if (2 * i + 1 < EIGHTS) mma_16816<T>(s[2 * i + 1], ra[c], kk[2], kk[3]);
        }
      }
    }
    const float unit = BIAS == kWindowDense ? kLog2e : p.scale_log2;
    uint32_t probs[2 * GROUPS][2];
    if constexpr (EIGHTS % 2 != 0) probs[EIGHTS][0] = probs[EIGHTS][1] = 0;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if constexpr (BIAS == kWindowDense) {  // natural units, s * scale + bias; log2(e) rides on the FMA in front of the exponential
#pragma unroll
        for (int j = 0; j < EIGHTS; ++j) {
          const float2 x = ffma2(make_float2(s[j][2 * r], s[j][2 * r + 1]), make_float2(p.scale, p.scale), unpack2(bw[r][j], p.bias_half != 0));
          s[j][2 * r] = x.x;
          s[j][2 * r + 1] = x.y;
        }
      }
#pragma unroll
      for (int j = EIGHTS - 2 < 0 ? 0 : EIGHTS - 2; j < EIGHTS; ++j)  // the keys that pad the last group
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (8 * j + 2 * t + e >= p.kv_tokens) s[j][2 * r + e] = kNone;
      float top = fmaxf(s[0][2 * r], s[0][2 * r + 1]);
#pragma unroll
      for (int j = 1; j < EIGHTS; ++j) top = max3(top, s[j][2 * r], s[j][2 * r + 1]);
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2)) * unit;
      const float shift = top == kNone ? 0.f : -top;
      float2 part = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < EIGHTS; ++j) {
        const float2 x = ffma2(make_float2(s[j][2 * r], s[j][2 * r + 1]), make_float2(unit, unit), make_float2(shift, shift));
        const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
        part = fadd2(part, e);
        probs[j][r] = pack2<T>(e.x, e.y);
      }
      sum[r] += part.x + part.y;
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
      sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    }

    float acc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
    for (int i = 0; i < GROUPS; ++i) {
      const uint32_t a[4] = {probs[2 * i][0], probs[2 * i][1], probs[2 * i + 1][0], probs[2 * i + 1][1]};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t vv[4];
        ldmatrix_x4_trans(vv, swizzled_chunk(sv, i * 16 + (lane & 15), 2 * j + (lane >> 4)));
        mma_16816<T>(acc[2 * j], a, vv[0], vv[1]);
        mma_16816<T>(acc[2 * j + 1], a, vv[2], vv[3]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float inv = 1.f / sum[r];
      T* dst = static_cast<T*>(p.o) + b * p.o_stride[0] + h * p.o_stride[2] + row_of(r) * p.o_stride[1];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = pack2<T>(acc[4 * half + j][2 * r] * inv, acc[4 * half + j][2 * r + 1] * inv);
        quad_transpose(w, lane);
        if (row_of(r) < p.q_tokens) reinterpret_cast<uint4*>(dst)[4 * half + t] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

}  // namespace b200
