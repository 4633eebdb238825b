// The two products behind SAM's decomposed relative-position bias, for every query of a square grid:
//   rel_h[b, head, (y, x), k] = q[b, (y, x), head, :] . rel_pos_h[y - k + side - 1, :]
//   rel_w[b, head, (y, x), k] = q[b, (y, x), head, :] . rel_pos_w[x - k + side - 1, :]      (k = 0 .. side - 1)
// q is the UNSCALED query of head dim 64, read in place from the packed qkv tensor; the tables are the module's
// parameters themselves ([2 * side - 1, 64]): the [side, side, 64] gather the upstream code builds first
// (get_rel_pos) never exists.
//
// One query token is a 16 x 64 operand (its heads) against `side` rows of either table: two small products on the same
// left operand, so q is read once. A warp takes a token, the CTA's tables lie in shared memory. mma.sync fits: the
// operands are 16 rows high and change their table rows from token to token, and the work is bound by the bytes of the
// result (12.6 MB for SAM's global grid), not by the products. On the FMA pipe, a thread per query and table row, the
// global grid took 44 us and 25 windows of 14 x 14 19 us.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "sm100_ptx.cuh"

namespace b200 {

struct RelTermsParams {
  const void* q;
  int64_t q_sb, q_sn, q_sh;  // element strides of q: batch, token, head
  const void* rel_pos_h;     // [2 * side - 1, 64]
  const void* rel_pos_w;
  void* rel_h;               // [batch, heads, side * side, side], contiguous
  void* rel_w;
  int batch, heads, side;
  int parts;                 // CTAs per grid row
  int tables_wide, out_wide; // both tables / results are 16-byte aligned (else 4-byte)
};

constexpr int kRelWarps = 4;
constexpr int kRelMaxSide = 64;

template <typename T>
__device__ __forceinline__ uint32_t rel_pack2(float lo, float hi) {
  if constexpr (std::is_same<T, __half>::value) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}

// NT: 8-column tiles of a result row, ceil(side / 8). The order of the 64 products of a sum and of the columns in a tile
// is free, so both are chosen for wide accesses: a lane's k values are 16-byte chunks of q's and the tables' rows (chunk
// t and t + 4 of eight), and its columns are the 2 NT consecutive ones from 2 NT t on (t = lane % 4).
template <typename T, int NT>
__global__ void __launch_bounds__(kRelWarps * 32) sam_rel_terms_kernel(const RelTermsParams p) {
  // Table rows as eight 16-byte chunks; odd rows have their halves swapped, so that two neighbouring rows, which a quarter
  // of a warp reads together, use all banks.
  extern __shared__ uint4 rel_tables[];
  const int side = p.side, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int row_id = blockIdx.x / p.parts, part = blockIdx.x - row_id * p.parts;
  const int b = row_id / side, y = row_id - b * side;
  uint4* const table_h = rel_tables;              // row k: rel_pos_h[y - k + side - 1]
  uint4* const table_w = rel_tables + side * 8;   // rel_pos_w as it is
  grid_dependency_wait();
  grid_launch_dependents();
  const auto load = [&](const void* table, int row, int c) {
    const uint32_t* src = static_cast<const uint32_t*>(table) + row * 32 + c * 4;
    return p.tables_wide ? __ldg(reinterpret_cast<const uint4*>(src)) : make_uint4(__ldg(src), __ldg(src + 1), __ldg(src + 2), __ldg(src + 3));
  };
  for (int i = threadIdx.x; i < side * 8; i += kRelWarps * 32) {
    const int k = i >> 3, c = i & 7;
    table_h[k * 8 + (c ^ ((k & 1) << 2))] = load(p.rel_pos_h, y - k + side - 1, c);
  }
  for (int i = threadIdx.x; i < (2 * side - 1) * 8; i += kRelWarps * 32) {
    const int k = i >> 3, c = i & 7;
    table_w[k * 8 + (c ^ ((k & 1) << 2))] = load(p.rel_pos_w, k, c);
  }
  __syncthreads();
  const int x_end = side * (part + 1) / p.parts;
  const int n_tokens = side * side;
  for (int x = side * part / p.parts + warp; x < x_end; x += kRelWarps) {
    const int n = y * side + x;
    const T* q_token = static_cast<const T*>(p.q) + b * p.q_sb + n * p.q_sn;
    for (int h0 = 0; h0 < p.heads; h0 += 16) {
      // heads h0 + g and h0 + g + 8, 16-byte chunks t and t + 4 (rows past the last head repeat it; they are not stored)
      const T* q_lo = q_token + min(h0 + g, p.heads - 1) * p.q_sh;
      const T* q_hi = q_token + min(h0 + g + 8, p.heads - 1) * p.q_sh;
      uint4 lo[2], hi[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        lo[i] = __ldg(reinterpret_cast<const uint4*>(q_lo) + t + 4 * i);
        hi[i] = __ldg(reinterpret_cast<const uint4*>(q_hi) + t + 4 * i);
      }
      uint32_t a[4][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[2 * i][0] = lo[i].x; a[2 * i][1] = hi[i].x; a[2 * i][2] = lo[i].y; a[2 * i][3] = hi[i].y;
        a[2 * i + 1][0] = lo[i].z; a[2 * i + 1][1] = hi[i].z; a[2 * i + 1][2] = lo[i].w; a[2 * i + 1][3] = hi[i].w;
      }
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        float acc[NT][4];
#pragma unroll
        for (int j = 0; j < NT; ++j) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
          // lane group g holds column 2 NT (g / 2) + 2 j + g % 2 of the result: table row for that k
          const int k = min(2 * NT * (g >> 1) + 2 * j + (g & 1), side - 1);
          const int row = which == 0 ? k : x - k + side - 1;
          const uint4* table = (which == 0 ? table_h : table_w) + row * 8;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint4 v = table[(t + 4 * i) ^ ((row & 1) << 2)];
            mma_16816<T>(acc[j], a[2 * i], v.x, v.y);
            mma_16816<T>(acc[j], a[2 * i + 1], v.z, v.w);
          }
        }
        T* out = static_cast<T*>(which == 0 ? p.rel_h : p.rel_w);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int head = h0 + g + 8 * half;
          if (head >= p.heads) continue;
          T* dst = out + ((static_cast<int64_t>(b) * p.heads + head) * n_tokens + n) * side + 2 * NT * t;
          uint32_t words[NT];
#pragma unroll
          for (int j = 0; j < NT; ++j) words[j] = rel_pack2<T>(acc[j][2 * half], acc[j][2 * half + 1]);
          if (NT % 4 == 0 && side == 8 * NT && p.out_wide) {  // whole 16-byte groups, rows of whole groups
#pragma unroll
            for (int j = 0; j + 3 < NT; j += 4) *reinterpret_cast<uint4*>(dst + 2 * j) = make_uint4(words[j], words[j + 1], words[j + 2], words[j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < NT; ++j)
              if (2 * NT * t + 2 * j < side) *reinterpret_cast<uint32_t*>(dst + 2 * j) = words[j];  // side is even
          }
        }
      }
    }
  }
}

}  // namespace b200
