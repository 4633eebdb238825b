// The two products behind SAM's decomposed relative-position bias, for every query of a square grid:
//   rel_h[b, head, (y, x), k] = q[b, (y, x), head, :] . rel_pos_h[y - k + side - 1, :]
//   rel_w[b, head, (y, x), k] = q[b, (y, x), head, :] . rel_pos_w[x - k + side - 1, :]      (k = 0 .. side - 1)
// q is the UNSCALED query of head dim 64, read in place from the packed qkv tensor; the tables are the module's
// parameters themselves ([2 * side - 1, 64]): the [side, side, 64] gather the upstream code builds first
// (get_rel_pos) never exists.
//
// Three kernels, launch_rel_terms() in b200_linear.cu chooses; all add the 64 products of a term in the same order, so the choice
// shows in no bit. In two of them one query token is a 16 x 64 operand (its heads) against `side` rows of either table, two small
// products on the same left operand; mma.sync fits operands of 16 rows that change their table rows from token to token:
// sam_rel_terms_kernel has a warp per token, for small grids, sam_rel_rows_kernel takes a grid row's tokens in turn behind whole
// tables, for many. sam_rel_lines_kernel, for large sides: the tokens of a grid row or column share their table rows and go through
// tensor memory together. All are bound by latency at one image and by the bytes of the result (12.6 MB for SAM's global grid) at several.
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
  uint32_t magic_heads;      // floor(2^32 / heads) + 1
  int tiles;                 // by lines: tiles of 128 rows at a time
  uint32_t* status;
  int early_tables;          // the tables were complete before the kernel in front of this one started: load them without waiting for that one
};

constexpr int kRelWarps = 8, kRelRowWarps = 4;
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
// Table rows are eight 16-byte chunks in shared memory; odd rows have their halves swapped, so that two neighbouring rows, which a
// quarter of a warp reads together, use all banks.

// Sixteen heads of a token from h0 on, chunks t and t + 4 of heads h0 + g (lo) and h0 + g + 8 (hi); rows past the last head repeat
// it and are not stored.
template <typename T>
__device__ __forceinline__ void rel_load_q(const RelTermsParams& p, const T* q_token, int g, int t, int h0, uint4* lo, uint4* hi) {
  const T* q_lo = q_token + min(h0 + g, p.heads - 1) * p.q_sh;
  const T* q_hi = q_token + min(h0 + g + 8, p.heads - 1) * p.q_sh;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    lo[i] = __ldg(reinterpret_cast<const uint4*>(q_lo) + t + 4 * i);
    hi[i] = __ldg(reinterpret_cast<const uint4*>(q_hi) + t + 4 * i);
  }
}

// Both products of those heads of token n, in grid column x, and their stores, MOST tiles at a time. Row k of table_h belongs to column
// k of rel_h, row k of table_w is rel_pos_w[w_first + k].
template <typename T, int NT, int MOST>
__device__ __forceinline__ void rel_token(const RelTermsParams& p, const uint4* lo, const uint4* hi, const uint4* table_h, const uint4* table_w, int w_first, int x, int b, int n, int n_tokens, int side, int g, int t, int h0) {
  uint32_t a[4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    a[2 * i][0] = lo[i].x; a[2 * i][1] = hi[i].x; a[2 * i][2] = lo[i].y; a[2 * i][3] = hi[i].y;
    a[2 * i + 1][0] = lo[i].z; a[2 * i + 1][1] = hi[i].z; a[2 * i + 1][2] = lo[i].w; a[2 * i + 1][3] = hi[i].w;
  }
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    T* const out = static_cast<T*>(which == 0 ? p.rel_h : p.rel_w);
#pragma unroll
    for (int j0 = 0; j0 < NT; j0 += MOST) {
      float acc[MOST][4];
#pragma unroll
      for (int j = 0; j < MOST; ++j) {
        if (j0 + j >= NT) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
        // lane group g holds column 2 NT (g / 2) + 2 (j0 + j) + g % 2 of the result: table row for that k
        const int k = min(2 * NT * (g >> 1) + 2 * (j0 + j) + (g & 1), side - 1);
        const int row = which == 0 ? k : x - w_first - k + side - 1;
        const uint4* table = (which == 0 ? table_h : table_w) + row * 8;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 v = table[(t + 4 * i) ^ ((row & 1) << 2)];
          mma_16816<T>(acc[j], a[2 * i], v.x, v.y);
          mma_16816<T>(acc[j], a[2 * i + 1], v.z, v.w);
        }
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int head = h0 + g + 8 * half;
        if (head >= p.heads) continue;
        T* dst = out + ((static_cast<int64_t>(b) * p.heads + head) * n_tokens + n) * side + 2 * NT * t + 2 * j0;
        uint32_t words[MOST];
#pragma unroll
        for (int j = 0; j < MOST; ++j)
          if (j0 + j < NT) words[j] = rel_pack2<T>(acc[j][2 * half], acc[j][2 * half + 1]);
        if constexpr (NT % 4 == 0) {
          if (side == 8 * NT && p.out_wide) {  // whole 16-byte groups, rows of whole groups
#pragma unroll
            for (int j = 0; j < MOST; j += 4) *reinterpret_cast<uint4*>(dst + 2 * j) = make_uint4(words[j], words[j + 1], words[j + 2], words[j + 3]);
            continue;
          }
        }
#pragma unroll
        for (int j = 0; j < MOST; ++j)
          if (j0 + j < NT && 2 * NT * t + 2 * (j0 + j) < side) *reinterpret_cast<uint32_t*>(dst + 2 * j) = words[j];  // side is even
      }
    }
  }
}

// A token per warp and the rows of the tables that the CTA's tokens need, all in flight together with q.
// Four tiles at a time: registers for four CTAs per SM (and up to 80 bytes of spills).
template <typename T, int NT>
__global__ void __launch_bounds__(kRelWarps * 32, 4) sam_rel_terms_kernel(const RelTermsParams p) {
  extern __shared__ uint4 rel_tables[];
  const int side = p.side, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, n_tokens = side * side;
  const int row_id = blockIdx.x / p.parts, part = blockIdx.x - row_id * p.parts;
  const int b = row_id / side, y = row_id - b * side;
  const int x_begin = side * part / p.parts, x_end = side * (part + 1) / p.parts;  // at most kRelWarps tokens
  uint4* const table_h = rel_tables;              // row k: rel_pos_h[y - k + side - 1]
  uint4* const table_w = rel_tables + side * 8;   // row k: rel_pos_w[x_begin + k]
  const auto load = [&](uint4* to, int k, int c, const void* table, int row) {
    uint4* const spot = to + k * 8 + (c ^ ((k & 1) << 2));
    const uint32_t* src = static_cast<const uint32_t*>(table) + row * 32 + c * 4;
    if (p.tables_wide) cp_async_16(smem_u32(spot), src, true);
    else *spot = make_uint4(__ldg(src), __ldg(src + 1), __ldg(src + 2), __ldg(src + 3));
  };
  const auto load_tables = [&] {
    for (int i = threadIdx.x; i < side * 8; i += kRelWarps * 32) load(table_h, i >> 3, i & 7, p.rel_pos_h, y - (i >> 3) + side - 1);
    const int rows_w = side - 1 + x_end - x_begin;
    for (int i = threadIdx.x; i < rows_w * 8; i += kRelWarps * 32) load(table_w, i >> 3, i & 7, p.rel_pos_w, x_begin + (i >> 3));
    cp_async_commit();
  };
  if (p.early_tables) load_tables();
  grid_dependency_wait();
  grid_launch_dependents();
  if (!p.early_tables) load_tables();
  const int x = x_begin + warp, n = y * side + x;
  const bool here = x < x_end;
  const T* const q_token = static_cast<const T*>(p.q) + b * p.q_sb + (here ? n : 0) * p.q_sn;
  uint4 lo[2], hi[2];
  rel_load_q(p, q_token, g, t, 0, lo, hi);
  cp_async_wait<0>();
  __syncthreads();
  if (!here) return;
  for (int h0 = 0; h0 < p.heads; h0 += 16) {
    if (h0 > 0) rel_load_q(p, q_token, g, t, h0, lo, hi);
    rel_token<T, NT, NT < 4 ? NT : 4>(p, lo, hi, table_h, table_w, x_begin, x, b, n, n_tokens, side, g, t, h0);
  }
}

// The tokens of a grid row, or of a part of it, in turn on four warps: each row of the tables is read once for all of them.
template <typename T, int NT>
__global__ void __launch_bounds__(kRelRowWarps * 32) sam_rel_rows_kernel(const RelTermsParams p) {
  extern __shared__ uint4 rel_tables[];
  const int side = p.side, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, n_tokens = side * side;
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
  for (int i = threadIdx.x; i < side * 8; i += kRelRowWarps * 32) {
    const int k = i >> 3, c = i & 7;
    table_h[k * 8 + (c ^ ((k & 1) << 2))] = load(p.rel_pos_h, y - k + side - 1, c);
  }
  for (int i = threadIdx.x; i < (2 * side - 1) * 8; i += kRelRowWarps * 32) {
    const int k = i >> 3, c = i & 7;
    table_w[k * 8 + (c ^ ((k & 1) << 2))] = load(p.rel_pos_w, k, c);
  }
  __syncthreads();
  const int x_end = side * (part + 1) / p.parts;
  for (int x = side * part / p.parts + warp; x < x_end; x += kRelRowWarps) {
    const int n = y * side + x;
    const T* const q_token = static_cast<const T*>(p.q) + b * p.q_sb + n * p.q_sn;
    for (int h0 = 0; h0 < p.heads; h0 += 16) {
      uint4 lo[2], hi[2];
      rel_load_q(p, q_token, g, t, h0, lo, hi);
      rel_token<T, NT, NT>(p, lo, hi, table_h, table_w, 0, x, b, n, n_tokens, side, g, t, h0);
    }
  }
}

// ---- large grids ------------------------------------------------------------------------------------------------
// The queries of one grid row (rel_h) or column (rel_w), all heads, use the same `side` table rows: a product of side * heads
// rows, `side` columns and 64 values for the tensor memory. A CTA takes such a line: its q rows and table rows come into shared
// memory together (128-byte swizzle), the products are a handful of tcgen05.mma, and a warp writes whole rows of the result (a
// thread per row, 16 bytes of 32 rows per instruction, cost the 64 x 64 grid another 1.8 us).
constexpr int kRelLineThreads = 256, kRelLineTiles = 8;  // at most so many tiles of 128 rows at a time: all of tensor memory at 64 columns
constexpr int rel_lines_smem(int tiles) { return 1024 + 64 * 128 + tiles * 128 * 128; }  // tables, q tiles
enum : uint32_t { kStatusRelTerms = 512 };

template <typename T>
__global__ void __launch_bounds__(kRelLineThreads, 2) sam_rel_lines_kernel(const RelTermsParams p) {
  extern __shared__ uint8_t rel_smem_raw[];
  __shared__ uint64_t done, drain;  // a round's products have finished; abort path: all of this CTA's have
  __shared__ uint32_t tmem_base, abort;
  uint8_t* const table = smem_align_1024(rel_smem_raw);
  const int side = p.side, n_cols = (side + 15) & ~15;
  constexpr int stride_cols = 64;
  uint8_t* const tiles = table + 64 * 128;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int line = blockIdx.x % side, which = (blockIdx.x / side) & 1, b = blockIdx.x / (2 * side);
  const int n_rows = side * p.heads, n_tiles = (n_rows + 127) >> 7;
  const uint32_t tmem_cols = p.tiles >= 5 ? 8 * stride_cols : p.tiles >= 3 ? 4 * stride_cols : 2 * stride_cols;
  if (threadIdx.x == 0) {
    mbar_init(&done, 1);
    mbar_init(&drain, 1);
    abort = 0;
    mbar_init_fence();
  }
  // Chunk c of a 128-byte row, from the halves of two chunks of `src`: a product's 16 values are those the kernel above takes together,
  // the first four of chunks 0 to 3, then their last four, then those of chunks 4 to 7, and the two kernels give the same bits. (By
  // whole chunks, some 4 in 10000 values were the other neighbour.) us, whole chunks -> halves: [1,12,64] 7.65 -> 7.6,
  // [4,12,64] 21.8 -> 22.5, [8,12,64] 40.8 -> 40.9.
  const auto stage = [](uint8_t* to, int row, int c, const void* src, bool valid) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
      cp_async_8(smem_u32(to) + row * 128 + ((c ^ (row & 7)) << 4) + 8 * e, static_cast<const uint2*>(src) + 2 * ((c & 4) + 2 * (c & 1) + e) + ((c >> 1) & 1), valid);
  };
  const auto load_table = [&] {
    const uint4* src = static_cast<const uint4*>(which == 0 ? p.rel_pos_h : p.rel_pos_w);
    for (int i = threadIdx.x; i < n_cols * 8; i += kRelLineThreads) {
      const int k = i >> 3, c = i & 7;
      stage(table, k, c, src + (k < side ? line - k + side - 1 : 0) * 8, k < side);
    }
  };
  // row r of the line: position r / heads, head r % heads
  const auto token_of = [&](int r, int* head) {
    const int i = static_cast<int>(__umulhi(static_cast<uint32_t>(r), p.magic_heads));
    *head = r - i * p.heads;
    return which == 0 ? line * side + i : i * side + line;
  };
  if (p.early_tables) load_table();
  grid_dependency_wait();
  if (!p.early_tables) load_table();
  uint32_t phase = 0;
  for (int t0 = 0; t0 < n_tiles; t0 += p.tiles) {
    const int now = min(n_tiles - t0, p.tiles);
    for (int i = threadIdx.x; i < now * 128 * 8; i += kRelLineThreads) {
      const int row = i >> 3, c = i & 7, r = t0 * 128 + row;
      int head = 0;
      const int n = r < n_rows ? token_of(r, &head) : 0;
      const T* src = static_cast<const T*>(p.q) + b * p.q_sb + n * p.q_sn + head * p.q_sh;
      stage(tiles, row, c, src, r < n_rows);
    }
    cp_async_commit();
    __syncwarp();
    if (t0 == 0 && warp == 1) {  // behind the loads: another CTA of this SM may still hold the columns
      tmem_alloc(&tmem_base, tmem_cols);
      tmem_relinquish();
      // Only now: a kernel behind this one allocates in its set-up and then waits for this grid. Started any earlier, a CTA of it could
      // take columns this one has yet to get, and both would wait for ever.
      grid_launch_dependents();
    }
    cp_async_wait<0>();
    fence_proxy_async_smem();  // the products read what these copies wrote
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = tmem_base;
    if (warp == 1) {
      const uint32_t idesc = umma_idesc_f16(std::is_same<T, __half>::value ? UMMA_F16 : UMMA_BF16, 128, n_cols, 0, 0);
      const uint64_t a = umma_smem_desc_sw128(smem_u32(tiles), 1024, 16), w = umma_smem_desc_sw128(smem_u32(table), 1024, 16);
      if (elect_one()) {
        for (int t = 0; t < now; ++t)
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_ss(tmem + t * stride_cols, a + t * (128 * 128 >> 4) + 2 * kk, w + 2 * kk, idesc, kk > 0 ? 1u : 0u);
        umma_commit(&done);
      }
      __syncwarp();
    }
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&done, phase, &abort)) != 0;
    if (!ok && lane == 0 && atomicExch(&abort, 1u) == 0) atomicOr(p.status, kStatusRelTerms);
    phase ^= 1;
    tc_fence_after_sync();
    T* const out = static_cast<T*>(which == 0 ? p.rel_h : p.rel_w);
    for (int t = warp >> 2; t < now && ok; t += 2) {
      // Through the q tile, which the products have read: a warp then stores four whole rows at a time instead of a piece of 32.
      const uint32_t rows = smem_u32(tiles) + (t * 128 + (warp & 3) * 32) * 128;
      for (int c0 = 0; c0 < side; c0 += 32) {
        float v[32];
        tmem_ld_x32(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + t * stride_cols + c0, reinterpret_cast<uint32_t*>(v));
#pragma unroll
        for (int e = 0; e < 4; ++e)
          st_shared_v4(rows + lane * 128 + (((c0 / 8 + e) ^ (lane & 7)) << 4),
                       make_uint4(rel_pack2<T>(v[8 * e], v[8 * e + 1]), rel_pack2<T>(v[8 * e + 2], v[8 * e + 3]), rel_pack2<T>(v[8 * e + 4], v[8 * e + 5]),
                                  rel_pack2<T>(v[8 * e + 6], v[8 * e + 7])));
      }
      __syncwarp();
      const int chunk = lane & 7;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = 4 * i + (lane >> 3), r = (t0 + t) * 128 + (warp & 3) * 32 + row;
        if (r >= n_rows || 8 * chunk >= side) continue;
        int head = 0;
        const int n = token_of(r, &head);
        reinterpret_cast<uint4*>(out + ((static_cast<int64_t>(b) * p.heads + head) * side * side + n) * side)[chunk] = ld_shared_v4(rows + row * 128 + ((chunk ^ (row & 7)) << 4));
      }
    }
    tc_fence_before_sync();
    __syncthreads();  // tiles and tensor memory have been read
    tc_fence_after_sync();
    if (abort != 0) {  // written in front of that barrier only, so all leave together: the products may still read the tiles
      if (warp == 1) {  // no product may be running when tensor memory is freed
        uint32_t no_abort = 0;
        if (elect_one()) umma_commit(&drain);
        mbar_wait(&drain, 0, &no_abort);
        __syncwarp();
      }
      break;
    }
  }
  if (warp == 1) tmem_dealloc(tmem_base, tmem_cols);
}

}  // namespace b200
