// GEMM with a fused epilogue for the layers around attention, on sm_100a:
//
//   y[p, n] = act((sum_k x[p, k] w[n, k] + bias[n]) * scale[n] + res[p, n])         (bias, scale, res optional)
//
// x [M, K] (row stride lda) and w [N, K] (row-major) are fp16 or bf16, accumulation is fp32 in tensor memory, bias
// and res have the type of x, scale is fp32, y has the type of x and may alias res (the residual of a piece of the
// tile is read before that piece is written, by the same warp, and nobody else touches it). act: 0 none, 1 relu,
// 5 gelu (erf), 6 gelu (tanh form). One more epilogue serves SwiGLU layers: w holds 2 * N rows, the gate's and then
// the value's, and y[p, n] = silu(gate) * value (see kActSwiGlu).
//
// Two kernels; gemm_plan() in b200_linear.cu chooses:
//   * gemm_pair_kernel, for problems that fill the GPU: pairs of CTAs (cta_group::2) compute tiles of 256 rows x BN
//     columns, so that a CTA loads 128 rows of x and only half of the columns of w for a product of M = 256 (no load is
//     multicast). At BN = 256 that is 32 KB from L2 per 2 * 128 * 256 * 64 flops and SM, half of what two separate
//     CTAs with 128 x 256 tiles would pull, and the accumulator takes 256 of the 512 tensor-memory columns: two
//     alternate, and a tile's epilogue runs under the next tile's products.
//   * gemm_split_kernel, for problems with few tiles: one 128 x 64 tile per cluster of S CTAs, each of which takes
//     1 / S of the k range; the partial sums meet through distributed shared memory (no atomics, fixed order).
// Every barrier wait is bounded (sm100_ptx.cuh); a wait that runs out sets the CTA's abort flag and the role bit
// in the status word, and all warps fall through to the common exit.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstddef>
#include <type_traits>

#include "sm100_ptx.cuh"

namespace b200 {

constexpr int kGemmBK = 64;
constexpr int kGemmTileBytes = 128 * kGemmBK * 2;  // 128 rows of 64 k-values, the 128-byte swizzle
enum : uint32_t { kStatusGemmLoader = 64, kStatusGemmMma = 128, kStatusGemmEpilogue = 256 };
enum : int { kActNone = 0, kActRelu = 1, kActGelu = 5, kActGeluTanh = 6, kActSwiGlu = 100 };

struct GemmParams {
  int m, n, k;         // n: columns of y (a SwiGLU layer's w has 2 n rows)
  int bn;              // pair kernel: columns of w per tile, a multiple of 64 up to 256 (always 256 with SwiGLU)
  int tiles_m, tiles_n;
  int group_m;         // pair kernel: row tiles per raster group (item_at)
  int stages;          // pair kernel: ring stages of 16 KB of x and 64 bn bytes of w
  int whole_tiles;     // pair kernel: tiles worked on whole; each of the others is tail_parts items of tail_bn columns
  int tail_parts, tail_bn;
  const void* bias;    // [n] (SwiGLU: [2 n]) or null
  const float* scale;  // [n] or null
  const void* res;     // [m, lres] or null
  int64_t lres;
  void* y;
  int64_t ldy;
  int act;
  int early_w;         // w was complete before the kernel in front of this one started: load it without waiting for that one
  int backwards;       // pair kernel: row tiles from the last to the first
  uint32_t* status;
};

template <typename T>
__device__ __forceinline__ float2 gemm_unpack2(uint32_t v) {
  if constexpr (std::is_same<T, __half>::value) return __half22float2(*reinterpret_cast<const __half2*>(&v));
  else return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ uint32_t gemm_pack2(float lo, float hi) {
  if constexpr (std::is_same<T, __half>::value) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}

// The epilogues work on two values at a time: ffma2 and its like move as many values per clock as the plain forms in half the
// instructions, and two epilogue warps per SM sub-partition are bound by instructions. us, plain -> packed: [4096,3072,768] with erf
// GELU 24.8 -> 23.5, with its tanh form 20.8 -> 19.9, [5480,4096,1024] with that 39.4 -> 38.0.

// v Phi(v) with Phi the normal distribution, as max(v, 0) - |v| Phi(-|v|): no cancellation on the negative side, where
// 0.5 v (1 + erf) loses digits. Phi(-x) = exp(-x^2 / 2) t P(t), t = 1 / (1 + 0.3 x), where P is a degree-7 least-maximum
// fit of 0.5 erfcx(x / sqrt 2) / t on 0 <= x <= 13.5 (relative error 1.3e-7; the whole within 2e-6 of v Phi(v) down to
// v = -5, where erff gave 1e-3). Two MUFU operations and a dozen multiply-adds: a third of the time of erff, which took
// longer than the products of a 256 x 256 tile at k = 768. max(v, 0) is written v / 2 + |v| / 2, which keeps NaN and gives
// it for -inf as v Phi(v) does; the tail's argument ends where the tail is zero, so that +inf meets no inf * 0.
__device__ __forceinline__ float2 gelu_erf2(float2 v) {
  const auto both = [](float c) { return make_float2(c, c); };
  const float2 a = make_float2(fabsf(v.x), fabsf(v.y)), x = make_float2(fminf(a.x, 64.f), fminf(a.y, 64.f));
  const float2 s = ffma2(x, both(0.3f), both(1.f)), g = fmul2(fmul2(x, x), both(-0.72134752f));
  float2 t, e;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t.x) : "f"(s.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t.y) : "f"(s.y));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(g.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(g.y));
  float2 p = both(0.0359317549f);
  p = ffma2(p, t, both(-0.158276081f));
  p = ffma2(p, t, both(0.208206728f));
  p = ffma2(p, t, both(-0.0553939454f));
  p = ffma2(p, t, both(0.129469246f));
  p = ffma2(p, t, both(0.0996374786f));
  p = ffma2(p, t, both(0.120798357f));
  p = ffma2(p, t, both(0.119626388f));
  const float2 tail = fmul2(make_float2(-x.x, -x.y), fmul2(t, p));
  return ffma2(tail, e, ffma2(both(0.5f), v, fmul2(both(0.5f), a)));
}

template <int ACT>
__device__ __forceinline__ float2 gemm_act2(float2 v) {
  if constexpr (ACT == kActRelu) return make_float2(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f));
  if constexpr (ACT == kActGelu) return gelu_erf2(v);
  if constexpr (ACT == kActGeluTanh) {
    const auto both = [](float c) { return make_float2(c, c); };
    const float2 u = fmul2(fmul2(both(0.7978845608028654f), v), ffma2(fmul2(both(0.044715f), v), v, both(1.f)));
    float2 t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.x) : "f"(u.x));
    asm("tanh.approx.f32 %0, %1;" : "=f"(t.y) : "f"(u.y));
    return fmul2(fmul2(both(0.5f), v), fadd2(both(1.f), t));
  }
  return v;
}
// silu(g) * u = g u / (1 + exp(-g))
__device__ __forceinline__ float gemm_swiglu(float g, float u) { return __fdividef(g, 1.f + __expf(-g)) * u; }

// Runs f(integral_constant<int, ACT>) for the launch's activation: one decision per chunk, not one per value.
template <typename F>
__device__ __forceinline__ void for_act(int act, F&& f) {
  if (act == kActGeluTanh) f(std::integral_constant<int, kActGeluTanh>{});
  else if (act == kActGelu) f(std::integral_constant<int, kActGelu>{});
  else if (act == kActRelu) f(std::integral_constant<int, kActRelu>{});
  else f(std::integral_constant<int, kActNone>{});
}

// ---- pair kernel ----------------------------------------------------------------------------------------------
constexpr int kPairThreads = 320;  // warp 0 loader, warp 1 MMA, warps 2..9 epilogue
constexpr int kPairRingBytes = 160 * 1024, kPairMaxStages = 8;
constexpr int kPairChunkBytes = 32 * 64 * 2;  // what an epilogue warp stages at a time: its 32 rows, 64 columns

struct PairSmem {
  alignas(1024) uint8_t ring[kPairRingBytes];          // per stage: 128 rows of x, then bn / 2 rows of w
  alignas(1024) uint8_t stage[8][2][kPairChunkBytes];  // per epilogue warp, two deep: residual in, result out
  uint64_t full[kPairMaxStages];   // the leader's: both CTAs' tiles of the stage have landed     (TMA of both CTAs)
  uint64_t empty[kPairMaxStages];  // the stage has been read by its products                     (MMA commit, both CTAs)
  uint64_t acc_full[2];         // accumulator finished                                        (MMA commit, both CTAs)
  uint64_t acc_empty[2];        // the leader's: read by the epilogue warps of both CTAs       (16 warps)
  uint64_t res_full[8][2];      // per epilogue warp: the residual of a piece has landed       (TMA)
  uint64_t drain;               // abort path: the leader's products have finished             (MMA commit, both CTAs)
  uint32_t tmem_base;
  uint32_t abort;
};
constexpr int kPairBarriers = 2 * kPairMaxStages + 2 + 2 + 16 + 1;
static_assert(offsetof(PairSmem, drain) == offsetof(PairSmem, full) + (kPairBarriers - 1) * sizeof(uint64_t), "the set-up walks the barriers as one array");
static_assert(sizeof(PairSmem) + 1024 <= 227 * 1024, "shared memory of one CTA");

struct GemmItem {
  int tm;    // row tile
  int col0;  // first column of y
  int bn;    // columns of w: p.bn, or p.tail_bn for a part of a tile
};
// Items are the tiles in groups of `group_m` row tiles, row tiles fastest inside a group: the pairs that run at the same
// time then share both w tiles and x tiles, and what they read together stays in L2. The tiles behind the last whole
// round of the grid come in parts where gemm_plan() in b200_linear.cu says so, parts of a tile one after another.
__device__ __forceinline__ GemmItem item_at(const GemmParams& p, int item, int out_cols) {
  GemmItem t;
  int tile = item, sub = 0;
  t.bn = p.bn;
  if (item >= p.whole_tiles) {
    const int i = item - p.whole_tiles, behind = i / p.tail_parts;
    tile = p.whole_tiles + behind;
    sub = (i - behind * p.tail_parts) * p.tail_bn;
    t.bn = p.tail_bn;
  }
  const int per_group = p.group_m * p.tiles_n;
  const int g = tile / per_group;
  const int in = tile - g * per_group;
  const int rows = min(p.group_m, p.tiles_m - g * p.group_m);
  const int tn = in / rows;
  t.tm = g * p.group_m + (in - tn * rows);
  if (p.backwards) t.tm = p.tiles_m - 1 - t.tm;
  t.col0 = tn * out_cols + sub;
  return t;
}

// Bounded by the L2 -> SM operand traffic and, above about 1.4 PFLOP/s sustained, the power cap. ACT and FORM are template
// parameters: decided at run time, the branches alone cost 400 clocks per piece.
// A residual without a scale (ViT-B, SAM) has a form of its own: two shuffles less per pair of columns, [4096,768,768] 9.3 -> 9.0 us,
// [4096,768,3072] 20.8 -> 20.3. Sixteen epilogue warps with a piece each instead of eight with two: [4096,3072,768] 16.6 -> 17.5.
enum : int { kPairPlain = 0, kPairResidual = 1, kPairScaled = 2 };  // ... ; a residual; a scale, and a residual or none
template <typename T, int ACT, int FORM>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                 const __grid_constant__ CUtensorMap tm_w_tail, const __grid_constant__ CUtensorMap tm_y,
                 const __grid_constant__ CUtensorMap tm_res, const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  PairSmem& sm = *reinterpret_cast<PairSmem*>(smem_align_1024(smem_raw));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_cta_rank());  // 0: the leader, rows 0..127 of the tile
  constexpr bool swiglu = ACT == kActSwiGlu, FULL = FORM != kPairPlain;

  // Set-up. The loader goes on as soon as both CTAs' barriers exist, the other warps once tensor memory has been allocated too.
  // Neither this hand-over, nor that of an accumulator, nor the one at the end passes data through memory: relaxed, without the
  // wait for a thread's own traffic that a release brings, they take some 100 clocks instead of 1000. us of a launch, before and
  // with both: [4096,768,768] 9.2 and 8.0, [4096,2304,768] 13.9 and 12.6, [4096,3072,768] with erf GELU 22.4 and 19.6,
  // [1370,1536,384] 7.3 and 5.9.
  if (warp == 0) {
    uint64_t* const first = &sm.full[0];  // the barriers lie one after another
    for (int i = lane; i < kPairBarriers; i += 32) mbar_init(first + i, first + i == &sm.acc_empty[0] || first + i == &sm.acc_empty[1] ? 16 : 1);
    if (lane == 0) sm.abort = 0;
    mbar_init_fence();
    __syncwarp();
  }
  cluster_arrive_relaxed();
  if (warp == 0) {
    named_barrier_arrive(1, kPairThreads);
    if (lane == 0) {
      tma_prefetch_desc(&tm_x);
      tma_prefetch_desc(&tm_w);
      tma_prefetch_desc(&tm_y);
      if (FULL && p.res != nullptr) tma_prefetch_desc(&tm_res);
    }
    __syncwarp();
  } else {
    if (warp == 1) {
      tmem_alloc_pair(&sm.tmem_base, 512);
      tmem_relinquish_pair();
    }
    tc_fence_before_sync();
    named_barrier_sync(1, kPairThreads);
    tc_fence_after_sync();
  }
  cluster_wait();  // the other CTA's barriers exist before anything of this one reaches for them
  const uint32_t tmem = sm.tmem_base;  // (not the loader's)
  volatile uint32_t* abort_flag = &sm.abort;
  const int items = p.whole_tiles + (p.tiles_m * p.tiles_n - p.whole_tiles) * p.tail_parts;
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const int k_blocks = (p.k + kGemmBK - 1) / kGemmBK;
  const int stages = p.stages;
  const uint32_t stage_size = kGemmTileBytes + static_cast<uint32_t>(p.bn) * kGemmBK;  // of one CTA: 128 rows of x, bn / 2 of w
  const int out_cols = swiglu ? 128 : p.bn;  // columns of y per tile

  if (warp == 0) {
    // ======================= loader (the whole warp, one lane issues: see elect_one) ==================
    bool ok = true;
    int g = 0, st = 0;  // stage uses so far, ring position
    uint32_t ph = 1;    // parity of the empty barriers: a ring that was never used is empty
    // Both CTAs count their bytes on the leader's barrier.
    auto load_x = [&](int s, const GemmItem& t, int kb) {
      tma_load_2d_pair(sm.ring + s * stage_size, &tm_x, cluster_map(smem_u32(&sm.full[s]), 0), kb * kGemmBK, t.tm * 256 + rank * 128);
    };
    auto load_w = [&](int s, const GemmItem& t, int kb) {
      // SwiGLU: the leader's half are 128 gate columns, the other CTA's the value columns that belong to them
      const int row = swiglu ? t.col0 + rank * p.n : t.col0 + rank * (t.bn >> 1);
      tma_load_2d_pair(sm.ring + s * stage_size + kGemmTileBytes, t.bn == p.bn ? &tm_w : &tm_w_tail, cluster_map(smem_u32(&sm.full[s]), 0), kb * kGemmBK, row);
    };
    auto expect = [&](int s, const GemmItem& t) {
      if (rank == 0) mbar_arrive_expect_tx(&sm.full[s], 2u * (kGemmTileBytes + static_cast<uint32_t>(t.bn) * kGemmBK));
    };
    int early = 0;  // stages whose w tile is on its way before the wait for the kernel in front
    if (p.early_w && first_tile < items) {
      const GemmItem t = item_at(p, first_tile, out_cols);
      for (; early < stages && early < k_blocks; ++early) {
        if (elect_one()) {
          expect(early, t);
          load_w(early, t, early);
        }
      }
    }
    grid_dependency_wait();
    for (int tile = first_tile; tile < items && ok; tile += tile_step) {
      const GemmItem t = item_at(p, tile, out_cols);
      for (int kb = 0; kb < k_blocks; ++kb, ++g) {
        if (g < early) {
          if (elect_one()) load_x(st, t, kb);
        } else {
          ok = __all_sync(0xffffffffu, mbar_wait(&sm.empty[st], ph, abort_flag));
          if (!ok) break;
          if (elect_one()) {
            expect(st, t);
            load_x(st, t, kb);
            load_w(st, t, kb);
          }
        }
        if (++st == stages) {
          st = 0;
          ph ^= 1;
        }
      }
    }
    if (!ok && lane == 0 && atomicExch(const_cast<uint32_t*>(abort_flag), 1u) == 0) atomicOr(p.status, kStatusGemmLoader);
    if (__any_sync(0xffffffffu, *abort_flag != 0) && rank == 0) {  // let every copy that was issued land (both CTAs count on the leader's barriers)
      uint32_t no_abort = 0;
      for (int j = (g > stages ? g - stages : 0); j < g; ++j) mbar_wait(&sm.full[j % stages], (j / stages) & 1, &no_abort);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ======================= MMA issuer (leader only) =================================================
    // The next kernel may start from here on: this warp's CTA holds its tensor memory, which the loader does not wait for.
    grid_dependency_wait();
    grid_launch_dependents();
    if (rank == 0) {
      constexpr uint32_t fmt = std::is_same<T, __half>::value ? UMMA_F16 : UMMA_BF16;
      const uint32_t idesc_whole = umma_idesc_f16(fmt, 256, p.bn, 0, 0), idesc_tail = umma_idesc_f16(fmt, 256, p.tail_bn, 0, 0);
      const uint64_t a_desc0 = umma_smem_desc_sw128(smem_u32(sm.ring), 1024, 16);
      const uint64_t b_desc0 = umma_smem_desc_sw128(smem_u32(sm.ring) + kGemmTileBytes, 1024, 16);
      bool ok = true;
      int st = 0, it = 0;
      uint32_t ph = 0;
      bool landed = false;  // this stage's barrier, tested while the stage before was being issued (a test takes some 100 clocks)
      for (int tile = first_tile; tile < items && ok; tile += tile_step, ++it) {
        if (it >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&sm.acc_empty[it & 1], ((it >> 1) - 1) & 1, abort_flag));
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t acc = tmem + (it & 1) * 256;
        const uint32_t idesc = tile < p.whole_tiles ? idesc_whole : idesc_tail;
        for (int kb = 0; kb < k_blocks; ++kb) {
          ok = __all_sync(0xffffffffu, landed || mbar_wait(&sm.full[st], ph, abort_flag));
          if (!ok) break;
          tc_fence_after_sync();
          const int next = st + 1 == stages ? 0 : st + 1;
          const uint32_t next_ph = st + 1 == stages ? ph ^ 1 : ph;
          landed = mbar_test_wait(&sm.full[next], next_ph);
          const uint64_t a = a_desc0 + static_cast<uint64_t>(st) * (stage_size >> 4);
          const uint64_t b = b_desc0 + static_cast<uint64_t>(st) * (stage_size >> 4);
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < kGemmBK / 16; ++kk) umma_ss_pair(acc, a + 2 * kk, b + 2 * kk, idesc, (kb | kk) != 0 ? 1u : 0u);
            umma_commit_pair(&sm.empty[st]);
            if (kb == k_blocks - 1) umma_commit_pair(&sm.acc_full[it & 1]);
          }
          st = next;
          ph = next_ph;
        }
      }
      // The other CTA's epilogue warps signal `acc_empty` here, a lane per barrier: those of the last two items are waited for by nobody else,
      // and they have landed before this CTA goes. (In a warp that has nothing else to do any more: no launch took longer.)
      if (ok) ok = __all_sync(0xffffffffu, lane >= min(it, 2) || mbar_wait(&sm.acc_empty[lane], ((it - 1 - lane) / 2) & 1, abort_flag));
      if (!ok && lane == 0 && atomicExch(const_cast<uint32_t*>(abort_flag), 1u) == 0) atomicOr(p.status, kStatusGemmMma);
      if (__any_sync(0xffffffffu, *abort_flag != 0)) {  // no product may be running when tensor memory is freed
        uint32_t no_abort = 0;
        if (elect_one()) umma_commit_pair(&sm.drain);
        mbar_wait(&sm.drain, 0, &no_abort);
      }
    }
    __syncwarp();
  } else {
    // ======================= epilogue warps ==========================================================
    // A warp owns 32 rows (its quarter of the tensor-memory lanes) and every second 64-column piece of the tile. A
    // piece goes: accumulator -> registers -> epilogue -> the warp's staging area (128-byte swizzle) -> TMA store, which
    // clips rows and columns past the end; a residual comes the same way in. No other warp is waited for.
    grid_dependency_wait();
    const int e = warp - 2, part = e >> 2, quarter = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t acc_empty_at[2] = {cluster_map(smem_u32(&sm.acc_empty[0]), 0), cluster_map(smem_u32(&sm.acc_empty[1]), 0)};
    const bool has_res = FULL && p.res != nullptr;
    const uint32_t stage_row = smem_u32(sm.stage[e][0]) + lane * 128;
    auto row_of = [&](const GemmItem& t) { return t.tm * 256 + rank * 128 + quarter * 32; };
    auto inside = [&](int row, int col) { return row < p.m && col < p.n; };
    bool ok = true;
    int it = 0;
    uint32_t loads[2] = {0, 0};  // residual loads into either buffer so far (phases of res_full)
    for (int tile = first_tile; tile < items && ok; tile += tile_step, ++it) {
      const GemmItem t = item_at(p, tile, out_cols);
      const int row0 = row_of(t), col0 = t.col0;
      const int pieces = swiglu ? 2 : t.bn / 64;
      // What the epilogue needs besides the accumulator is asked for before the wait for it: the residual of this warp's
      // two pieces, one per buffer, and bias and scale.
      // The first tile's residual stands back (for a while) until the ring's first loads are in, which it held up. With this and the
      // waits below where they are: [4096,768,768] 8.0 -> 7.7, [4096,768,3072] 16.5 -> 16.0.
      if (it == 0 && has_res)
        for (int polls = 0; polls < 32 && !mbar_test_wait(&sm.empty[0], 0); ++polls) {}
      if (has_res && lane == 0) {
        tma_store_wait_read<0>();  // the stores of the tile before have read both buffers
        for (int i = 0; i < 2; ++i) {
          const int c = part + 2 * i;
          if (c < pieces && inside(row0, col0 + c * 64)) {  // asked(i) below
            mbar_arrive_expect_tx(&sm.res_full[e][i], kPairChunkBytes);
            tma_load_2d(sm.stage[e][i], &tm_res, &sm.res_full[e][i], col0 + c * 64, row0);
          }
        }
      }
      // Lane l holds bias and scale of columns 2 l and 2 l + 1 of either piece; the lanes pass them round with shuffles.
      // (Loads at one address for the whole warp, where a value is needed, took half of the epilogue's time.)
      uint32_t bias2[2] = {0, 0}, bias_up = 0;
      float2 scale2[2] = {make_float2(1.f, 1.f), make_float2(1.f, 1.f)};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int c = col0 + (part + 2 * i) * 64 + 2 * lane;
        if (part + 2 * i < pieces && c < p.n) {
          if (p.bias != nullptr) bias2[i] = __ldg(reinterpret_cast<const uint32_t*>(static_cast<const T*>(p.bias) + c));
          if (swiglu && p.bias != nullptr) bias_up = __ldg(reinterpret_cast<const uint32_t*>(static_cast<const T*>(p.bias) + p.n + c));
          if (p.scale != nullptr) scale2[i] = __ldg(reinterpret_cast<const float2*>(p.scale + c));
        }
      }
      // The residual has landed long before the accumulator is finished: its waits cost nothing here, some 350 clocks each behind that.
      if (has_res) {
        auto asked = [&](int i) { return part + 2 * i < pieces && inside(row0, col0 + (part + 2 * i) * 64); };
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (asked(i)) ok = ok && __all_sync(0xffffffffu, mbar_wait(&sm.res_full[e][i], loads[i] & 1, abort_flag)) != 0;
        if (!ok) {  // given up: a residual still on its way must land before the CTA goes
          uint32_t no_abort = 0;
          for (int i = 0; i < 2; ++i)
            if (asked(i)) mbar_wait(&sm.res_full[e][i], loads[i] & 1, &no_abort);
          break;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) loads[i] += asked(i) ? 1 : 0;
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&sm.acc_full[it & 1], (it >> 1) & 1, abort_flag))) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const uint32_t acc = tmem + lane_addr + (it & 1) * 256;
      if (part >= pieces) {
        if (lane == 0) mbar_arrive_cluster(acc_empty_at[it & 1]);
        continue;
      }
#pragma unroll 1
      for (int c = part; c < pieces; c += 2) {
        const int buf = c >> 1;
        const int col = col0 + c * 64;
        const bool here = inside(row0, col);
        if (!has_res && lane == 0) {  // the store that used this buffer last has read it
          if (part + 2 < pieces) tma_store_wait_read<1>();
          else tma_store_wait_read<0>();
        }
        __syncwarp();
        if (here) {
          const uint32_t at = stage_row + buf * kPairChunkBytes;
          const uint32_t piece_bias = buf == 0 ? bias2[0] : bias2[1];
          const float2 piece_scale = buf == 0 ? scale2[0] : scale2[1];
          // one lane's row: eight 16-byte groups of eight columns at the positions of the 128-byte swizzle, in two halves
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            [[maybe_unused]] uint4 r4[FULL ? 4 : 1];
            if constexpr (FULL) {
#pragma unroll
              for (int q = 0; q < 4; ++q) r4[q] = has_res ? ld_shared_v4(at + (((4 * half + q) ^ (lane & 7)) << 4)) : make_uint4(0, 0, 0, 0);
            }
            float v[32];
            [[maybe_unused]] float u[swiglu ? 32 : 1];
            tmem_ld_x32(acc + c * 64 + half * 32, reinterpret_cast<uint32_t*>(v));
            if constexpr (swiglu) tmem_ld_x32(acc + 128 + c * 64 + half * 32, reinterpret_cast<uint32_t*>(u));
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float x[8];
              const uint32_t spot = at + (((4 * half + q) ^ (lane & 7)) << 4);
              [[maybe_unused]] uint32_t rw[4] = {0, 0, 0, 0};
              if constexpr (FULL) { rw[0] = r4[q].x; rw[1] = r4[q].y; rw[2] = r4[q].z; rw[3] = r4[q].w; }
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int pair = 16 * half + 4 * q + i, at_v = 8 * q + 2 * i;
                const float2 b = gemm_unpack2<T>(__shfl_sync(0xffffffffu, piece_bias, pair));
                if constexpr (swiglu) {
                  const float2 bu = gemm_unpack2<T>(__shfl_sync(0xffffffffu, bias_up, pair));
                  x[2 * i] = gemm_swiglu(v[at_v] + b.x, u[at_v] + bu.x);
                  x[2 * i + 1] = gemm_swiglu(v[at_v + 1] + b.y, u[at_v + 1] + bu.y);
                } else {
                  float2 y = fadd2(make_float2(v[at_v], v[at_v + 1]), b);
                  if constexpr (FORM == kPairResidual) y = fadd2(y, gemm_unpack2<T>(rw[i]));
                  if constexpr (FORM == kPairScaled)
                    y = ffma2(y, make_float2(__shfl_sync(0xffffffffu, piece_scale.x, pair), __shfl_sync(0xffffffffu, piece_scale.y, pair)), gemm_unpack2<T>(rw[i]));
                  y = gemm_act2<ACT>(y);
                  x[2 * i] = y.x;
                  x[2 * i + 1] = y.y;
                }
              }
              st_shared_v4(spot, make_uint4(gemm_pack2<T>(x[0], x[1]), gemm_pack2<T>(x[2], x[3]), gemm_pack2<T>(x[4], x[5]), gemm_pack2<T>(x[6], x[7])));
            }
          }
          fence_proxy_async_smem();
        }
        if (c + 2 >= pieces) tc_fence_before_sync();  // this warp has read all it needs of the accumulator
        __syncwarp();
        if (c + 2 >= pieces && lane == 0) mbar_arrive_cluster(acc_empty_at[it & 1]);
        if (lane == 0) {
          if (here) tma_store_2d(&tm_y, sm.stage[e][buf], col, row0);
          tma_store_commit();
        }
      }
    }
    if (!ok && lane == 0 && atomicExch(const_cast<uint32_t*>(abort_flag), 1u) == 0) atomicOr(p.status, kStatusGemmEpilogue);
    if (lane == 0) tma_store_wait_read<0>();
    __syncwarp();
  }

  tc_fence_before_sync();
  __syncthreads();
  // Neither CTA goes while the other may still multiply into its tensor memory or signal its barriers. The barrier itself, relaxed, orders no such
  // signal: the leader has waited for those of the accumulators, and the last ones of the stages go out in front of the accumulator's,
  // which every epilogue warp has waited for.
  cluster_arrive_relaxed();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem, 512);
  }
}

// ---- split kernel ---------------------------------------------------------------------------------------------
constexpr int kSplitEpilogueThreads = 256;
constexpr int kSplitThreads = 64 + kSplitEpilogueThreads;  // warp 0 loader, warp 1 MMA, warps 2..9 epilogue
// A round trip to L2 covers some four stages; with six a CTA left no room on its SM for one of the kernels in front or behind.
constexpr int kSplitStages = 4;
constexpr int kSplitBN = 64;

template <int S>
struct SplitSmem {
  static constexpr int kRows = (128 + S - 1) / S;  // rows of the tile each CTA of the cluster finishes (the last one what is left)
  static constexpr int kStride = kRows | 1;        // in float4: odd, so that rows and columns are both read without conflicts
  alignas(1024) uint8_t a[kSplitStages][kGemmTileBytes];
  alignas(1024) uint8_t b[kSplitStages][kSplitBN * kGemmBK * 2];
  float4 recv[S][kSplitBN / 4][kStride];     // [from CTA][four columns][row]: partial sums of this CTA's rows
  uint64_t full[kSplitStages], empty[kSplitStages];
  uint64_t acc_full;
  uint32_t tmem_base;
  uint32_t abort;
};

// Latency-bound: a few tiles of a small problem. The k range is cut over the S CTAs of a cluster so that more SMs pull
// operands; every CTA sends each of its 128 rows' partial sums to the CTA that finishes that row, and adds the S parts
// of its own rows in rank order.
template <typename T, int S>
__global__ void __launch_bounds__(kSplitThreads)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, const GemmParams p) {
  using Smem = SplitSmem<S>;
  extern __shared__ uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_align_1024(smem_raw));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = S > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  const int tile = blockIdx.x / S;
  const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
  const int k_blocks = (p.k + kGemmBK - 1) / kGemmBK;
  const int kb0 = k_blocks * rank / S, kb1 = k_blocks * (rank + 1) / S;  // at least one each (gemm_plan)

  if (threadIdx.x == 0) {
    for (int i = 0; i < kSplitStages; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], 1);
    }
    mbar_init(&sm.acc_full, 1);
    sm.abort = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 64);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_w);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if constexpr (S > 1) cluster_arrive_relaxed();  // this CTA runs; waited for before anybody writes into its receive area
  const uint32_t tmem = sm.tmem_base;
  volatile uint32_t* abort_flag = &sm.abort;

  if (warp == 0) {
    bool ok = true;
    constexpr uint32_t kBytes = kGemmTileBytes + kSplitBN * kGemmBK * 2;
    int early = 0;
    if (p.early_w) {
      for (; early < kSplitStages && kb0 + early < kb1; ++early) {
        if (elect_one()) {
          mbar_arrive_expect_tx(&sm.full[early], kBytes);
          tma_load_2d(sm.b[early], &tm_w, &sm.full[early], (kb0 + early) * kGemmBK, tn * kSplitBN);
        }
      }
    }
    grid_dependency_wait();
    grid_launch_dependents();
    int g = 0, st = 0;
    uint32_t ph = 1;
    for (int kb = kb0; kb < kb1; ++kb, ++g) {
      if (g < early) {
        if (elect_one()) tma_load_2d(sm.a[st], &tm_x, &sm.full[st], kb * kGemmBK, tm * 128);
      } else {
        // the first round of the ring needs no wait: nothing has been in it
        ok = __all_sync(0xffffffffu, g < kSplitStages || mbar_wait(&sm.empty[st], ph, abort_flag));
        if (!ok) break;
        if (elect_one()) {
          mbar_arrive_expect_tx(&sm.full[st], kBytes);
          tma_load_2d(sm.b[st], &tm_w, &sm.full[st], kb * kGemmBK, tn * kSplitBN);
          tma_load_2d(sm.a[st], &tm_x, &sm.full[st], kb * kGemmBK, tm * 128);
        }
      }
      if (++st == kSplitStages) {
        st = 0;
        ph ^= 1;
      }
    }
    if (!ok && lane == 0 && atomicExch(const_cast<uint32_t*>(abort_flag), 1u) == 0) atomicOr(p.status, kStatusGemmLoader);
    if (__any_sync(0xffffffffu, *abort_flag != 0)) {
      uint32_t no_abort = 0;
      for (int j = (g > kSplitStages ? g - kSplitStages : 0); j < g; ++j) mbar_wait(&sm.full[j % kSplitStages], (j / kSplitStages) & 1, &no_abort);
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t fmt = std::is_same<T, __half>::value ? UMMA_F16 : UMMA_BF16;
    constexpr uint32_t idesc = umma_idesc_f16(fmt, 128, kSplitBN, 0, 0);
    const uint64_t a_desc0 = umma_smem_desc_sw128(smem_u32(sm.a[0]), 1024, 16);
    const uint64_t b_desc0 = umma_smem_desc_sw128(smem_u32(sm.b[0]), 1024, 16);
    bool ok = true, landed = false;
    int st = 0;
    uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      ok = __all_sync(0xffffffffu, landed || mbar_wait(&sm.full[st], ph, abort_flag));
      if (!ok) break;
      tc_fence_after_sync();
      const int next = st + 1 == kSplitStages ? 0 : st + 1;
      const uint32_t next_ph = st + 1 == kSplitStages ? ph ^ 1 : ph;
      landed = mbar_test_wait(&sm.full[next], next_ph);
      const uint64_t a = a_desc0 + static_cast<uint64_t>(st) * (kGemmTileBytes >> 4);
      const uint64_t b = b_desc0 + static_cast<uint64_t>(st) * ((kSplitBN * kGemmBK * 2) >> 4);
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < kGemmBK / 16; ++kk) umma_ss(tmem, a + 2 * kk, b + 2 * kk, idesc, (kb != kb0 || kk != 0) ? 1u : 0u);
        umma_commit(&sm.empty[st]);
      }
      st = next;
      ph = next_ph;
    }
    if (!ok && lane == 0 && atomicExch(const_cast<uint32_t*>(abort_flag), 1u) == 0) atomicOr(p.status, kStatusGemmMma);
    __syncwarp();
    if (elect_one()) umma_commit(&sm.acc_full);  // also on the abort path: the epilogue's wait then ends when the products in flight have
    __syncwarp();
  }

  // Epilogue thread: four columns (the same for all its items) of every sixteenth row. What the epilogue needs besides the
  // sums is in flight while the products run.
  constexpr int kItems = (Smem::kRows * (kSplitBN / 4) + kSplitEpilogueThreads - 1) / kSplitEpilogueThreads, kRowStep = kSplitEpilogueThreads / 16;
  const int et = threadIdx.x - 64, c4 = et & 15;
  const int first_row = rank * Smem::kRows, end_row = min(min(first_row + Smem::kRows, 128), p.m - tm * 128);  // in the tile
  const int row0 = tm * 128 + first_row + (et >> 4), row_end = tm * 128 + end_row, col = tn * kSplitBN + c4 * 4;
  const bool col_in = col < p.n;
  uint2 bias = make_uint2(0, 0), res[kItems];
  float4 scale = make_float4(1.f, 1.f, 1.f, 1.f);
  if (warp >= 2) {
    grid_dependency_wait();
    if (p.bias != nullptr && col_in) bias = __ldg(reinterpret_cast<const uint2*>(static_cast<const T*>(p.bias) + col));
    if (p.scale != nullptr && col_in) scale = __ldg(reinterpret_cast<const float4*>(p.scale + col));
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      res[i] = make_uint2(0, 0);
      if (p.res != nullptr && col_in && row0 + kRowStep * i < row_end)
        res[i] = *reinterpret_cast<const uint2*>(static_cast<const T*>(p.res) + static_cast<int64_t>(row0 + kRowStep * i) * p.lres + col);
    }
    if (!__all_sync(0xffffffffu, mbar_wait(&sm.acc_full, 0, abort_flag)) && lane == 0 &&
        atomicExch(const_cast<uint32_t*>(abort_flag), 1u) == 0)
      atomicOr(p.status, kStatusGemmEpilogue);
    tc_fence_after_sync();
  }
  if constexpr (S > 1) cluster_wait();
  if (warp >= 2) {
    const int row = (warp & 3) * 32 + lane, half = (warp - 2) >> 2;  // this thread's row of the tile, its 32 columns
    float v[kSplitBN / 2];
    tmem_ld_x32(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + half * (kSplitBN / 2), reinterpret_cast<uint32_t*>(v));
    uint32_t dst = smem_u32(&sm.recv[rank][half * (kSplitBN / 8)][row % Smem::kRows]);
    if constexpr (S > 1) dst = cluster_map(dst, row / Smem::kRows);
#pragma unroll
    for (int c4 = 0; c4 < kSplitBN / 8; ++c4)
      st_cluster_v4(dst + c4 * (Smem::kStride * 16), make_float4(v[4 * c4], v[4 * c4 + 1], v[4 * c4 + 2], v[4 * c4 + 3]));
  }
  tc_fence_before_sync();
  if constexpr (S > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (warp >= 2) {
    const float2 b0 = gemm_unpack2<T>(bias.x), b1 = gemm_unpack2<T>(bias.y);
    for_act(p.act, [&](auto act_tag) {
      constexpr int kAct = decltype(act_tag)::value;
#pragma unroll
      for (int i = 0; i < kItems; ++i) {
        const int r = min((et >> 4) + kRowStep * i, Smem::kRows - 1);  // past the last row: read what is there, write nothing
        float4 x = sm.recv[0][c4][r];
#pragma unroll
        for (int s = 1; s < S; ++s) {
          const float4 o = sm.recv[s][c4][r];
          x.x += o.x; x.y += o.y; x.z += o.z; x.w += o.w;
        }
        const float2 r0 = gemm_unpack2<T>(res[i].x), r1 = gemm_unpack2<T>(res[i].y);
        const float2 y0 = gemm_act2<kAct>(ffma2(fadd2(make_float2(x.x, x.y), b0), make_float2(scale.x, scale.y), r0));
        const float2 y1 = gemm_act2<kAct>(ffma2(fadd2(make_float2(x.z, x.w), b1), make_float2(scale.z, scale.w), r1));
        if (col_in && row0 + kRowStep * i < row_end)
          *reinterpret_cast<uint2*>(static_cast<T*>(p.y) + static_cast<int64_t>(row0 + kRowStep * i) * p.ldy + col) =
              make_uint2(gemm_pack2<T>(y0.x, y0.y), gemm_pack2<T>(y1.x, y1.y));
      }
    });
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 64);
  }
}

}  // namespace b200
