// Rule and launch of the attention kernel for few keys (attn_window_sm100.cuh).
#include <algorithm>

#include "attn_window_sm100.cuh"
#include "window_host.h"

namespace b200 {
namespace {

// Blocks of 64 queries per SM, in tenths, up to which this kernel is the faster one (0: any number of them). All us in CUDA graphs, persistent
// kernel and this one, [images, heads, queries] on keys.
//
// A head of up to 64 queries leaves half of a 128-row query tile empty: this kernel up to 64 keys at every size that was tried (3 to 12288
// heads: 0.2 to 0.55 of the time). Many queries fill the tiles; the persistent kernel then takes two of them in the same time whatever the
// key count, while this one's work for a block grows with it and loads K and V once per block:
//   [8,16,4096] on 32 keys 36.0 and 30.7, on 49 35.8 and 40.1, on 64 35.1 and 42.1; with a dense bias 51.4 and 33.2, 51.5 and 49.4, 48.5 and 56.2;
//   with tables 71 and 43, 78 and 57, 65 and 55. The lines lie where the two meet: without a bias [12,12,4096] on 36 keys 39.7 and 40.1 (62 blocks
//   per SM), [6,12,4096] on 49 21.9 and 21.5 (31), on 57 22.1 and 22.7, [4,12,4096] on 64 15.7 and 15.4 (21), with a bias 20.9 and 21.3.
// An odd number of query tiles leaves it one of its own, 0.78 of two, in every head: [26,16,839] on 56 30.5 and 27.4 (39), [69,3,1408] on 62 24.6
// and 22.5 (31), [16,16,1656] on 56 35.5 and 33.8 (45), but [64,12,896] on 64 51.4 and 54.3 (73): twice as far. Heads with fewer than 3 1/3 blocks
// to two tiles stay here: [256,12,300] on 64 84 and 72, [64,12,384] 24.3 and 24.5, [256,12,128] 41.9 and 32.5, but with a bias 47.9 and 51.8.
//
// Above 64 keys a tile is better filled: [4,12,2048] on 80 keys 10.4 and 10.3 (10 blocks per SM), with a bias 13.1 and 13.3, tables 17.7 and 14.3;
// [2,12,2048] on 96 7.5 and 7.2 (5), 9.8 and 9.8, 12.5 and 9.9, [3,12,2048] on 96 8.4 and 9.1 (8), 10.7 and 12.0, 14.0 and 12.2, but heads of one tile,
// [44,12,100] on 100 keys, 9.2 and 9.4 (7), 12.3 and 11.3, 14.2 and 12.6; [2,12,1536] on 128 6.7 and 6.3 (4), [1,12,2048] with a bias 7.6 and 8.4
// (2.6; on 120 keys, where the persistent kernel has columns to mask, 8.2 and 7.8), [2,12,2048] with tables 12.2 and 11.8 (5).
int64_t window_block_limit(const B200AttnArgs* a, int bias, int64_t q_blocks) {
  const int groups = (a->kv_tokens + 15) / 16, q_tiles = (a->q_tokens + 127) / 128;
  const bool filled = 3 * q_blocks >= 10 * static_cast<int64_t>((q_tiles + 1) / 2);
  if (a->kv_tokens > 64) {
    if (bias != kWindowCallRel && groups == 8) return bias == kWindowCallDense && a->kv_tokens == kWindowMaxKeys ? 20 : 40;
    return bias != kWindowCallRel && filled && groups > 5 ? 60 : 520 / groups;
  }
  const int eights = window_eights(a->kv_tokens);
  if (bias == kWindowCallRel || eights <= 4 || (bias == kWindowCallDense && eights < 8)) return 0;
  if (!filled && !(bias == kWindowCallDense && q_blocks == 2)) return 0;
  return (eights == 8 ? 240 : eights == 7 ? 330 : 620) * (q_tiles > 1 ? q_tiles % 2 + 1 : 1);
}

}  // namespace

bool window_pays(const B200AttnArgs* a, const WindowCall& call, int sms) {
  static_assert(kWindowCallMaxKeys == kWindowMaxKeys, "the caller has looked at the key count");
  if (call.bias == kWindowCallRel && a->rel_kh + a->rel_kw > kWindowMaxRel) return false;
  const int64_t q_blocks = (static_cast<int64_t>(a->q_tokens) + kWindowRows - 1) / kWindowRows, blocks = q_blocks * a->batch * a->heads;
  const int64_t limit = window_block_limit(a, call.bias, q_blocks);
  return blocks <= 0x7fffffffLL && (limit == 0 || 10 * blocks <= limit * sms);
}

namespace {

template <typename T, int BIAS>
const void* window_kernel(int keys) {
  switch (window_eights(keys)) {
    case 2: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 2>);
    case 4: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 4>);
    case 6: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 6>);
    case 7: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 7>);
    case 8: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 8>);
    case 10: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 10>);
    case 12: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 12>);
    case 14: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 14>);
    default: return reinterpret_cast<const void*>(attn_window_kernel<T, BIAS, 16>);
  }
}
template <typename T>
const void* window_kernel(int bias, int keys) {
  return bias == kWindowDense ? window_kernel<T, kWindowDense>(keys) : bias == kWindowRel ? window_kernel<T, kWindowRel>(keys) : window_kernel<T, kWindowPlain>(keys);
}

}  // namespace

int launch_window(const B200AttnArgs* a, const WindowCall& call, cudaStream_t stream) {
  WindowParams prm{};
  prm.q = a->q;
  prm.k = a->k;
  prm.v = a->v;
  prm.o = a->o;
  std::copy_n(a->q_stride, 3, prm.q_stride);
  std::copy_n(a->k_stride, 3, prm.k_stride);
  std::copy_n(a->v_stride, 3, prm.v_stride);
  std::copy_n(a->o_stride, 3, prm.o_stride);
  prm.batch = a->batch;
  prm.heads = a->heads;
  prm.q_tokens = a->q_tokens;
  prm.kv_tokens = a->kv_tokens;
  prm.q_blocks = (a->q_tokens + kWindowRows - 1) / kWindowRows;
  prm.magic_blocks = div_magic(prm.q_blocks);
  prm.magic_inner = div_magic(call.batch_fastest ? a->batch : a->heads);
  prm.scale = a->scale;
  prm.scale_log2 = a->scale * kLog2e;
  prm.batch_fastest = call.batch_fastest ? 1 : 0;
  if (call.bias == kWindowCallDense) {
    prm.bias = a->bias;
    std::copy_n(a->bias_stride, 3, prm.bias_stride);
    prm.bias_half = a->bias_dtype == B200_ATTN_F16;
  } else if (call.bias == kWindowCallRel) {
    prm.rel_h = static_cast<const uint16_t*>(a->rel_h);
    prm.rel_w = static_cast<const uint16_t*>(a->rel_w);
    std::copy_n(a->rel_h_stride, 3, prm.rel_h_stride);
    std::copy_n(a->rel_w_stride, 3, prm.rel_w_stride);
    prm.rel_kh = a->rel_kh;
    prm.rel_kw = a->rel_kw;
    prm.rel_pairs = call.rel_align >= 4 && a->rel_kh % 2 == 0 && a->rel_kw % 2 == 0;
    prm.rel_one = call.rel_one;
  }
  const void* kernel = a->dtype == B200_ATTN_F16 ? window_kernel<__half>(call.bias, a->kv_tokens) : window_kernel<__nv_bfloat16>(call.bias, a->kv_tokens);
  void* args[] = {&prm};
  return launch_kernel(kernel, static_cast<unsigned>(prm.q_blocks * a->batch * a->heads), 1, kWindowThreads, 0, 1, stream, args, "attention kernel launch");
}

}  // namespace b200
