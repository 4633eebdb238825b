// Rule and launch of the attention kernel for few keys (attn_window_sm100.cuh).
#include <algorithm>

#include "attn_window_sm100.cuh"
#include "window_host.h"

namespace b200 {

// Up to 64 keys this kernel is the faster one at every size that was tried (3 to 12288 heads: 0.2 to 0.55 of the persistent kernel's
// time). Above, a 128 x 128 tile is better filled, and it pays while the blocks of 64 queries are few rounds of CTAs. Ratio of the times
// here and there by blocks x groups of 16 keys per SM: [16,16,98] with a dense bias 24: 0.88, [16,24,80] likewise 26: 0.76, [25,12,100]
// with 10 x 10 tables 28: 0.77, [64,12,80] 52: 0.91; [64,12,112] 73: 1.10, [64,16,98] 97: 1.13, [64,16,128] 111: 1.31.
constexpr int kWindowGroupsPerSm = 52;

bool window_pays(const B200AttnArgs* a, const WindowCall& call, int sms) {
  static_assert(kWindowCallMaxKeys == kWindowMaxKeys, "one limit");
  if (a->kv_tokens > kWindowMaxKeys) return false;
  if (call.bias == kWindowCallRel && a->rel_kh + a->rel_kw > kWindowMaxRel) return false;
  const int64_t blocks = (static_cast<int64_t>(a->q_tokens) + kWindowRows - 1) / kWindowRows * a->batch * a->heads;
  const int groups = (a->kv_tokens + 15) / 16;
  return blocks <= 0x7fffffffLL && (a->kv_tokens <= 64 || blocks * groups <= static_cast<int64_t>(kWindowGroupsPerSm) * sms);
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
