// Whole-encoder forwards (include/b200_encoder.h): every kernel of a ViT's or SAM's image encoder launched from one
// native call. A block is eight to ten launches of a few microseconds; issued one by one from Python, with the checks
// and allocations of each operator in between, one image took 1.6 ms where the kernels take a fifth of that.
#include "../../include/b200_encoder.h"

#include <algorithm>
#include <cstring>

#include "../../include/b200_attn.h"
#include "encoder_kernels.cuh"
#include "gemm_sm100.cuh"
#include "host_common.h"
#include "linear_host.h"

namespace {

using namespace b200;

int64_t align256(int64_t bytes) { return (bytes + 255) & ~int64_t(255); }

// Buffers of one forward, as offsets into the workspace.
struct Layout {
  int64_t x, y, qkv, att, hid, rel_h, rel_w, neck, patch_w, neck_w1, total;
  int64_t rows, most_rows;  // tokens of all images; rows of the largest partition into padded windows
};

// Whether the patch embedding's weights have to be padded, and the neck's 3 x 3 weights reordered, in this call.
bool pads_patch_w(const B200EncoderArgs* a) { return a->images != nullptr && a->patch_w_raw != 0 && a->patch_k != 3 * a->patch * a->patch; }
bool reorders_neck_w1(const B200EncoderArgs* a) { return a->neck_w0 != nullptr && a->neck_w1_conv != 0; }

int windows_of(int grid, int side) { return (grid + side - 1) / side; }

int64_t window_rows(const B200EncoderArgs* a, int side) {
  return a->batch * static_cast<int64_t>(windows_of(a->grid_h, side)) * windows_of(a->grid_w, side) * side * side;
}
constexpr int64_t kMaxRows = 0x3fffffff / 9;  // the neck has nine copies of a row, and row numbers are 32-bit

Layout layout_of(const B200EncoderArgs* a) {
  Layout l{};
  const int64_t tokens = a->prefix + static_cast<int64_t>(a->grid_h) * a->grid_w;
  l.rows = a->batch * tokens;
  l.most_rows = l.rows;
  int64_t rel = 0;
  for (int i = 0; i < a->n_blocks; ++i) {
    const B200EncoderBlock& k = a->blocks[i];
    int64_t rows = l.rows, side = a->grid_h;
    if (k.window > 0) {
      side = k.window;
      rows = window_rows(a, k.window);
      l.most_rows = std::max(l.most_rows, rows);
    }
    if (k.rel_pos_h != nullptr) rel = std::max(rel, rows * a->heads * side);
  }
  int64_t wide = l.rows * a->hidden;
  if (a->images != nullptr) wide = std::max(wide, l.rows * a->patch_k);
  if (a->neck_w0 != nullptr) wide = std::max(wide, l.rows * 9 * a->neck_channels);
  int64_t at = 0;
  const auto take = [&](int64_t values) {
    const int64_t here = at;
    at += align256(values * 2);
    return here;
  };
  l.x = take(a->x == nullptr ? l.rows * a->dim : 0);
  l.y = take(l.most_rows * a->dim);
  l.qkv = take(l.most_rows * 3 * a->dim);
  l.att = take(l.most_rows * a->dim);
  l.hid = take(wide);
  l.rel_h = take(rel);
  l.rel_w = take(rel);
  l.neck = take(a->neck_w0 != nullptr ? l.rows * a->neck_channels : 0);
  l.patch_w = take(pads_patch_w(a) ? static_cast<int64_t>(a->dim) * a->patch_k : 0);
  l.neck_w1 = take(reorders_neck_w1(a) ? 9LL * a->neck_channels * a->neck_channels : 0);
  l.total = at;
  return l;
}

template <typename T>
const void* norm_kernel(int chunks) {
  switch (chunks) {
    case 1: return reinterpret_cast<const void*>(layer_norm_kernel<T, 1>);
    case 2: return reinterpret_cast<const void*>(layer_norm_kernel<T, 2>);
    case 3: return reinterpret_cast<const void*>(layer_norm_kernel<T, 3>);
    case 4: return reinterpret_cast<const void*>(layer_norm_kernel<T, 4>);
    case 5: return reinterpret_cast<const void*>(layer_norm_kernel<T, 5>);
    case 6: return reinterpret_cast<const void*>(layer_norm_kernel<T, 6>);
    case 7: return reinterpret_cast<const void*>(layer_norm_kernel<T, 7>);
    default: return reinterpret_cast<const void*>(layer_norm_kernel<T, 8>);
  }
}

int launch_norm(uint32_t dtype, NormParams prm, cudaStream_t stream) {
  const int chunks = (prm.dim + 255) / 256;
  const void* kernel = dtype == B200_ATTN_F16 ? norm_kernel<__half>(chunks) : norm_kernel<__nv_bfloat16>(chunks);
  void* args[] = {&prm};
  return launch_kernel(kernel, static_cast<unsigned>((prm.rows + kNormWarps - 1) / kNormWarps), 1, kNormWarps * 32, 0, 1, stream, args, "layer norm launch");
}

int check(const B200EncoderArgs* a) {
  if (a == nullptr) return fail(B200_ATTN_BAD_CONFIG, "args is NULL");
  if (a->struct_size != sizeof(B200EncoderArgs))
    return fail(B200_ATTN_BAD_CONFIG, "struct_size %u does not match this library's B200EncoderArgs (%zu bytes)", a->struct_size, sizeof(B200EncoderArgs));
  if (a->dtype != B200_ATTN_F16 && a->dtype != B200_ATTN_BF16) return fail(B200_ATTN_BAD_CONFIG, "dtype %u: fp16 (0) or bf16 (1)", a->dtype);
  if (a->batch < 1 || a->grid_h < 1 || a->grid_w < 1 || a->prefix < 0 || a->n_blocks < 0 || (a->n_blocks > 0 && a->blocks == nullptr))
    return fail(B200_ATTN_BAD_CONFIG, "batch %d grid %d x %d prefix %d blocks %d", a->batch, a->grid_h, a->grid_w, a->prefix, a->n_blocks);
  if (a->heads < 1 || a->dim != a->heads * 64 || a->dim > 2048) return fail(B200_ATTN_UNSUPPORTED, "dim %d: heads (%d) * 64, at most 2048", a->dim, a->heads);
  if (a->hidden < 8 || a->hidden % 8 != 0) return fail(B200_ATTN_UNSUPPORTED, "hidden %d must be a positive multiple of 8", a->hidden);
  if (a->ffn < B200_FFN_GELU_TANH || a->ffn > B200_FFN_GELU) return fail(B200_ATTN_BAD_CONFIG, "ffn %d unknown", a->ffn);
  const int64_t rows = a->batch * (a->prefix + static_cast<int64_t>(a->grid_h) * a->grid_w);
  if (rows > kMaxRows) return fail(B200_ATTN_UNSUPPORTED, "too many tokens for one call");
  if (a->images != nullptr) {
    if (a->patch < 2 || a->patch % 2 != 0 || a->patch_k < 3 * a->patch * a->patch || a->patch_k % 8 != 0 || a->width % 2 != 0 ||
        a->height < a->grid_h * a->patch || a->width < a->grid_w * a->patch || (a->image_dtype != B200_ATTN_F32 && a->image_dtype != a->dtype))
      return fail(B200_ATTN_UNSUPPORTED, "images %d x %d with patches of %d, patch_k %d, image_dtype %u", a->height, a->width, a->patch, a->patch_k, a->image_dtype);
    if (a->patch_w == nullptr || a->start == nullptr) return fail(B200_ATTN_BAD_CONFIG, "images need patch_w and start");
  } else if (a->x == nullptr) {
    return fail(B200_ATTN_BAD_CONFIG, "neither images nor x");
  }
  for (int i = 0; i < a->n_blocks; ++i) {
    const B200EncoderBlock& k = a->blocks[i];
    if (k.window < 0 || (k.window > 0 && a->prefix != 0)) return fail(B200_ATTN_BAD_CONFIG, "block %d: window %d with %d prefix tokens", i, k.window, a->prefix);
    if (k.rel_pos_h != nullptr && k.window == 0 && a->grid_h != a->grid_w) return fail(B200_ATTN_UNSUPPORTED, "block %d: relative positions need a square grid", i);
    const int side = k.window > 0 ? k.window : a->grid_h;
    if (k.rel_pos_h != nullptr && (side < 2 || side > 64 || side % 2 != 0)) return fail(B200_ATTN_UNSUPPORTED, "block %d: relative positions over a side of %d: even, 2 .. 64", i, side);
    if (k.window > 0 && (k.window > 0x7fff || window_rows(a, k.window) > kMaxRows)) return fail(B200_ATTN_UNSUPPORTED, "block %d: too many tokens in windows of %d for one call", i, k.window);
  }
  if (a->neck_w0 != nullptr && (a->prefix != 0 || a->neck_channels < 8 || a->neck_channels % 8 != 0 || a->neck_channels > kNeckChunks * 256 || a->neck_out == nullptr))
    return fail(B200_ATTN_UNSUPPORTED, "neck of %d channels", a->neck_channels);
  return B200_ATTN_OK;
}

// What every kernel takes for granted of the addresses: there and on 16-byte boundaries (vector and TMA accesses).
int check_pointers(const B200EncoderArgs* a) {
  int rc = B200_ATTN_OK;
  const auto look = [&](const char* what, int i, const char* name, const void* ptr, bool required) {
    if (rc != B200_ATTN_OK) return;
    if (ptr == nullptr && required) rc = fail(B200_ATTN_BAD_CONFIG, "%s %d: %s is NULL", what, i, name);
    else if (!aligned16(ptr)) rc = fail(B200_ATTN_UNSUPPORTED, "%s %d: %s is not 16-byte aligned", what, i, name);
  };
  const bool images = a->images != nullptr, neck = a->neck_w0 != nullptr;
  look("call", 0, "images", a->images, false);
  look("call", 0, "x", a->x, false);
  look("call", 0, "patch_w", a->patch_w, images);
  look("call", 0, "start", a->start, images);
  look("call", 0, "patch_b", a->patch_b, false);
  look("call", 0, "first", a->first, false);
  if (a->n_taps < 0 || (a->n_taps > 0 && a->taps == nullptr)) return fail(B200_ATTN_BAD_CONFIG, "n_taps %d without taps", a->n_taps);
  look("call", 0, "norm_w", a->norm_w, a->n_taps > 0);
  look("call", 0, "norm_b", a->norm_b, a->n_taps > 0);
  for (int i = 0; i < a->n_taps; ++i) look("tap", i, "out", a->taps[i].out, true);
  look("neck", 0, "neck_w0", a->neck_w0, false);
  look("neck", 0, "neck_n0_w", a->neck_n0_w, neck);
  look("neck", 0, "neck_n0_b", a->neck_n0_b, neck);
  look("neck", 0, "neck_w1", a->neck_w1, neck);
  look("neck", 0, "neck_n1_w", a->neck_n1_w, neck);
  look("neck", 0, "neck_n1_b", a->neck_n1_b, neck);
  look("neck", 0, "neck_out", a->neck_out, neck);
  for (int i = 0; i < a->n_blocks; ++i) {
    const B200EncoderBlock& k = a->blocks[i];
    look("block", i, "norm1_w", k.norm1_w, true);
    look("block", i, "norm1_b", k.norm1_b, true);
    look("block", i, "qkv_w", k.qkv_w, true);
    look("block", i, "qkv_b", k.qkv_b, false);
    look("block", i, "proj_w", k.proj_w, true);
    look("block", i, "proj_b", k.proj_b, false);
    look("block", i, "gamma1", k.gamma1, false);
    look("block", i, "norm2_w", k.norm2_w, true);
    look("block", i, "norm2_b", k.norm2_b, true);
    look("block", i, "fc1_w", k.fc1_w, true);
    look("block", i, "fc1_b", k.fc1_b, false);
    look("block", i, "fc2_w", k.fc2_w, true);
    look("block", i, "fc2_b", k.fc2_b, false);
    look("block", i, "gamma2", k.gamma2, false);
    look("block", i, "rel_pos_h", k.rel_pos_h, k.rel_pos_w != nullptr);
    look("block", i, "rel_pos_w", k.rel_pos_w, k.rel_pos_h != nullptr);
  }
  return rc;
}

// The launches of one forward.
struct Forward {
  const B200EncoderArgs* a;
  Layout l;
  cudaStream_t stream;
  char* ws;
  void* x;
  mutable bool started = false;  // a kernel of this forward is in front: the weights were complete before that one started

  void* at(int64_t offset) const { return ws + offset; }

  // y = act((x w^T + b) * gamma + res). A product behind a kernel of this forward may load its weights ahead of that
  // kernel's end: they were complete before it started. Not so in front (the neck of an encoder without blocks on given
  // tokens may follow the kernel that writes them), and weights repacked in this forward are left to the wait as well.
  int linear(const void* in, int m, int k, const void* w, const void* b, int n, void* out, int act, const float* gamma = nullptr, const void* res = nullptr, bool made_here = false, bool backwards = false) const {
    const GemmCall c{a->dtype, m, n, k, act, in, k, w, b, gamma, res, n, out, n, started && !made_here, backwards};
    started = true;
    return launch_gemm(c, stream);
  }

  int norm(const void* in, const void* w, const void* b, void* out, int rows, float eps, WindowMap map = WindowMap{}, void* x_out = nullptr, const void* delta = nullptr) const {
    NormParams p{};
    p.x = in; p.x_out = x_out; p.delta = delta; p.weight = w; p.bias = b; p.y = out;
    p.rows = rows; p.dim = a->dim; p.eps = eps; p.map = map;
    p.early_w = started ? 1 : 0;
    started = true;
    return launch_norm(a->dtype, p, stream);
  }

  int repack(const void* src, int rows, int cols, int out_cols, int taps, int64_t to) const {
    RepackParams p{src, at(to), cols, out_cols, taps};
    started = true;
    void* args[] = {&p};
    return launch_kernel(reinterpret_cast<const void*>(repack_kernel), static_cast<unsigned>(rows), 1, kRepackThreads, 0, 1, stream, args, "weight repacking launch");
  }

  int start_tokens() const {
    const void* w = a->patch_w;
    if (pads_patch_w(a)) {
      w = at(l.patch_w);
      if (int rc = repack(a->patch_w, a->dim, 3 * a->patch * a->patch, a->patch_k, 0, l.patch_w)) return rc;
    }
    TokensParams p{};
    p.images = a->images;
    p.image_f32 = a->image_dtype == B200_ATTN_F32;
    p.batch = a->batch; p.height = a->height; p.width = a->width; p.patch = a->patch;
    p.grid_h = a->grid_h; p.grid_w = a->grid_w; p.prefix = a->prefix;
    p.k = 3 * a->patch * a->patch; p.k_padded = a->patch_k;
    p.patches = at(l.hid); p.start = a->start; p.x = x; p.dim = a->dim;
    p.start_f32 = a->start_f32; p.patch_b = a->patch_b; p.first = a->first;
    started = true;
    void* args[] = {&p};
    const void* kernel = a->dtype == B200_ATTN_F16 ? reinterpret_cast<const void*>(encoder_tokens_kernel<__half>) : reinterpret_cast<const void*>(encoder_tokens_kernel<__nv_bfloat16>);
    if (int rc = launch_kernel(kernel, static_cast<unsigned>(a->batch * a->grid_h), static_cast<unsigned>(tokens_parts(a->patch)), kTokensThreads, 0, 1, stream, args, "encoder tokens launch")) return rc;
    return linear(at(l.hid), static_cast<int>(l.rows), a->patch_k, w, nullptr, a->dim, x, kActNone, nullptr, x, pads_patch_w(a));
  }

  int attention(const B200EncoderBlock& k, int batch, int tokens, int side) const {
    const int dim = a->dim;
    B200AttnArgs t;
    std::memset(&t, 0, sizeof(t));
    t.struct_size = sizeof(t);
    t.dtype = a->dtype;
    char* qkv = static_cast<char*>(at(l.qkv));
    t.q = qkv; t.k = qkv + 2 * dim; t.v = qkv + 4 * dim;
    t.o = at(l.att);
    for (int64_t* s : {t.q_stride, t.k_stride, t.v_stride}) {
      s[0] = static_cast<int64_t>(tokens) * 3 * dim;
      s[1] = 3 * dim;
      s[2] = 64;
    }
    t.o_stride[0] = static_cast<int64_t>(tokens) * dim;
    t.o_stride[1] = dim;
    t.o_stride[2] = 64;
    t.batch = batch; t.heads = a->heads; t.q_tokens = tokens; t.kv_tokens = tokens; t.head_dim = 64;
    t.scale = 0.125f;
    t.workspace = a->attn_workspace;
    t.workspace_bytes = a->attn_workspace_bytes;
    if (k.rel_pos_h != nullptr) {
      B200RelTermsArgs r;
      std::memset(&r, 0, sizeof(r));
      r.struct_size = sizeof(r);
      r.dtype = a->dtype;
      r.q = t.q;
      std::memcpy(r.q_stride, t.q_stride, sizeof(r.q_stride));
      r.rel_pos_h = k.rel_pos_h; r.rel_pos_w = k.rel_pos_w;
      r.rel_h = at(l.rel_h); r.rel_w = at(l.rel_w);
      r.batch = batch; r.heads = a->heads; r.side = side; r.head_dim = 64;
      if (int rc = launch_rel_terms(&r, started, stream)) return rc;  // always behind a product of this forward
      t.rel_h = r.rel_h; t.rel_w = r.rel_w;
      t.rel_dtype = a->dtype;
      t.rel_kh = t.rel_kw = side;
      for (int64_t* s : {t.rel_h_stride, t.rel_w_stride}) {
        s[0] = static_cast<int64_t>(a->heads) * tokens * side;
        s[1] = static_cast<int64_t>(tokens) * side;
        s[2] = side;
      }
    }
    return b200_attn_fwd(&t, stream);
  }

  // Activations of a large batch do not fit L2. What a kernel wrote last is still there, and one that begins with that finds it: with norms
  // and attention going forwards through the rows, qkv, projection and fc1 go backwards, and fc2 forwards. The line is drawn by the qkv tensor
  // of the tokens (padded windows add up to a third to it). us for twelve blocks, all forwards and so, 518 px images, medians of five in turn:
  // at 34 to 38 MB the same (ViT-L/14 at 4 2440 and 2443, ViT-B/14 at 6 2295 and 2300, ViT-S/14 at 12 1781 and 1801; SAM ViT-B at two images of 1024 px
  // 2830 and 2831), at 42 to 44 hardly less (ViT-L/14 at 5 2854 and 2845, ViT-B/14 at 7 2701 and 2686), from 51 on 0.4 to 2 % less (ViT-L/14 at 6 3423
  // and 3371, ViT-B/14 at 8 2933 and 2902, ViT-g/14 at 4 4288 and 4231; SAM at three, 57 MB, 4087 and 4044, at four 5415 and 5344; ViT-L/14 at 16, 135 MB,
  // 8598 and 8495, ViT-B/14 at 16 5687 and 5555, ViT-g/14 at 16, 202 MB, 15955 and 15760).
  static constexpr int64_t kLargeQkvBytes = 48 << 20;
  int block(const B200EncoderBlock& k) const {
    const int rows = static_cast<int>(l.rows), dim = a->dim;
    const bool back = l.rows * 6 * dim > kLargeQkvBytes;
    const int tokens = a->prefix + a->grid_h * a->grid_w;
    if (k.window > 0) {
      // Windowed attention (SAM): the first norm writes the padded windows, the projection stays in window order, and the
      // second norm takes it back to token order while it adds it to the residual stream.
      const WindowMap map{k.window, a->grid_h, a->grid_w, windows_of(a->grid_w, k.window), windows_of(a->grid_h, k.window)};
      const int windows = a->batch * map.per_row * map.per_col, area = k.window * k.window, wrows = windows * area;
      if (int rc = norm(x, k.norm1_w, k.norm1_b, at(l.y), wrows, a->eps, map)) return rc;
      if (int rc = linear(at(l.y), wrows, dim, k.qkv_w, k.qkv_b, 3 * dim, at(l.qkv), kActNone, nullptr, nullptr, false, back)) return rc;
      if (int rc = attention(k, windows, area, k.window)) return rc;
      if (int rc = linear(at(l.att), wrows, dim, k.proj_w, k.proj_b, dim, at(l.y), kActNone, k.gamma1, nullptr, false, back)) return rc;
      if (int rc = norm(x, k.norm2_w, k.norm2_b, at(l.att), rows, a->eps, map, x, at(l.y))) return rc;
    } else {
      if (int rc = norm(x, k.norm1_w, k.norm1_b, at(l.y), rows, a->eps)) return rc;
      if (int rc = linear(at(l.y), rows, dim, k.qkv_w, k.qkv_b, 3 * dim, at(l.qkv), kActNone, nullptr, nullptr, false, back)) return rc;
      if (int rc = attention(k, a->batch, tokens, a->grid_h)) return rc;
      if (int rc = linear(at(l.att), rows, dim, k.proj_w, k.proj_b, dim, x, kActNone, k.gamma1, x, false, back)) return rc;
      if (int rc = norm(x, k.norm2_w, k.norm2_b, at(l.att), rows, a->eps)) return rc;
    }
    const int act = a->ffn == B200_FFN_SWIGLU ? kActSwiGlu : a->ffn == B200_FFN_GELU ? kActGelu : kActGeluTanh;
    if (int rc = linear(at(l.att), rows, dim, k.fc1_w, k.fc1_b, a->hidden, at(l.hid), act, nullptr, nullptr, false, back)) return rc;
    return linear(at(l.hid), rows, a->hidden, k.fc2_w, k.fc2_b, dim, x, kActNone, k.gamma2, x);
  }

  int neck() const {
    const int rows = static_cast<int>(l.rows), ch = a->neck_channels;
    if (int rc = linear(x, rows, a->dim, a->neck_w0, nullptr, ch, at(l.neck), kActNone)) return rc;
    const void* w1 = a->neck_w1;
    if (reorders_neck_w1(a)) {
      w1 = at(l.neck_w1);
      if (int rc = repack(a->neck_w1, ch, 9 * ch, 9 * ch, 9, l.neck_w1)) return rc;
    }
    NeckParams p{};
    p.x = at(l.neck); p.weight = a->neck_n0_w; p.bias = a->neck_n0_b; p.out = at(l.hid);
    p.batch = a->batch; p.grid_h = a->grid_h; p.grid_w = a->grid_w; p.channels = ch; p.eps = a->neck_eps;
    void* args[] = {&p};
    const bool f16 = a->dtype == B200_ATTN_F16;
    const void* im2col = f16 ? reinterpret_cast<const void*>(neck_norm_im2col_kernel<__half>) : reinterpret_cast<const void*>(neck_norm_im2col_kernel<__nv_bfloat16>);
    if (int rc = launch_kernel(im2col, static_cast<unsigned>((rows + kNeckWarps - 1) / kNeckWarps), 1, kNeckWarps * 32, 0, 1, stream, args, "neck norm launch")) return rc;
    if (int rc = linear(at(l.hid), rows, 9 * ch, w1, nullptr, ch, at(l.neck), kActNone, nullptr, nullptr, reorders_neck_w1(a))) return rc;
    p.weight = a->neck_n1_w; p.bias = a->neck_n1_b; p.out = a->neck_out;
    const void* chw = f16 ? reinterpret_cast<const void*>(neck_norm_chw_kernel<__half>) : reinterpret_cast<const void*>(neck_norm_chw_kernel<__nv_bfloat16>);
    const int area = a->grid_h * a->grid_w;
    const unsigned grid = static_cast<unsigned>(a->batch * ((area + kNeckTokens - 1) / kNeckTokens));
    return launch_kernel(chw, grid, 1, kNeckWarps * 32, static_cast<size_t>(ch) * (kNeckTokens + 2) * 2, 1, stream, args, "neck norm launch");
  }
};

}  // namespace

extern "C" {

int b200_encoder_workspace(const B200EncoderArgs* a, int64_t* bytes) {
  if (int rc = check(a)) return rc;
  if (bytes == nullptr) return fail(B200_ATTN_BAD_CONFIG, "bytes is NULL");
  *bytes = layout_of(a).total;
  return B200_ATTN_OK;
}

int b200_encoder_forward(const B200EncoderArgs* a, void* stream_ptr) {
  if (int rc = check(a)) return rc;
  if (int rc = check_pointers(a)) return rc;
  Forward f{a, layout_of(a), static_cast<cudaStream_t>(stream_ptr), static_cast<char*>(a->workspace), nullptr};
  if (a->workspace == nullptr || (reinterpret_cast<uintptr_t>(a->workspace) & 255) != 0 || a->workspace_bytes < f.l.total)
    return fail(B200_ATTN_BAD_CONFIG, "workspace of %lld bytes: %lld, 256-byte aligned, are needed", static_cast<long long>(a->workspace_bytes), static_cast<long long>(f.l.total));
  f.x = a->x != nullptr ? a->x : f.at(f.l.x);
  if (a->images != nullptr)
    if (int rc = f.start_tokens()) return rc;
  int tap = 0;
  for (int i = -1; i < a->n_blocks; ++i) {
    if (i >= 0)
      if (int rc = f.block(a->blocks[i])) return rc;
    for (; tap < a->n_taps && a->taps[tap].after == i; ++tap)
      if (int rc = f.norm(f.x, a->norm_w, a->norm_b, a->taps[tap].out, static_cast<int>(f.l.rows), a->eps)) return rc;
  }
  if (tap != a->n_taps) return fail(B200_ATTN_BAD_CONFIG, "tap %d of %d names no block, or the taps are out of order", tap, a->n_taps);
  if (a->neck_w0 != nullptr)
    if (int rc = f.neck()) return rc;
  clear_error();
  return B200_ATTN_OK;
}

}  // extern "C"
