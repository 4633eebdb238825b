// C entry points of the layers around attention: the GEMM with fused epilogue, the producer of SAM's decomposed bias and
// DINOv3's rotary embedding. Declarations are in include/b200_attn.h.
#include "../../include/b200_attn.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "gemm_sm100.cuh"
#include "host_common.h"
#include "linear_host.h"
#include "rope_sm100.cuh"
#include "sam_rel_terms.cuh"

namespace b200 {

namespace {

constexpr int kHeadDim = 64;

// 2-D tensor maps (rows of contiguous 16-bit values, boxes of 64 columns, 128-byte swizzle) made before, per thread: an
// encoder passes the same weights and, through the caching allocator, the same activations in every forward, and a map
// depends on nothing but the key, so a hit is exact.
struct MatrixMapKey {
  const void* base;
  int64_t stride, rows;
  int cols, box_rows;
  uint32_t dtype;
  bool operator==(const MatrixMapKey& o) const {
    return base == o.base && stride == o.stride && rows == o.rows && cols == o.cols && box_rows == o.box_rows && dtype == o.dtype;
  }
};
constexpr int kMatrixMapSets = 512, kMatrixMapWays = 2;  // a 40-block encoder has 160 weight matrices
struct MatrixMapCache {
  MatrixMapKey key[kMatrixMapSets][kMatrixMapWays];
  CUtensorMap map[kMatrixMapSets][kMatrixMapWays];
  bool used[kMatrixMapSets][kMatrixMapWays];
  uint8_t next[kMatrixMapSets];
};
thread_local MatrixMapCache tl_matrix_maps{};

int matrix_map(CUtensorMap* map, const void* base, uint32_t dtype, int64_t rows, int cols, int64_t stride, int box_rows, const char* name) {
  const MatrixMapKey key{base, stride, rows, cols, box_rows, dtype};
  const size_t h = ((reinterpret_cast<uintptr_t>(base) >> 8) + static_cast<size_t>(box_rows)) * 0x9E3779B97F4A7C15ull >> 55;  // 9 bits
  MatrixMapCache& c = tl_matrix_maps;
  for (int w = 0; w < kMatrixMapWays; ++w)
    if (c.used[h][w] && c.key[h][w] == key) {
      *map = c.map[h][w];
      return B200_ATTN_OK;
    }
  EncodeTiledFn enc = encode_tiled_fn();
  if (enc == nullptr) return fail(B200_ATTN_CUDA_ERROR_BASE, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(stride) * 2};
  const cuuint32_t box[2] = {kGemmBK, static_cast<cuuint32_t>(box_rows)}, elem[2] = {1, 1};
  const CUresult r = enc(map, dtype == B200_ATTN_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                         const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(B200_ATTN_UNSUPPORTED, "tensor map for %s rejected by the driver (CUresult %d)", name, static_cast<int>(r));
  const int w = c.next[h];
  c.next[h] = static_cast<uint8_t>((w + 1) % kMatrixMapWays);
  c.key[h][w] = key;
  c.map[h][w] = *map;
  c.used[h][w] = true;
  return B200_ATTN_OK;
}

int opt_in(DeviceState& dev, int form, const void* kernel, int smem) {
  if (dev.linear_opted_in[form].load(std::memory_order_acquire)) return B200_ATTN_OK;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(shared memory)");
  dev.linear_opted_in[form].store(true, std::memory_order_release);
  return B200_ATTN_OK;
}

}  // namespace

// Estimated microseconds, from timings of every form in CUDA graphs at 197 .. 21920 rows (B200, 1.93 GHz). A pair tile
// of 256 x bn pays 3.6 + bn / 180 for launch, set-up and the epilogue nothing hides, then so much per k-block when the
// whole GPU pulls operands: at bn = 256 the products (0.27 alone), below it what the issuing thread and the L2 allow. (Set-up and exit have
// become 1.2 shorter since. Of 180 products of 197 to 5480 rows, run in every way, the plan took one within 2 % of the best for all but 15,
// the worst 10 % behind at 4.1 us.)
double pair_k_block_us(int bn) { return bn == 256 ? 0.298 : bn == 192 ? 0.25 : bn == 128 ? 0.21 : 0.205; }
constexpr double kPairRoundUs = 0.15;
// Row tiles per raster group: 74 pairs then work on four rows of x tiles and a dozen or two of w tiles at a time. us with groups of
// 16 and of 4 (1 to 6 are within 0.5 %): [5480,3072,1024] 33.7 and 32.9, [5480,1024,4096] 49.2 and 48.3, [4096,3072,768] 25.5 and 24.1,
// [32928,3072,1024] 172.8 and 169.9, [21920,4608,1536] 236.1 and 233.9, all in loops of some milliseconds; of few products
// [21920,1536,4096] 181 and 175, [4096,8192,1024] 54.1 and 50.0, [16384,9216,1024] 218 and 215, but [4096,4096,4096] 91.7 and 92.5. With more than
// 10240 rows of w every group reads a w that the outputs have pushed out of L2: [16384,16384,1024] 387 and 401,
// [4096,12288,4096] 264 and 279, [4096,16384,2048] 182 and 190.
constexpr int pair_group(int64_t w_rows) { return w_rows > 10240 ? 16 : 4; }
// A CTA of the split kernel: 2.5 for set-up, first loads and epilogue, 0.2 per k-block, 0.3 for the merge of a cluster.
constexpr double kSplitRoundUs = 2.5, kSplitKBlockUs = 0.2, kSplitMergeUs = 0.3, kSplitLaunchUs = 0.6;
static_assert(kGemmSplits == 6, "split counts");
constexpr int kSplits[kGemmSplits] = {1, 2, 3, 4, 6, 8};

GemmPlan gemm_plan(int m, int n, int k, bool swiglu, int sms, const int* split_clusters) {
  const int k_blocks = (k + kGemmBK - 1) / kGemmBK;
  GemmPlan best{256, 0, 0};
  if (swiglu) return best;
  const long long pairs = std::max(1, sms / 2);
  double best_us = 1e300;
  for (int bn = 256; bn >= 64; bn -= 64) {
    if (bn > 64 && bn - 64 >= n) continue;  // a narrower tile covers all columns
    const long long tiles = static_cast<long long>((m + 255) / 256) * ((n + bn - 1) / bn);
    const long long whole = tiles / pairs, behind = tiles % pairs;
    const double start = 3.6 + bn / 180.0, round = k_blocks * pair_k_block_us(bn) + kPairRoundUs;
    const double us = start + static_cast<double>(whole + (behind > 0 ? 1 : 0)) * round;
    if (us < best_us) {
      best_us = us;
      best = GemmPlan{bn, 0, 0};
    }
    // The tiles behind the last whole round in narrow parts: a thin last round (proj and fc2 of ViT-L/14 at four images:
    // 88 tiles on 74 pairs) then takes 0.7 of a round instead of a whole one.
    for (int tail = 128; tail >= 64 && whole > 0 && behind > 0 && bn == 256; tail -= 64) {
      const long long parts = behind * (bn / tail);
      const double split_us = start + static_cast<double>(whole) * round + static_cast<double>((parts + pairs - 1) / pairs) * (k_blocks * pair_k_block_us(tail) + kPairRoundUs);
      if (split_us < 0.98 * best_us) {
        best_us = split_us;
        best = GemmPlan{bn, 0, tail};
      }
    }
  }
  const long long tiles = static_cast<long long>((m + 127) / 128) * ((n + kSplitBN - 1) / kSplitBN);
  for (const int s : kSplits) {
    const int at_once = *split_clusters++;
    if (s > k_blocks || at_once < 1 || tiles > 3LL * at_once) continue;
    const double rounds = static_cast<double>((tiles + at_once - 1) / at_once);
    const double us = kSplitLaunchUs + rounds * (kSplitRoundUs + (k_blocks + s - 1) / s * kSplitKBlockUs + (s > 1 ? kSplitMergeUs : 0.0));
    if (us < best_us) {
      best_us = us;
      best = GemmPlan{64, s, 0};
    }
  }
  return best;
}

struct SplitForm {
  const void* f16;
  const void* bf16;
  size_t smem;
};
template <int S>
SplitForm split_form() {
  return {reinterpret_cast<const void*>(gemm_split_kernel<__half, S>), reinterpret_cast<const void*>(gemm_split_kernel<__nv_bfloat16, S>), sizeof(SplitSmem<S>)};
}

const SplitForm* split_forms() {
  static const SplitForm forms[kGemmSplits] = {split_form<1>(), split_form<2>(), split_form<3>(), split_form<4>(), split_form<6>(), split_form<8>()};
  return forms;
}

// How many clusters of every split fit the device at once (clusters do not cross the GPU's processing clusters, so it is
// fewer than SMs / S), asked once per device.
int split_clusters(DeviceState& dev) {
  if (dev.splits_ready.load(std::memory_order_acquire)) return B200_ATTN_OK;
  int fit[kGemmSplits];
  for (int i = 0; i < kGemmSplits; ++i) {
    const SplitForm& f = split_forms()[i];
    const int smem = static_cast<int>(f.smem) + 1024;
    for (const void* kernel : {f.f16, f.bf16}) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(shared memory)");
    }
    if (kSplits[i] == 1) {
      fit[i] = dev.sms;
      continue;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(kSplits[i]) * 64u);
    config.blockDim = dim3(kSplitThreads);
    config.dynamicSmemBytes = static_cast<size_t>(smem);
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = static_cast<unsigned>(kSplits[i]);
    attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    fit[i] = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&fit[i], f.f16, &config);
    if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveClusters");
  }
  for (int i = 0; i < kGemmSplits; ++i) dev.split_clusters[i].store(fit[i], std::memory_order_relaxed);
  dev.splits_ready.store(true, std::memory_order_release);
  return B200_ATTN_OK;
}

// [dtype][act][form]; SwiGLU layers have neither scale nor residual.
int pair_act_index(int act) { return act == kActNone ? 0 : act == kActRelu ? 1 : act == kActGelu ? 2 : act == kActGeluTanh ? 3 : 4; }
template <typename T, int ACT>
const void* pair_kernel_of(int form) {
  switch (form) {
    case kPairResidual: return reinterpret_cast<const void*>(gemm_pair_kernel<T, ACT, kPairResidual>);
    case kPairScaled: return reinterpret_cast<const void*>(gemm_pair_kernel<T, ACT, kPairScaled>);
    default: return reinterpret_cast<const void*>(gemm_pair_kernel<T, ACT, kPairPlain>);
  }
}
template <typename T>
const void* pair_kernel(int act, int form) {
  switch (act) {
    case kActRelu: return pair_kernel_of<T, kActRelu>(form);
    case kActGelu: return pair_kernel_of<T, kActGelu>(form);
    case kActGeluTanh: return pair_kernel_of<T, kActGeluTanh>(form);
    case kActSwiGlu: return reinterpret_cast<const void*>(gemm_pair_kernel<T, kActSwiGlu, kPairPlain>);
    default: return pair_kernel_of<T, kActNone>(form);
  }
}

int launch_gemm(const GemmCall& c, cudaStream_t stream) {
  DeviceState* dev = nullptr;
  if (int rc = device_state(&dev)) return rc;
  const bool swiglu = c.act == kActSwiGlu, f16 = c.dtype == B200_ATTN_F16;
  if (int rc = split_clusters(*dev)) return rc;
  int fit[kGemmSplits];
  for (int i = 0; i < kGemmSplits; ++i) fit[i] = dev->split_clusters[i].load(std::memory_order_relaxed);
  const GemmPlan plan = gemm_plan(c.m, c.n, c.k, swiglu, dev->sms, fit);
  GemmParams prm{};
  prm.m = c.m; prm.n = c.n; prm.k = c.k;
  prm.bias = c.bias; prm.scale = c.scale; prm.res = c.res; prm.lres = c.lres;
  prm.y = c.y; prm.ldy = c.ldy; prm.act = c.act;
  prm.early_w = c.early_w ? 1 : 0;
  prm.backwards = c.backwards ? 1 : 0;
  prm.status = dev->status;
  const int64_t w_rows = swiglu ? 2LL * c.n : c.n;
  CUtensorMap mx, mw;
  if (int rc = matrix_map(&mx, c.x, c.dtype, c.m, c.k, c.lda, 128, "x")) return rc;
  if (plan.split == 0) {
    prm.bn = plan.bn;
    const int out_cols = swiglu ? 128 : plan.bn;
    prm.tiles_m = (c.m + 255) / 256;
    prm.tiles_n = (c.n + out_cols - 1) / out_cols;
    prm.group_m = std::min(prm.tiles_m, pair_group(w_rows));
    const long long tiles = static_cast<long long>(prm.tiles_m) * prm.tiles_n;
    if (tiles > 0x3fffffffLL) return fail(B200_ATTN_UNSUPPORTED, "problem too large for one launch");
    prm.stages = std::min(kPairMaxStages, kPairRingBytes / (kGemmTileBytes + plan.bn * kGemmBK));
    prm.whole_tiles = static_cast<int>(plan.tail_bn == 0 ? tiles : tiles / (dev->sms / 2) * (dev->sms / 2));
    prm.tail_bn = plan.tail_bn == 0 ? plan.bn : plan.tail_bn;
    prm.tail_parts = (plan.bn + prm.tail_bn - 1) / prm.tail_bn;
    const long long items = prm.whole_tiles + (tiles - prm.whole_tiles) * prm.tail_parts;
    CUtensorMap my, mr, mwt;
    if (int rc = matrix_map(&mw, c.w, c.dtype, w_rows, c.k, c.k, plan.bn / 2, "w")) return rc;
    mwt = mw;
    if (plan.tail_bn != 0)
      if (int rc = matrix_map(&mwt, c.w, c.dtype, w_rows, c.k, c.k, plan.tail_bn / 2, "w")) return rc;
    if (int rc = matrix_map(&my, c.y, c.dtype, c.m, c.n, c.ldy, 32, "y")) return rc;
    mr = my;
    if (c.res != nullptr && (c.res != c.y || c.lres != c.ldy))
      if (int rc = matrix_map(&mr, c.res, c.dtype, c.m, c.n, c.lres, 32, "res")) return rc;
    const int form = c.scale != nullptr ? kPairScaled : c.res != nullptr ? kPairResidual : kPairPlain;
    const void* kernel = f16 ? pair_kernel<__half>(c.act, form) : pair_kernel<__nv_bfloat16>(c.act, form);
    const int smem = static_cast<int>(sizeof(PairSmem)) + 1024;
    if (int rc = opt_in(*dev, (pair_act_index(c.act) * 3 + form) * 2 + (f16 ? 0 : 1), kernel, smem)) return rc;
    void* args[] = {&mx, &mw, &mwt, &my, &mr, &prm};
    return launch_kernel(kernel, static_cast<unsigned>(2 * std::min<long long>(items, dev->sms / 2)), 1, kPairThreads, smem, 2, stream, args, "gemm kernel launch");
  }
  prm.tiles_m = (c.m + 127) / 128;
  prm.tiles_n = (c.n + kSplitBN - 1) / kSplitBN;
  if (int rc = matrix_map(&mw, c.w, c.dtype, w_rows, c.k, c.k, kSplitBN, "w")) return rc;
  const int s = plan.split;
  int i = 0;
  while (kSplits[i] != s) ++i;
  const SplitForm& form = split_forms()[i];
  const void* kernel = f16 ? form.f16 : form.bf16;
  const int smem = static_cast<int>(form.smem) + 1024;
  void* args[] = {&mx, &mw, &prm};
  return launch_kernel(kernel, static_cast<unsigned>(prm.tiles_m * prm.tiles_n * s), 1, kSplitThreads, smem, static_cast<unsigned>(s), stream, args, "gemm kernel launch");
}

namespace {

template <typename T, int NT>
const void* rel_kernel_at(bool rows) {
  if constexpr (NT <= 4 || NT == 8)  // sides rel_by_tokens() may choose
    if (!rows) return reinterpret_cast<const void*>(sam_rel_terms_kernel<T, NT>);
  return reinterpret_cast<const void*>(sam_rel_rows_kernel<T, NT>);
}
template <typename T>
const void* rel_kernel_of(int tiles, bool rows) {
  switch (tiles) {
    case 1: return rel_kernel_at<T, 1>(rows);
    case 2: return rel_kernel_at<T, 2>(rows);
    case 3: return rel_kernel_at<T, 3>(rows);
    case 4: return rel_kernel_at<T, 4>(rows);
    case 5: return rel_kernel_at<T, 5>(rows);
    case 6: return rel_kernel_at<T, 6>(rows);
    case 7: return rel_kernel_at<T, 7>(rows);
    default: return rel_kernel_at<T, 8>(rows);
  }
}
// Which of the three kernels; us ([images, heads, side]) by rows, by tokens and by lines.
// By lines (rows and addresses in whole 16-byte groups, heads to divide by) from side 48 on: [1,12,48] 7.6, 7.8, 7.1; [2,12,48] 10.8, 13.9,
// 11.5; [4,12,48] 19.7, 24.8, 16.0; [1,12,64] 12.0, 10.0, 7.6; [4,12,64] 27.5, 30.4, 22.5; [16,16,56] 178, 195, 87; [16,16,64] 99.7, 127, 105. At side 40
// where an SM has one line or at least four: [1,12,40] 6.5, 6.0, 5.9; [2,12,40] 7.9, 9.6, 9.3; [4,12,40] 12.3, 13.8, 12.9; [16,12,40] 39.5, 46, 35.1.
bool rel_by_lines(int side, long long lines, int sms) { return side >= 48 || (side >= 40 && (lines <= sms || lines >= 4LL * sms)); }
// Two CTAs fit an SM's shared memory with six tiles at a time: one loads while the other holds the tensor memory. us, eight at a
// time and the fewest even shares of at most six: [2,16,56] 17.4 and 14.6, [4,16,64] 37.3 and 30.1, [8,16,64] 66.7 and 53.6; at a line per SM there is
// nothing to overlap, [1,16,64] 9.5 and 10.6.
int rel_line_tiles(int tiles, long long lines, int sms) {
  const int most = lines <= sms ? kRelLineTiles : 6, passes = (tiles + most - 1) / most;
  return (tiles + passes - 1) / passes;
}
// By tokens up to side 32 and at 64 (whole 16-byte groups per row; in between its stores are pieces of four bytes, a sector each), and
// up to 13 CTAs per SM, by rows beyond: [25,12,14] 6.1 and 4.9, [50,16,14] 11.1 and 8.4, [64,12,14] 9.9 and 10.1, [100,12,14] 12.6 and
// 14.4, [400,12,14] 44 and 58; [32,12,20] 17.1 and 13.5, [64,12,20] 23.7 and 25.0; [8,12,32] 11.5 and 8.8, [16,12,32] 15.1 and 16.1; [4,12,44] 15.5 and
// 22.1; [4,12,62] 55 and 63; [1,1,64] 11.1 and 8.1, [4,1,64] 23.7 and 24.5.
bool rel_by_tokens(int side, long long ctas, int sms) { return (side <= 32 || side == 64) && ctas <= 13LL * sms; }

}  // namespace

int launch_rel_terms(const B200RelTermsArgs* a, bool early_tables, cudaStream_t stream) {
  if (a == nullptr) return fail(B200_ATTN_BAD_CONFIG, "args is NULL");
  if (a->struct_size != sizeof(B200RelTermsArgs))
    return fail(B200_ATTN_BAD_CONFIG, "struct_size %u does not match this library's B200RelTermsArgs (%zu bytes)",
                a->struct_size, sizeof(B200RelTermsArgs));
  if (a->dtype != B200_ATTN_F16 && a->dtype != B200_ATTN_BF16)
    return fail(B200_ATTN_BAD_CONFIG, "dtype %u: q, the tables and the results must be fp16 (0) or bf16 (1)", a->dtype);
  if (a->head_dim != kHeadDim) return fail(B200_ATTN_UNSUPPORTED, "head_dim %d: only head dim 64 is built", a->head_dim);
  if (a->batch < 1 || a->heads < 1 || a->side < 2 || a->side > kRelMaxSide || a->side % 2 != 0)
    return fail(B200_ATTN_UNSUPPORTED, "batch %d heads %d side %d: side must be even, 2 .. %d", a->batch, a->heads, a->side, kRelMaxSide);
  if (static_cast<int64_t>(a->batch) * a->side > 0x7fffffffLL) return fail(B200_ATTN_UNSUPPORTED, "batch too large for one launch");
  const int tokens = a->side * a->side;
  if (int rc = check_view("q", a->q, a->q_stride, a->batch, a->heads, tokens)) return rc;
  const struct { const char* name; const void* ptr; int align; } ptrs[] = {
      {"rel_pos_h", a->rel_pos_h, 4}, {"rel_pos_w", a->rel_pos_w, 4}, {"rel_h", a->rel_h, 4}, {"rel_w", a->rel_w, 4}};
  for (const auto& x : ptrs) {
    if (x.ptr == nullptr) return fail(B200_ATTN_BAD_CONFIG, "%s is NULL", x.name);
    if (reinterpret_cast<uintptr_t>(x.ptr) % x.align != 0) return fail(B200_ATTN_UNSUPPORTED, "%s is not 4-byte aligned", x.name);
  }
  RelTermsParams prm{};
  prm.q = a->q;
  prm.q_sb = a->q_stride[0];
  prm.q_sn = a->q_stride[1];
  prm.q_sh = a->q_stride[2];
  prm.rel_pos_h = a->rel_pos_h;
  prm.rel_pos_w = a->rel_pos_w;
  prm.rel_h = a->rel_h;
  prm.rel_w = a->rel_w;
  prm.batch = a->batch;
  prm.heads = a->heads;
  prm.side = a->side;
  prm.tables_wide = aligned16(a->rel_pos_h) && aligned16(a->rel_pos_w);
  prm.out_wide = aligned16(a->rel_h) && aligned16(a->rel_w);
  prm.early_tables = early_tables ? 1 : 0;
  DeviceState* dev = nullptr;
  if (int rc = device_state(&dev)) return rc;
  const bool f16 = a->dtype == B200_ATTN_F16;
  const long long lines = 2LL * a->batch * a->side;
  if (a->side % 8 == 0 && rel_by_lines(a->side, lines, dev->sms) && prm.tables_wide && prm.out_wide && a->heads > 1 && a->heads <= 1024 && lines <= 0x7fffffffLL) {
    prm.status = dev->status;
    prm.magic_heads = static_cast<uint32_t>((uint64_t(1) << 32) / static_cast<uint32_t>(a->heads) + 1);  // exact for 64 * heads rows
    prm.tiles = rel_line_tiles((a->side * a->heads + 127) / 128, lines, dev->sms);
    const void* kernel = f16 ? reinterpret_cast<const void*>(sam_rel_lines_kernel<__half>) : reinterpret_cast<const void*>(sam_rel_lines_kernel<__nv_bfloat16>);
    if (int rc = opt_in(*dev, kLinearKernels - (f16 ? 2 : 1), kernel, rel_lines_smem(kRelLineTiles))) return rc;
    void* args[] = {&prm};
    if (int rc = launch_kernel(kernel, static_cast<unsigned>(lines), 1, kRelLineThreads, rel_lines_smem(prm.tiles), 1, stream, args, "sam_rel_terms kernel launch")) return rc;
    clear_error();
    return B200_ATTN_OK;
  }
  const long long grid_rows = static_cast<long long>(a->batch) * a->side;
  prm.parts = (a->side + kRelWarps - 1) / kRelWarps;
  const bool rows = !rel_by_tokens(a->side, grid_rows * prm.parts, dev->sms);
  if (rows)  // one CTA per grid row, and several where there are few rows: about four CTAs per SM, a token per warp at least
    prm.parts = static_cast<int>(std::max(1LL, std::min<long long>((4LL * dev->sms + grid_rows - 1) / grid_rows, (a->side + kRelRowWarps - 1) / kRelRowWarps)));
  if (grid_rows * prm.parts > 0x7fffffffLL) return fail(B200_ATTN_UNSUPPORTED, "batch too large for one launch");
  const int tiles = (a->side + 7) / 8;
  const void* kernel = f16 ? rel_kernel_of<__half>(tiles, rows) : rel_kernel_of<__nv_bfloat16>(tiles, rows);
  void* args[] = {&prm};
  const int table_rows = rows ? 3 * a->side - 1 : 2 * a->side - 1 + (a->side + prm.parts - 1) / prm.parts;
  if (int rc = launch_kernel(kernel, static_cast<unsigned>(grid_rows * prm.parts), 1, (rows ? kRelRowWarps : kRelWarps) * 32, table_rows * 128, 1, stream, args, "sam_rel_terms kernel launch"))
    return rc;
  clear_error();
  return B200_ATTN_OK;
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200_gemm(const B200GemmArgs* a, void* stream_ptr) {
  if (a == nullptr) return fail(B200_ATTN_BAD_CONFIG, "args is NULL");
  if (a->struct_size != sizeof(B200GemmArgs))
    return fail(B200_ATTN_BAD_CONFIG, "struct_size %u does not match this library's B200GemmArgs (%zu bytes)", a->struct_size,
                sizeof(B200GemmArgs));
  if (a->dtype != B200_ATTN_F16 && a->dtype != B200_ATTN_BF16)
    return fail(B200_ATTN_BAD_CONFIG, "dtype %u: x, w, bias, res, y must be fp16 (0) or bf16 (1)", a->dtype);
  if (a->act != kActNone && a->act != kActRelu && a->act != kActGelu && a->act != kActGeluTanh)
    return fail(B200_ATTN_BAD_CONFIG, "act %d: 0 none, 1 relu, 5 gelu (erf), 6 gelu (tanh form)", a->act);
  if (a->m < 1 || a->n < 1 || a->k < 1 || a->n % 8 != 0 || a->k % 8 != 0)
    return fail(B200_ATTN_UNSUPPORTED, "m %d n %d k %d: all positive, n and k multiples of 8", a->m, a->n, a->k);
  if (a->lda < a->k || a->lda % 8 != 0 || a->ldy < a->n || a->ldy % 8 != 0 || (a->res != nullptr && (a->lres < a->n || a->lres % 8 != 0)))
    return fail(B200_ATTN_UNSUPPORTED, "row strides lda %lld ldy %lld lres %lld must cover their rows and be multiples of 8",
                static_cast<long long>(a->lda), static_cast<long long>(a->ldy), static_cast<long long>(a->lres));
  if (a->lda >= (int64_t(1) << 38) || a->ldy >= (int64_t(1) << 38) || (a->res != nullptr && a->lres >= (int64_t(1) << 38)))
    return fail(B200_ATTN_UNSUPPORTED, "a row stride is too large for a tensor map");
  const struct { const char* name; const void* ptr; bool required; } ptrs[] = {
      {"x", a->x, true}, {"w", a->w, true}, {"y", a->y, true}, {"bias", a->bias, false}, {"scale", a->scale, false}, {"res", a->res, false}};
  for (const auto& x : ptrs) {
    if (x.ptr == nullptr && x.required) return fail(B200_ATTN_BAD_CONFIG, "%s is NULL", x.name);
    if (!aligned16(x.ptr)) return fail(B200_ATTN_UNSUPPORTED, "%s is not 16-byte aligned", x.name);
  }
  const GemmCall call{a->dtype, a->m, a->n, a->k, a->act, a->x, a->lda, a->w, a->bias, a->scale, a->res, a->lres, a->y, a->ldy, false, false};
  if (int rc = launch_gemm(call, static_cast<cudaStream_t>(stream_ptr))) return rc;
  clear_error();
  return B200_ATTN_OK;
}

int b200_gemm_plan(int32_t m, int32_t n, int32_t k, int32_t sms, const int32_t* clusters, int32_t* plan) {
  if (m < 1 || n < 1 || k < 1 || sms < 0 || plan == nullptr || (sms > 0 && clusters == nullptr))
    return fail(B200_ATTN_BAD_CONFIG, "b200_gemm_plan: m %d n %d k %d sms %d, plan and (with sms) split_clusters not NULL", m, n, k, sms);
  int fit[kGemmSplits];
  if (sms > 0) {
    std::copy_n(clusters, kGemmSplits, fit);
  } else {
    DeviceState* dev = nullptr;
    if (int rc = device_state(&dev)) return rc;
    if (int rc = split_clusters(*dev)) return rc;
    for (int i = 0; i < kGemmSplits; ++i) fit[i] = dev->split_clusters[i].load(std::memory_order_relaxed);
    sms = dev->sms;
  }
  const GemmPlan p = gemm_plan(m, n, k, false, sms, fit);
  plan[0] = p.bn;
  plan[1] = p.split;
  plan[2] = p.tail_bn;
  clear_error();
  return B200_ATTN_OK;
}

int b200_sam_rel_terms(const B200RelTermsArgs* a, void* stream_ptr) { return launch_rel_terms(a, false, static_cast<cudaStream_t>(stream_ptr)); }

int b200_rope_qk(const B200RopeArgs* a, void* stream_ptr) {
  if (a == nullptr) return fail(B200_ATTN_BAD_CONFIG, "args is NULL");
  if (a->struct_size != sizeof(B200RopeArgs))
    return fail(B200_ATTN_BAD_CONFIG, "struct_size %u does not match this library's B200RopeArgs (%zu bytes)",
                a->struct_size, sizeof(B200RopeArgs));
  if (a->dtype != B200_ATTN_F16 && a->dtype != B200_ATTN_BF16)
    return fail(B200_ATTN_BAD_CONFIG, "dtype %u: q and k must be fp16 (0) or bf16 (1)", a->dtype);
  if (a->head_dim != kHeadDim) return fail(B200_ATTN_UNSUPPORTED, "head_dim %d: only head dim 64 is built", a->head_dim);
  if (a->batch < 1 || a->heads < 1 || a->tokens < 1 || a->prefix < 0 || a->prefix > a->tokens)
    return fail(B200_ATTN_BAD_CONFIG, "batch %d heads %d tokens %d prefix %d", a->batch, a->heads, a->tokens, a->prefix);
  if (!(a->q_scale > 0.f) || !std::isfinite(a->q_scale)) return fail(B200_ATTN_BAD_CONFIG, "q_scale must be positive and finite");
  if (int rc = check_view("q", a->q, a->q_stride, a->batch, a->heads, a->tokens)) return rc;
  if (int rc = check_view("k", a->k, a->k_stride, a->batch, a->heads, a->tokens)) return rc;
  if (a->prefix < a->tokens) {
    if (a->cs == nullptr) return fail(B200_ATTN_BAD_CONFIG, "cs is NULL");
    if (!aligned16(a->cs)) return fail(B200_ATTN_UNSUPPORTED, "cs is not 16-byte aligned");
  }
  DeviceState* dev = nullptr;
  if (int rc = device_state(&dev)) return rc;
  RopeParams prm{};
  prm.q = a->q;
  prm.k = a->k;
  prm.q_sb = a->q_stride[0];
  prm.q_sn = a->q_stride[1];
  prm.q_sh = a->q_stride[2];
  prm.k_sb = a->k_stride[0];
  prm.k_sn = a->k_stride[1];
  prm.k_sh = a->k_stride[2];
  prm.cs = a->cs;
  prm.batch = a->batch;
  prm.heads = a->heads;
  prm.tokens = a->tokens;
  prm.prefix = a->prefix;
  prm.q_scale = a->q_scale;
  void* args[] = {&prm};
  const void* kernel = a->dtype == B200_ATTN_F16 ? reinterpret_cast<const void*>(rope_qk_kernel<__half>) : reinterpret_cast<const void*>(rope_qk_kernel<__nv_bfloat16>);
  if (int rc = launch_kernel(kernel, static_cast<unsigned>(a->tokens), static_cast<unsigned>(std::min(a->batch, 65535)), kRopeThreads, 0, 1, static_cast<cudaStream_t>(stream_ptr), args, "rope_qk kernel launch")) return rc;
  clear_error();
  return B200_ATTN_OK;
}

}  // extern "C"
