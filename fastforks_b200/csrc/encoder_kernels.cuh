// The memory-bound kernels between an encoder's products: layer norms (with SAM's window partition and the residual of
// a windowed block folded in), patches and initial tokens, and the two norms of SAM's neck. One read and one write of
// each tensor, 16 bytes per thread and access, fp32 arithmetic, one rounding of the result.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

#include "sm100_ptx.cuh"

namespace b200 {

template <typename T>
__device__ __forceinline__ float2 enc_unpack2(uint32_t v) {
  if constexpr (std::is_same<T, __half>::value) return __half22float2(*reinterpret_cast<const __half2*>(&v));
  else return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ uint32_t enc_pack2(float lo, float hi) {
  if constexpr (std::is_same<T, __half>::value) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  } else {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
  }
}
template <typename T>
__device__ __forceinline__ void enc_unpack8(const uint4& v, float* f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 p = enc_unpack2<T>(w[i]);
    f[2 * i] = p.x;
    f[2 * i + 1] = p.y;
  }
}
template <typename T>
__device__ __forceinline__ uint4 enc_pack8(const float* f) {
  return make_uint4(enc_pack2<T>(f[0], f[1]), enc_pack2<T>(f[2], f[3]), enc_pack2<T>(f[4], f[5]), enc_pack2<T>(f[6], f[7]));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Square windows over a grid of tokens, zero-padded to whole windows: row r of the partitioned tensor is
// (image, window row, window column, row in the window, column in the window).
struct WindowMap {
  int side;            // window side; 0: no windows
  int grid_h, grid_w;  // tokens
  int per_row, per_col;  // windows per grid row and column
};

struct NormParams {
  const void* x;       // [tokens of all images, dim]
  void* x_out;         // with `delta`: the sum x + delta, may be x
  const void* delta;   // null, or what is added to x first: [rows, dim] in window order if map.side > 0, else in token order
  const void* weight;
  const void* bias;
  void* y;             // [rows, dim]; in window order if map.side > 0 and there is no delta
  int rows;            // rows of y
  int dim;
  float eps;
  int early_w;         // weight and bias were complete before the kernel in front started: read them ahead of the dependency wait
  WindowMap map;
};

// Token index of a row in window order, or -1 for a padding row.
__device__ __forceinline__ int token_of_window_row(const WindowMap& m, int r) {
  const int area = m.side * m.side;
  const int win = r / area, in = r - win * area;
  const int i = in / m.side, j = in - i * m.side;
  const int per_image = m.per_row * m.per_col;
  const int b = win / per_image, w = win - b * per_image;
  const int wy = w / m.per_row, wx = w - wy * m.per_row;
  const int y = wy * m.side + i, x = wx * m.side + j;
  return y < m.grid_h && x < m.grid_w ? (b * m.grid_h + y) * m.grid_w + x : -1;
}
__device__ __forceinline__ int window_row_of_token(const WindowMap& m, int t) {
  const int per_image = m.grid_h * m.grid_w;
  const int b = t / per_image, in = t - b * per_image;
  const int y = in / m.grid_w, x = in - y * m.grid_w;
  const int wy = y / m.side, i = y - wy * m.side, wx = x / m.side, j = x - wx * m.side;
  return (((b * m.per_col + wy) * m.per_row + wx) * m.side + i) * m.side + j;
}

constexpr int kNormWarps = 4;

template <typename T, int CHUNKS>
__device__ __forceinline__ void norm_row(const NormParams& p, int row, const uint4* raw, const uint4* weight, const uint4* bias, uint4* out, int lane) {
  float v[CHUNKS][8];
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) enc_unpack8<T>(raw[c], v[c]);
  if (p.delta != nullptr) {
    const int delta_row = p.map.side > 0 ? window_row_of_token(p.map, row) : row;
    const uint4* add = reinterpret_cast<const uint4*>(static_cast<const T*>(p.delta) + static_cast<int64_t>(delta_row) * p.dim);
    uint4* sum_out = reinterpret_cast<uint4*>(static_cast<T*>(p.x_out) + static_cast<int64_t>(row) * p.dim);
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (c * 256 + lane * 8 < p.dim) {
        float d[8];
        enc_unpack8<T>(add[c * 32 + lane], d);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[c][i] += d[i];
        const uint4 rounded = enc_pack8<T>(v[c]);
        sum_out[c * 32 + lane] = rounded;
        enc_unpack8<T>(rounded, v[c]);  // the norm sees the stored residual stream
      }
    }
  }
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
    for (int i = 0; i < 8; ++i) s += v[c][i];  // lanes past the end hold zeros
  const float mean = warp_sum(s) / static_cast<float>(p.dim);
  float q = 0.f;
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
    if (c * 256 + lane * 8 < p.dim) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[c][i] -= mean;
        q = fmaf(v[c][i], v[c][i], q);
      }
    }
  const float rstd = rsqrtf(warp_sum(q) / static_cast<float>(p.dim) + p.eps);
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    if (c * 256 + lane * 8 < p.dim) {
      float w[8], b[8];
      enc_unpack8<T>(weight[c * 32 + lane], w);
      enc_unpack8<T>(bias[c * 32 + lane], b);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[c][i] = fmaf(v[c][i] * rstd, w[i], b[i]);
      out[c * 32 + lane] = enc_pack8<T>(v[c]);
    }
  }
}

// One warp per row, the row in registers (CHUNKS x 8 values per lane): mean, then the variance of the differences.
// Bound by HBM at many rows and by a chain of latencies at few: weights and biases leave it, read into shared memory ahead
// of the dependency wait where they are older than the kernel in front. Inside a forward, 197 rows of 768 took 3.6 us and
// take 2.5, 5480 of 1024 6.9 and 5.4, 21920 of 1536 (135 MB, 21 us) 35.9 and 32.1. (Kept in registers they cost occupancy
// where rows are wide: 34.1. Several rows per warp with the next one in flight: 32.2, and 25 % more at 4900 rows of 768.)
template <typename T, int CHUNKS>
__global__ void __launch_bounds__(kNormWarps * 32) layer_norm_kernel(const NormParams p) {
  const int lane = threadIdx.x & 31;
  __shared__ uint4 weight[CHUNKS * 32], bias[CHUNKS * 32];
  const auto load_weights = [&] {
    for (int i = threadIdx.x; i < p.dim / 8; i += kNormWarps * 32) {
      weight[i] = static_cast<const uint4*>(p.weight)[i];
      bias[i] = static_cast<const uint4*>(p.bias)[i];
    }
  };
  if (p.early_w) load_weights();
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = blockIdx.x * kNormWarps + (threadIdx.x >> 5);
  int src = row < p.rows ? row : -1;
  if (p.map.side > 0 && p.delta == nullptr && src >= 0) src = token_of_window_row(p.map, row);
  uint4 raw[CHUNKS];
  const uint4* in = reinterpret_cast<const uint4*>(static_cast<const T*>(p.x) + static_cast<int64_t>(src) * p.dim);
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    raw[c] = make_uint4(0, 0, 0, 0);
    if (src >= 0 && c * 256 + lane * 8 < p.dim) raw[c] = in[c * 32 + lane];
  }
  if (!p.early_w) load_weights();
  __syncthreads();
  if (row >= p.rows) return;
  uint4* out = reinterpret_cast<uint4*>(static_cast<T*>(p.y) + static_cast<int64_t>(row) * p.dim);
  if (src < 0) {
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c)
      if (c * 256 + lane * 8 < p.dim) out[c * 32 + lane] = make_uint4(0, 0, 0, 0);
  } else {
    norm_row<T, CHUNKS>(p, row, raw, weight, bias, out, lane);
  }
}

struct TokensParams {
  const void* images;   // [batch, 3, height, width] contiguous; fp32 or the encoder's type
  int image_f32;
  int batch, height, width, patch;
  int grid_h, grid_w, prefix;  // tokens per image: prefix (class token) + grid_h * grid_w
  int k, k_padded;      // 3 * patch * patch, and the row stride of `patches`
  void* patches;        // [batch * tokens, k_padded]: one row of pixels per token (channel, row, column), zeros for prefix tokens
  const void* start;    // [tokens, dim], fp32 or the encoder's type: what the patch product is added to (position embedding) ...
  int start_f32;
  const void* patch_b;  // ... plus, for patch tokens, [dim] (patch bias) ...
  const void* first;    // ... and, for prefix tokens, [prefix, dim] (class token); either may be null
  void* x;              // [batch * tokens, dim]
  int dim;
};

constexpr int kTokensThreads = 256;
constexpr int kTokensRows = 4;    // pixel rows of one channel per block: as many loads of a thread in flight
constexpr int kTokensStarts = 4;  // blocks that copy the start values of a row of patches
constexpr int tokens_parts(int patch) { return kTokensStarts + 3 * ((patch + kTokensRows - 1) / kTokensRows); }

// The patch embedding is a convolution whose stride is its kernel: a product with the pixels of each patch as a row. This
// writes those rows and, for the product to be added to, the start values of the residual stream. Memory-bound; grid:
// (batch * grid_h rows of patches, tokens_parts(patch)), so that even one image keeps every SM's loads in flight: 13.9 us at
// one image of 1024 x 1024 and patches of 16 (one block per row and channel, a load at a time: 26.8), 12.1 at four of 518 x
// 518 and patches of 14 (13.4).
template <typename T>
__global__ void __launch_bounds__(kTokensThreads) encoder_tokens_kernel(const TokensParams p) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int b = blockIdx.x / p.grid_h, gy = blockIdx.x - b * p.grid_h;
  const int tokens = p.prefix + p.grid_h * p.grid_w;
  const int64_t first_row = static_cast<int64_t>(b) * tokens + p.prefix + static_cast<int64_t>(gy) * p.grid_w;
  const int part = static_cast<int>(blockIdx.y) - kTokensStarts;
  if (part >= 0) {
    const int groups = (p.patch + kTokensRows - 1) / kTokensRows;
    const int channel = part / groups, ky0 = (part - channel * groups) * kTokensRows;
    const int half_w = p.width >> 1;  // a pair of pixels never straddles a patch: the patch side is even
    const int used = (p.grid_w * p.patch) >> 1;
    const int64_t plane = (static_cast<int64_t>(b) * 3 + channel) * p.height + static_cast<int64_t>(gy) * p.patch + ky0;
    for (int px = threadIdx.x; px < used; px += kTokensThreads) {
      const int gx = (2 * px) / p.patch, kx = 2 * px - gx * p.patch;
      const int64_t from = plane * half_w + px;
      T* to = static_cast<T*>(p.patches) + (first_row + gx) * p.k_padded + (channel * p.patch + ky0) * p.patch + kx;
      uint32_t v[kTokensRows];
#pragma unroll
      for (int r = 0; r < kTokensRows; ++r) {
        if (ky0 + r >= p.patch) continue;
        if (p.image_f32) {
          const float2 f = __ldg(reinterpret_cast<const float2*>(p.images) + from + static_cast<int64_t>(r) * half_w);
          v[r] = enc_pack2<T>(f.x, f.y);
        } else {
          v[r] = __ldg(static_cast<const uint32_t*>(p.images) + from + static_cast<int64_t>(r) * half_w);
        }
      }
#pragma unroll
      for (int r = 0; r < kTokensRows; ++r)
        if (ky0 + r < p.patch) *reinterpret_cast<uint32_t*>(to + r * p.patch) = v[r];
    }
    return;
  }
  // start values of this row's tokens (with the image's first row of patches, of the prefix tokens too), zeros where a row of
  // `patches` holds no pixel: all of a prefix token's, and the padding
  const int slice = blockIdx.y;
  const int n0 = gy == 0 ? 0 : p.prefix + gy * p.grid_w, n1 = p.prefix + (gy + 1) * p.grid_w;
  const int vec = p.dim / 8;
  const uint4* start = static_cast<const uint4*>(p.start);
  uint4* x = static_cast<uint4*>(p.x) + static_cast<int64_t>(b) * tokens * vec;
  if (!p.start_f32 && p.patch_b == nullptr && p.first == nullptr) {
#pragma unroll 4
    for (int i = n0 * vec + slice * kTokensThreads + threadIdx.x; i < n1 * vec; i += kTokensStarts * kTokensThreads) x[i] = __ldg(start + i);
  } else {  // the sum in fp32, rounded once
#pragma unroll 2
    for (int i = n0 * vec + slice * kTokensThreads + threadIdx.x; i < n1 * vec; i += kTokensStarts * kTokensThreads) {
      const int n = i / vec;
      const uint4* add = static_cast<const uint4*>(n < p.prefix ? p.first : p.patch_b);
      float f[8], a[8];
      if (p.start_f32) {
        const float4 lo = __ldg(static_cast<const float4*>(p.start) + 2 * i), hi = __ldg(static_cast<const float4*>(p.start) + 2 * i + 1);
        f[0] = lo.x; f[1] = lo.y; f[2] = lo.z; f[3] = lo.w;
        f[4] = hi.x; f[5] = hi.y; f[6] = hi.z; f[7] = hi.w;
      } else {
        enc_unpack8<T>(__ldg(start + i), f);
      }
      if (add != nullptr) {
        enc_unpack8<T>(__ldg(add + (n < p.prefix ? i : i - n * vec)), a);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += a[e];
      }
      x[i] = enc_pack8<T>(f);
    }
  }
  if (slice != 0) return;
  T* rows = static_cast<T*>(p.patches) + static_cast<int64_t>(b) * tokens * p.k_padded;
  const T zero = T(0.f);
  if (gy == 0)
    for (int i = threadIdx.x; i < p.prefix * p.k_padded; i += kTokensThreads) rows[i] = zero;
  const int pad = p.k_padded - p.k;
  if (pad > 0)
    for (int i = threadIdx.x; i < p.grid_w * pad; i += kTokensThreads)
      static_cast<T*>(p.patches)[(first_row + i / pad) * p.k_padded + p.k + i % pad] = zero;
}

// A convolution's weights as the rows of a linear layer, in pairs of 16-bit values, a CTA per row: padded with zeros to a row
// of whole 16-byte groups (the patch embedding of patches of 14), or with the kernel's positions in front of the channels
// (the neck's 3 x 3, whose input rows are nine channel vectors). Done in every forward, on 1-2 MB, so that the convolution's
// own tensor is what a forward reads; a copy kept from the first one would not see that tensor change. With the start values
// summed in fp32 it adds 2.7 us to the 24.7 of patches, product and one norm at four images of 518 x 518 (1024 wide), 1.4 at one.
struct RepackParams {
  const void* src;  // [rows, cols]; taps > 0: [rows, cols / taps, taps]
  void* dst;        // [rows, out_cols], zeros from cols on; taps > 0: [rows, taps, cols / taps]
  int cols, out_cols;
  int taps;
};
constexpr int kRepackThreads = 256;
constexpr int kRepackMaxCols = 9 * 512;  // with taps: a row lies in shared memory

__global__ void __launch_bounds__(kRepackThreads) repack_kernel(const RepackParams p) {
  __shared__ uint32_t row[kRepackMaxCols / 2];
  grid_dependency_wait();
  grid_launch_dependents();
  const uint32_t* src = static_cast<const uint32_t*>(p.src) + static_cast<int64_t>(blockIdx.x) * (p.cols >> 1);
  uint32_t* dst = static_cast<uint32_t*>(p.dst) + static_cast<int64_t>(blockIdx.x) * (p.out_cols >> 1);
  if (p.taps == 0) {
    for (int i = threadIdx.x; i < p.out_cols >> 1; i += kRepackThreads) dst[i] = 2 * i < p.cols ? __ldg(src + i) : 0u;
    return;
  }
  for (int i = threadIdx.x; i < p.cols >> 1; i += kRepackThreads) row[i] = __ldg(src + i);
  __syncthreads();
  const uint16_t* values = reinterpret_cast<const uint16_t*>(row);
  const int channels = p.cols / p.taps;  // a multiple of eight: both values of a pair lie at one position
  for (int i = threadIdx.x; i < p.cols >> 1; i += kRepackThreads) {
    const int tap = 2 * i / channels, c = 2 * i - tap * channels;
    dst[i] = values[c * p.taps + tap] | static_cast<uint32_t>(values[(c + 1) * p.taps + tap]) << 16;
  }
}

// ---- SAM's neck -------------------------------------------------------------------------------------------------
// 1 x 1 convolution (a product), norm over the channels, 3 x 3 convolution (a product over nine shifted copies), norm,
// channels first.
struct NeckParams {
  const void* x;       // [batch * grid * grid, channels]
  const void* weight;
  const void* bias;
  void* out;           // im2col form: [batch * grid * grid, 9 * channels]; channels-first form: [batch, channels, grid * grid]
  int batch, grid_h, grid_w, channels;
  float eps;
};

constexpr int kNeckWarps = 8;
constexpr int kNeckChunks = 2;  // up to 512 channels
static_assert(kRepackMaxCols >= 9 * kNeckChunks * 256, "a row of the neck's 3 x 3 weights");

// The normalised row of one token per warp, in `v` (8 values per lane and chunk).
template <typename T>
__device__ __forceinline__ void neck_norm_row(const NeckParams& p, int64_t row, int lane, float v[kNeckChunks][8]) {
  const uint4* in = reinterpret_cast<const uint4*>(static_cast<const T*>(p.x) + row * p.channels);
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < kNeckChunks; ++c) {
    const bool here = c * 256 + lane * 8 < p.channels;
    enc_unpack8<T>(here ? in[c * 32 + lane] : make_uint4(0, 0, 0, 0), v[c]);
#pragma unroll
    for (int i = 0; i < 8; ++i) s += v[c][i];
  }
  const float mean = warp_sum(s) / static_cast<float>(p.channels);
  float q = 0.f;
#pragma unroll
  for (int c = 0; c < kNeckChunks; ++c)
    if (c * 256 + lane * 8 < p.channels) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[c][i] -= mean;
        q = fmaf(v[c][i], v[c][i], q);
      }
    }
  const float rstd = rsqrtf(warp_sum(q) / static_cast<float>(p.channels) + p.eps);
#pragma unroll
  for (int c = 0; c < kNeckChunks; ++c)
    if (c * 256 + lane * 8 < p.channels) {
      float w[8], b[8];
      enc_unpack8<T>(__ldg(static_cast<const uint4*>(p.weight) + c * 32 + lane), w);
      enc_unpack8<T>(__ldg(static_cast<const uint4*>(p.bias) + c * 32 + lane), b);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[c][i] = fmaf(v[c][i] * rstd, w[i], b[i]);
    }
}

// Norm, then the row goes to the nine output positions that read it: column block (ky, kx) of token (y - ky + 1,
// x - kx + 1). Blocks whose source lies outside the grid are zeros, written by the token they belong to.
template <typename T>
__global__ void __launch_bounds__(kNeckWarps * 32) neck_norm_im2col_kernel(const NeckParams p) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * kNeckWarps + (threadIdx.x >> 5);
  const int area = p.grid_h * p.grid_w;
  if (row >= static_cast<int64_t>(p.batch) * area) return;
  float v[kNeckChunks][8];
  neck_norm_row<T>(p, row, lane, v);
  const int in = static_cast<int>(row % area), y = in / p.grid_w, x = in - y * p.grid_w;
  const int64_t image = row - in;
  const int vec = p.channels / 8;
  uint4* out = static_cast<uint4*>(p.out);
#pragma unroll
  for (int c = 0; c < kNeckChunks; ++c) {
    if (c * 256 + lane * 8 >= p.channels) continue;
    const uint4 val = enc_pack8<T>(v[c]);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const int ky = k / 3, kx = k % 3;
      const int ty = y - ky + 1, tx = x - kx + 1;  // the token whose block k reads this row
      if (ty >= 0 && ty < p.grid_h && tx >= 0 && tx < p.grid_w) out[((image + ty * p.grid_w + tx) * 9 + k) * vec + c * 32 + lane] = val;
      const int sy = y + ky - 1, sx = x + kx - 1;  // what block k of this token reads
      if (sy < 0 || sy >= p.grid_h || sx < 0 || sx >= p.grid_w) out[(row * 9 + k) * vec + c * 32 + lane] = make_uint4(0, 0, 0, 0);
    }
  }
}

constexpr int kNeckTokens = 32;  // tokens per CTA of the channels-first form: 64 contiguous bytes per channel

// Norm, then channels first through shared memory.
template <typename T>
__global__ void __launch_bounds__(kNeckWarps * 32) neck_norm_chw_kernel(const NeckParams p) {
  extern __shared__ uint8_t neck_smem[];
  T* tile = reinterpret_cast<T*>(neck_smem);  // [channels][kNeckTokens + 2]
  grid_dependency_wait();
  grid_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int area = p.grid_h * p.grid_w;
  const int blocks_per_image = (area + kNeckTokens - 1) / kNeckTokens;
  const int b = blockIdx.x / blocks_per_image, t0 = (blockIdx.x - b * blocks_per_image) * kNeckTokens;
  const int count = min(kNeckTokens, area - t0);
  for (int t = warp; t < count; t += kNeckWarps) {
    float v[kNeckChunks][8];
    neck_norm_row<T>(p, static_cast<int64_t>(b) * area + t0 + t, lane, v);
#pragma unroll
    for (int c = 0; c < kNeckChunks; ++c)
      if (c * 256 + lane * 8 < p.channels) {
#pragma unroll
        for (int i = 0; i < 8; ++i) tile[(c * 256 + lane * 8 + i) * (kNeckTokens + 2) + t] = T(v[c][i]);
      }
  }
  __syncthreads();
  T* out = static_cast<T*>(p.out);
  for (int ch = warp; ch < p.channels; ch += kNeckWarps)
    if (lane < count) out[(static_cast<int64_t>(b) * p.channels + ch) * area + t0 + lane] = tile[ch * (kNeckTokens + 2) + lane];
}

}  // namespace b200
