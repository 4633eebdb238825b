/*
 * b200_encoder.h - whole-encoder entry points of libb200attn.so: the blocks of a ViT (DINOv2 / timm family) or of SAM's
 * image encoder as one call that launches every kernel of the forward on one stream.
 *
 * Conventions are those of b200_attn.h: plain pointers and sizes, every buffer is the caller's, nothing is allocated and
 * nothing synchronises, the return value is a status code. All tensors are of `dtype` and contiguous, pointers 16-byte
 * aligned.
 */
#ifndef B200_ENCODER_H_
#define B200_ENCODER_H_

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

#define B200_FFN_GELU_TANH 0 /* fc1, GELU (tanh form), fc2 */
#define B200_FFN_SWIGLU 1    /* w12 [2 * hidden, dim] (gate rows, then value rows), silu(gate) * value, w3 */
#define B200_FFN_GELU 2      /* fc1, GELU (erf), fc2 */

/* Parameters of one block; linear weights in the nn.Linear layout [out, in]. */
typedef struct B200EncoderBlock {
  const void* norm1_w;
  const void* norm1_b;
  const void* qkv_w;
  const void* qkv_b;
  const void* proj_w;
  const void* proj_b;
  const float* gamma1; /* LayerScale [dim] or NULL */
  const void* norm2_w;
  const void* norm2_b;
  const void* fc1_w;
  const void* fc1_b;
  const void* fc2_w;
  const void* fc2_b;
  const float* gamma2;
  const void* rel_pos_h; /* SAM: [2 * side - 1, 64] tables of the decomposed bias, or NULL */
  const void* rel_pos_w;
  int32_t window; /* SAM: window side, 0 = global attention */
  int32_t reserved;
} B200EncoderBlock;

/* A normalised copy of the tokens after block `after` (0-based; -1: of the input tokens). */
typedef struct B200EncoderTap {
  int32_t after;
  int32_t reserved;
  void* out; /* [batch * tokens, dim] */
} B200EncoderTap;

/*
 * x <- block_{n-1}( ... block_0(x)):  x += gamma1 * proj(attention(qkv(norm1(x)))), x += gamma2 * ffn(norm2(x)).
 * With `images` the residual stream starts as start + patches * patch_w^T (one row of `start` per token; position
 * embedding, patch bias and class token folded in), else x is read as given.
 */
typedef struct B200EncoderArgs {
  uint32_t struct_size; /* sizeof(B200EncoderArgs) */
  uint32_t dtype;       /* B200_ATTN_F16 or B200_ATTN_BF16 */
  int32_t batch;
  int32_t grid_h; /* patches */
  int32_t grid_w;
  int32_t prefix; /* tokens in front of the patches (class token); 0 for SAM */
  int32_t dim;    /* heads * 64 */
  int32_t heads;
  int32_t hidden; /* a multiple of 8 */
  int32_t ffn;    /* B200_FFN_* */
  float eps;
  int32_t n_blocks;
  const B200EncoderBlock* blocks; /* host memory */
  const void* images;             /* [batch, 3, grid_h * patch.., grid_w * patch..] or NULL */
  uint32_t image_dtype;           /* B200_ATTN_F32 or `dtype` */
  int32_t height;
  int32_t width;
  int32_t patch;         /* even */
  const void* patch_w;   /* [dim, patch_k]: (channel, row, column) of the kernel, zeros up to patch_k */
  int32_t patch_k;       /* 3 * patch * patch rounded up to a multiple of 8 */
  int32_t n_taps;
  const void* start;     /* [prefix + grid_h * grid_w, dim] */
  void* x;               /* [batch * tokens, dim]; NULL with `images`: the residual stream lives in the workspace */
  const void* norm_w;    /* final norm, for taps */
  const void* norm_b;
  const B200EncoderTap* taps; /* host memory, in the order of `after` */
  void* workspace;            /* b200_encoder_workspace() bytes, 256-byte aligned, contents do not matter */
  int64_t workspace_bytes;
  void* attn_workspace;       /* B200AttnArgs::workspace */
  int64_t attn_workspace_bytes;
  /* SAM's neck (NULL neck_w0: none): 1 x 1 convolution to `neck_channels`, norm, 3 x 3 convolution, norm, channels first */
  const void* neck_w0; /* [channels, dim] */
  const void* neck_n0_w;
  const void* neck_n0_b;
  const void* neck_w1; /* [channels, 9 * channels]: (kernel row, kernel column, channel) */
  const void* neck_n1_w;
  const void* neck_n1_b;
  void* neck_out; /* [batch, channels, grid_h, grid_w] */
  int32_t neck_channels;
  float neck_eps;
  /* Parameters as a model holds them, so that a forward reads the model's own tensors and no prepared copies (all 0 / NULL:
   * the prepared forms above) */
  const void* patch_b;  /* [dim], added to the start of every patch token, or NULL */
  const void* first;    /* [prefix, dim], added to the start of the prefix tokens (class token), or NULL */
  int32_t start_f32;    /* start is fp32 */
  int32_t patch_w_raw;  /* patch_w is [dim, 3 * patch * patch], without the columns up to patch_k */
  int32_t neck_w1_conv; /* neck_w1 is [channels, channels, 3, 3]: (channel, kernel row, kernel column) */
  int32_t reserved;
} B200EncoderArgs;

/* Bytes of workspace a call with these sizes needs (pointers are not looked at, except `blocks` for the windows and
 * whether `images`, `x` and `neck_w0` are NULL). */
int b200_encoder_workspace(const B200EncoderArgs* args, int64_t* bytes);
int b200_encoder_forward(const B200EncoderArgs* args, void* stream);

#ifdef __cplusplus
}
#endif

#endif /* B200_ENCODER_H_ */
