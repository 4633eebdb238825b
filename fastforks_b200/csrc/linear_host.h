// Host side of the layers around attention: internal launch functions shared by the C entry points and the encoder
// forwards. All launch on `stream` of the current device and return a status code.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/b200_attn.h"

namespace b200 {

// One product with its epilogue (gemm_sm100.cuh). `n` counts the columns of y; a SwiGLU layer (act = kActSwiGlu) has
// 2 n rows of w and 2 n biases. early_w: see GemmParams.
struct GemmCall {
  uint32_t dtype;
  int m, n, k, act;
  const void* x;
  int64_t lda;
  const void* w;
  const void* bias;
  const float* scale;
  const void* res;
  int64_t lres;
  void* y;
  int64_t ldy;
  bool early_w;
  bool backwards;  // a hint: rows from the last to the first, so that what the kernel in front wrote last is read first
};
int launch_gemm(const GemmCall& c, cudaStream_t stream);

// b200_sam_rel_terms; early_tables: see RelTermsParams.
int launch_rel_terms(const B200RelTermsArgs* a, bool early_tables, cudaStream_t stream);

// How a product is cut: the pair kernel with tiles of 256 x bn, those behind the last whole round of the grid cut into
// parts of 256 x tail_bn if tail_bn > 0, or, split > 0, the split kernel with 128 x 64 tiles and the k range cut in `split`.
struct GemmPlan {
  int bn, split, tail_bn;
};
// `split_clusters`: for 1, 2, 3, 4, 6 and 8 CTAs, how many clusters of the split kernel run at once.
GemmPlan gemm_plan(int m, int n, int k, bool swiglu, int sms, const int* split_clusters);

}  // namespace b200
