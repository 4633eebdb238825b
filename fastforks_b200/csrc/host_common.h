// Host-side helpers shared by the library's translation units: error reporting, per-device facts, TMA descriptor
// access. Defined in b200_attn.cu.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace b200 {

// Records the calling thread's error text and returns `code`.
int fail(int code, const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
void clear_error();

// cuTensorMapEncodeTiled, fetched through the runtime so that the library needs no link-time libcuda.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn();

// ceil(2^64 / d) for the attention kernels' fast_div; 0 stands for d <= 1.
inline uint64_t div_magic(int d) { return d <= 1 ? 0 : ~uint64_t(0) / static_cast<uint64_t>(d) + 1; }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Checks a [batch, tokens, heads, 64] view's pointer and strides against what the kernels take.
int check_view(const char* name, const void* ptr, const int64_t s[3], int batch, int heads, int tokens);

// What a launch needs to know about the current device, looked up once per device: the SM count, the address of the
// status word and which kernels already have their shared-memory opt-in (the opt-in is per device and per kernel).
// The runtime calls behind these cost more than the rest of the host path of a launch-bound call.
constexpr int kMaxDevices = 64;
constexpr int kKernelForms = 96;      // attention: 2 dtypes x 8 bias forms x (short, long) x (plain lists, twins, key split)
constexpr int kSmallForms = 16;      // attention of small calls: 2 dtypes x 8 key counts
constexpr int kLinearKernels = 32;    // of b200_linear.cu, with an opt-in: pair GEMM (5 activations x 3 epilogue forms x 2 dtypes), SAM's terms by lines (2 dtypes)
constexpr int kGemmSplits = 6;        // split counts of the split GEMM kernel
struct DeviceState {
  std::atomic<bool> ready{false};
  int sms = 0;
  uint32_t* status = nullptr;
  std::atomic<bool> opted_in[kKernelForms];
  std::atomic<bool> small_opted_in[kSmallForms];
  std::atomic<bool> linear_opted_in[kLinearKernels];
  std::atomic<bool> splits_ready;
  std::atomic<int> split_clusters[kGemmSplits];  // clusters of the split GEMM kernel that run at once
};
int device_state(DeviceState** out);

// Launch with programmatic stream serialisation (every kernel of this library waits on the device for the kernel
// before it, so its launch and set-up may overlap that kernel's tail), and optionally as clusters of `cluster` CTAs.
int launch_kernel(const void* kernel, unsigned grid_x, unsigned grid_y, unsigned threads, size_t smem, unsigned cluster,
                  cudaStream_t stream, void** args, const char* what);

}  // namespace b200
