// The attention kernel for few keys, as b200_attn_fwd calls it. Defined in b200_window.cu.
#pragma once

#include "../../include/b200_attn.h"
#include "host_common.h"

namespace b200 {

enum : int { kWindowCallPlain = 0, kWindowCallDense = 1, kWindowCallRel = 2 };
struct WindowCall {
  int bias;             // without, 16-bit dense with rows on 16 bytes, decomposed with tables of q's type and a scale whose inverse is exact in it
  bool batch_fastest;   // dense: every image has the same bias
  int rel_align;        // decomposed: bytes the rows of both tables begin on (16, 4 or 2)
  uint32_t rel_one;     // decomposed: 1 / scale, 16 bits
};
constexpr int kWindowCallMaxKeys = 128;  // no call with more keys goes there: nothing else needs to be looked at
// Whether a call that passed validation goes to the kernel, and the launch.
bool window_pays(const B200AttnArgs* a, const WindowCall& call, int sms);
int launch_window(const B200AttnArgs* a, const WindowCall& call, cudaStream_t stream);

}  // namespace b200
