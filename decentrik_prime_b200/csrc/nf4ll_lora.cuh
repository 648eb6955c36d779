// The rank-16 row reductions (nf4ll_lora.cu) as other files of the library launch them.
#pragma once

#include "nf4ll_common.cuh"

namespace nf4ll {

struct DownBranch {
  const uint8_t* mask;      // keep-mask of the activation, may be null
  int64_t ld_mask;
  float keep_scale;
  const __half* R;          // [16, C]
  float* t32;               // [M, 16]
};

// one or two branches over the same rows
int lora_down_launch(const void* act, int64_t ldact, const DownBranch* br, int n, float scale, int64_t M, int64_t C, int* zero_ptr, int zero_words,
                     cudaStream_t stream);
int lora_down_launch(const void* act, int64_t ldact, const uint8_t* mask, int64_t ld_mask, float keep_scale, const void* R, float scale, int64_t M,
                     int64_t C, void* t32, int* zero_ptr, int zero_words, cudaStream_t stream);

}  // namespace nf4ll
