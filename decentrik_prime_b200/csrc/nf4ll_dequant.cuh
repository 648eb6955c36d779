// The dequantisation pass and the small jobs it does for the GEMM launched behind it.
#pragma once

#include "nf4ll_common.cuh"

namespace nf4ll {

struct DequantSide {
  int n_left;                  // rank-16 products to round: left16[k] = fp16(left_scale[k] * left32[k])
  int64_t left_elems;          // elements of each (M * 16)
  const float* left32[4];
  float left_scale[4];
  __half* left16;
};

int dequant_launch(const uint8_t* nib, const uint8_t* qabs, const float* scale2, const float* offset2, const float* code2,
                   int64_t n_qblocks, void* out_f16, const DequantSide& side, cudaStream_t stream);

}  // namespace nf4ll
