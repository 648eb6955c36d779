// Parameters and plan of the large-batch GEMM over dequantised weights (nf4ll_dense.cu).
#pragma once

#include "nf4ll_pair.cuh"

namespace nf4ll {

struct DenseMaps {
  CUtensorMap act;                   // activation [M, KC], boxes of 128 rows x 64
  CUtensorMap w;                     // fp16 weight [N, K], boxes of 128 rows x 64 (forward) / 64 rows x 64 (backward)
  CUtensorMap out, out_u, out_h;     // results [M, NO], boxes of 32 rows x 64; gate|up: g, u, h
  CUtensorMap left;                  // rank-16 left operands [n_lora * M, 16] fp16, boxes of 128 rows x 8
  CUtensorMap right[kMaxSegments];   // forward: lora_B [rows, 16] of a segment, boxes 128 x 8; backward: lora_A [16, K], boxes 16 x 64
};

struct DenseParams {
  int64_t M, NO;
  __half* out;                       // [M, NO]
  int64_t ldo;
  int nkb;                           // 64-wide steps of the contraction
  int tiles_m, tiles_o;              // 512-row and 256-column (gate|up: 128 + 128) blocks
  int first_tile, end_tile;          // of this launch
  const __half* bias;
  int accumulate;                    // backward: out += result
  int n_lora;                        // rank-16 branches in maps.left
  int lora_index[kMaxSegments];      // segment -> block of maps.left, or -1
  int n_seg;                         // forward over stacked projections, 0: one projection
  int64_t seg_begin[kMaxSegments], seg_rows[kMaxSegments];
  int64_t gu_inter;                  // gate|up: columns of each half, else 0
  const uint8_t* mask;               // backward: keep-mask of the LoRA input [M, ld_mask], may be null
  int64_t ld_mask;
  float keep_scale;
  int32_t* status;
};

struct DensePlan {
  int nkb, parts;                    // parts: of each tile of the second launch
  int64_t tiles, tiles_m, tiles_o, whole;      // whole: tiles of the first launch, the others are cut
};

// What cutting tiles costs, in k-blocks of time (nf4ll_dense.cu)
constexpr int kDnExchange(int parts) { return 7 + 2 * parts; }
constexpr int kDnSecondLaunch = 8;

DensePlan dense_plan(int64_t M, int64_t NO, int64_t KC, int64_t gu_inter, int sms);
int dense_launch(int mode, const DenseMaps& maps, const DenseParams& p, const DensePlan& d, int sms, cudaStream_t stream);

}  // namespace nf4ll
