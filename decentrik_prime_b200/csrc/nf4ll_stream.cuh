// One call of the weight-streaming forward (nf4ll_stream.cu).
#pragma once

#include "nf4ll_gemm_shared.cuh"

namespace nf4ll {

struct StreamCall {
  const nf4ll_mat* W;
  const void* x;
  int64_t ldx, M;
  const void* bias;
  void* y;
  int64_t ldy;
  void* y2;                              // rows from `split` on go here, null: one output
  int64_t ldy2, split;
  int n_seg;                             // projections stacked along N
  int64_t seg_end[kMaxSegments];         // first row after the segment
  const float* seg_t[kMaxSegments];      // [M, 16] fp32 rank-16 product of the segment, null: no LoRA
  const __half* seg_b[kMaxSegments];     // its lora_B, indexed by the row of W
  float seg_scale[kMaxSegments];
};

// What the streaming kernel takes for M <= 16 tokens, up to the fixed cost of a launch: a fit through the times of five
// shapes from 3584 x 3584 to 27648 x 5120 at 1 to 16 tokens (0.6 us per block of the busiest warp, and the token rows).
double stream_time_us(int64_t N, int64_t K, int64_t M, int sms);
// `early`: the kernel launched right before on the stream is a rank-16 projection of the same call
int stream_forward_launch(const StreamCall& c, bool early, int force_team, cudaStream_t stream);

int zero_words_launch(int* words, int n, cudaStream_t stream);      // nf4ll_lora.cu

}  // namespace nf4ll
