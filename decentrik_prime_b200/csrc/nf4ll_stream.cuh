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
  int64_t split;                         // gate|up: rows of a half
  void* y2;                              // its second half's output
  int64_t ldy2;
  void* h;                               // silu(first half) * second half; null: not gate|up
  int64_t ldh;
  int n_seg;                             // projections stacked along N
  int64_t seg_end[kMaxSegments];         // first row after the segment
  const float* seg_t[kMaxSegments];      // [M, 16] fp32 rank-16 product of the segment, null: no LoRA
  const __half* seg_b[kMaxSegments];     // its lora_B, indexed by the row of W
  float seg_scale[kMaxSegments];
  int busy;                              // CTAs of the rank-16 projection launched right before, each on an SM for as long as that takes
  int withhold;                          // failure-detection hook
  uint32_t wait_us;
};

// What the kernel takes for M <= 16 tokens, behind other calls: a fit (nf4ll_stream.cu, stream_us). `busy`: CTAs of the rank-16 projection
// that the call launches before it, 0: none
double stream_time_us(int64_t M, int64_t N, int64_t K, bool gate_up, int busy);
// Whether the kernel takes M tokens, eight at a time, against weights of this size: rows as long as eight CTAs hold the tokens of them in
// registers, 43008 weights, and where a cluster of up to sixteen finds room, twice that
bool stream_takes(int64_t M, int64_t N, int64_t K, bool gate_up);
// `early`: the kernel launched right before on the stream is a rank-16 projection of the same call
int stream_forward_launch(const StreamCall& c, bool early, int force, int32_t* status, cudaStream_t stream);

int zero_words_launch(int* words, int n, cudaStream_t stream);      // nf4ll_lora.cu

}  // namespace nf4ll
