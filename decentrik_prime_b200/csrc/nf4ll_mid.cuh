// Middling batches (nf4ll_mid.cu): one call of the forward or of backward-dX.
#pragma once

#include "nf4ll_gemm_shared.cuh"

namespace nf4ll {

struct MidCall {
  int mode;                              // kFwd / kBwd
  const nf4ll_mat* W;
  const void* act;                       // x [M, K] or dy [M, N]
  int64_t ldact, M;
  const void* bias;                      // forward only, may be null
  void* out;
  int64_t ldo;
  int accumulate;                        // backward: out += result
  int n_seg;                             // projections stacked along N (1: one projection), row counts multiples of 128
  int64_t seg_end[kMaxSegments];         // first row after the segment
  const float* seg_left[kMaxSegments];   // [M, 16] fp32: T (forward) or s.U (backward), null: no LoRA
  const __half* seg_right[kMaxSegments]; // forward: lora_B indexed by the row of W; backward: A [16, K]
  float seg_scale[kMaxSegments];
  const uint8_t* mask;                   // backward: keep-mask of the LoRA input, may be null
  int64_t ld_mask;
  float keep_scale;
  int64_t gu_inter;                      // > 0: gate|up stacked, h = silu(g) * u from the epilogue
  void* out_u;
  int64_t ldu;
  void* out_h;
  int64_t ldh;
  int withhold;                          // failure-detection hook (nf4ll_test_mid_withhold), 0: off
  uint32_t wait_us;
};

// How a call is cut up. A unit is (128 * rb weight rows / output columns) x (nt tokens), worked on by one cluster.
struct MidPlan {
  int rb, nt, cl;              // row blocks of a unit, tokens of a unit, CTAs of a cluster (slices of the contraction)
  int tiles_o, tiles_t, units;
  int clusters;                // launched; units / clusters rounded up = units one after another in a cluster
  int nbuf, na, nx, nc;        // accumulators, slots of decoded weights, slots of token tiles, slots of codes
  bool x_alias;                // the exchange of partial sums reuses the operand rings
  bool split;                  // forward: the rank-16 product as two fp16 parts
  int64_t items;               // items of 128 x 128 weights that a CTA takes one after another
  double us;                   // expected time
};

// rb / nt / cl forced where not zero (tests). False: this kernel does not take the call.
bool mid_plan(int mode, int64_t M, int64_t NO, int64_t KC, bool mask, int64_t gu_inter, bool lora, int rb, int nt, int cl, MidPlan* plan);
int mid_clusters(int cl);    // clusters of `cl` CTAs that the current device holds at once
int64_t mid_searches();      // plans that the calling thread had to search for so far
int64_t mid_calls();         // calls of the thread that this kernel has taken
// `early`: the kernel launched right before on the stream is one of the same call that does not write act or the weight
int mid_launch(const MidCall& c, const MidPlan& p, bool early, int32_t* status, cudaStream_t stream);

}  // namespace nf4ll
