// The rank-16 row reductions (nf4ll_lora.cu) as other files of the library launch them.
#pragma once

#include "nf4ll_common.cuh"

namespace nf4ll {

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// 16 bytes global -> shared, or 16 zero bytes when `valid` is false (src must still be an address)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// An 8 x 8 block of 16-bit values, a row in four lanes: transposed
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
// two values as fp16 pairs hi + lo: 22 bits of each, of which those below 2^-24 are rounded away; values beyond fp16's range become NaN
__device__ __forceinline__ void split_half2(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_half2_rn(a, b);
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  lo = pack_half2_rn(a - f.x, b - f.y);
}

// Two values as N fp16 pairs of descending weight: 11 bits each, of which those below 2^-24 are rounded away. An infinity lies in the first.
template <int N>
__device__ __forceinline__ void split_parts(float a, float b, uint32_t (&p)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) {
    p[i] = pack_half2_rn(a, b);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&p[i]));
    a = fabsf(f.x) <= 65504.f ? a - f.x : 0.f;
    b = fabsf(f.y) <= 65504.f ? b - f.y : 0.f;
  }
}
// For the sixteen ranks of a row, of which this lane has four and `m` is the largest of them by magnitude (the others' lie in the three
// lanes beside it): the power of two that brings the row's largest to [2^14, 2^15), so that parts keep the bits of ranks far below it,
// and its reciprocal. Both are normal: a row below 2^-112 is brought to less, but then all its bits lie above 2^-24.
struct RowScale {
  float to, back;
};
__device__ __forceinline__ RowScale row_scale(float m) {
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
  int e = static_cast<int>(__float_as_uint(m) >> 23) - 127;
  e = e < -112 ? -112 : e;
  return RowScale{__uint_as_float(static_cast<uint32_t>(127 + 14 - e) << 23), __uint_as_float(static_cast<uint32_t>(127 - 14 + e) << 23)};
}

struct DownBranch {
  const uint8_t* mask;      // keep-mask of the activation, may be null
  int64_t ld_mask;
  float keep_scale;
  const __half* R;          // [16, C]
  float* t32;               // [M, 16]
};

// CTAs of the launch below for n branches of at most sixteen rows
int lora_down_ctas(int64_t M, int64_t C, int n, int sms);

// one or two branches over the same rows
int lora_down_launch(const void* act, int64_t ldact, const DownBranch* br, int n, float scale, int64_t M, int64_t C, int* zero_ptr, int zero_words,
                     cudaStream_t stream);
int lora_down_launch(const void* act, int64_t ldact, const uint8_t* mask, int64_t ld_mask, float keep_scale, const void* R, float scale, int64_t M,
                     int64_t C, void* t32, int* zero_ptr, int zero_words, cudaStream_t stream);

}  // namespace nf4ll
