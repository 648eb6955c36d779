// Standalone NF4 -> fp16 dequantisation: the launcher behind the k_nf4-compatible dequant_layer /
// dequant_range, and the weight pass in front of the large-batch GEMM (nf4ll_dense.cu).
// Replaces the reference's nf4_layer_dequant_kernel (solution/k_nf4.py:40-57).
//
// Memory-bound: 0.516 B read + 2 B written per weight. One thread decodes half a quantisation block (32 weights)
// per step: one 128-bit load of codes, coalesced across the warp, and two 256-bit stores, each a whole 32-byte
// sector (with four 128-bit stores per thread, 64 bytes apart across the warp, every store instruction touched 32
// half-written sectors). The 16 levels never touch memory: each thread builds the block's 16 fp16 products in
// registers and looks codes up with byte permutes. Operands are requested a step ahead. In a row of calls, with the table
// read before the wait, nothing requested ahead and eight CTAs per SM before / now: 8960 x 1536 7.1 / 7.4 us (the table's
// latency), 18944 x 3584 33.8 / 33.2, 27648 x 5120 69.2 / 68.2; with eight CTAs per SM 8.1 / 32.8 / 66.5, but a GEMM behind
// it starts later (backward of 1536 x 8960, 2048 rows: 70.2 us, 69.5 now).
#include "nf4ll_dequant.cuh"

namespace nf4ll {

constexpr int kDequantThreads = 256;
constexpr int kDequantCtas = 5;              // per SM, of up to 48 registers a thread: one wave

// ALIGNED: `out` starts on a 32-byte boundary. `side`: small jobs done on the way for the GEMM that follows.
template <bool ALIGNED>
__global__ void __launch_bounds__(kDequantThreads, kDequantCtas)
dequant_kernel(const uint4* __restrict__ nib, const uint8_t* __restrict__ qabs,
               const float* __restrict__ scale2, const float* __restrict__ offset2,
               const float* __restrict__ code2, int64_t n_half_blocks, uint4* __restrict__ out, const DequantSide side) {
  __shared__ float s_code2[256];
  pdl_wait();                  // before code2 too: whatever ran before this kernel may have written it
  pdl_launch_dependents();
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kDequantThreads;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kDequantThreads + threadIdx.x;
  // half a block's operands, requested a step ahead: the first ones travel together with code2
  uint4 codes = make_uint4(0, 0, 0, 0);
  uint32_t q = 0;
  float scale = 0.f, offset = 0.f;
  auto request = [&](int64_t h) {
    const int64_t qb = h >> 1;
    codes = __ldg(nib + h);
    q = __ldg(qabs + qb);
    scale = __ldg(scale2 + (qb >> 8));
    offset = __ldg(offset2 + (qb >> 8));
  };
  const float code2_mine = code2[threadIdx.x];
  if (first < n_half_blocks) request(first);
  for (int k = 0; k < side.n_left; ++k) {
    // the rank-16 left operand of the fused LoRA step, rounded as the in-kernel staging of the other GEMMs rounds it
    const float4* src = reinterpret_cast<const float4*>(side.left32[k]);
    uint2* dst = reinterpret_cast<uint2*>(side.left16 + static_cast<int64_t>(k) * side.left_elems);
    const float s = side.left_scale[k];
    for (int64_t i = first; i < side.left_elems / 4; i += stride) {
      const float4 v = src[i];
      dst[i] = make_uint2(pack_half2_rn(v.x * s, v.y * s), pack_half2_rn(v.z * s, v.w * s));
    }
  }
  s_code2[threadIdx.x] = code2_mine;
  __syncthreads();
  for (int64_t h = first; h < n_half_blocks; h += stride) {
    const uint4 c = codes;
    const float absmax = block_absmax(s_code2[q], scale, offset);
    if (h + stride < n_half_blocks) request(h + stride);
    const BlockTable t = make_block_table(absmax);
    uint4* dst = out + h * 4;
    if (ALIGNED) {
      store_sector(dst, decode_word(t, c.x), decode_word(t, c.y));
      store_sector(dst + 2, decode_word(t, c.z), decode_word(t, c.w));
    } else {
      dst[0] = decode_word(t, c.x);
      dst[1] = decode_word(t, c.y);
      dst[2] = decode_word(t, c.z);
      dst[3] = decode_word(t, c.w);
    }
  }
}

int dequant_launch(const uint8_t* nib, const uint8_t* qabs, const float* scale2, const float* offset2, const float* code2,
                   int64_t n_qblocks, void* out_f16, const DequantSide& side, cudaStream_t stream) {
  const int64_t n_half = n_qblocks * 2;
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int64_t blocks = (n_half + kDequantThreads - 1) / kDequantThreads;
  const int64_t cap = static_cast<int64_t>(sms) * kDequantCtas;      // one wave: the next kernel's blocks may then start early
  if (blocks > cap) blocks = cap;
  auto kernel = (reinterpret_cast<uintptr_t>(out_f16) & 31) ? dequant_kernel<false> : dequant_kernel<true>;
  PdlLaunch lc(dim3(static_cast<unsigned>(blocks)), dim3(kDequantThreads), 0, stream);
  NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, kernel, reinterpret_cast<const uint4*>(nib), qabs, scale2, offset2, code2, n_half,
                                reinterpret_cast<uint4*>(out_f16), side));
  return NF4LL_OK;
}

}  // namespace nf4ll

extern "C" int nf4ll_dequant(const uint8_t* nib, const uint8_t* qabs, const float* scale2, const float* offset2,
                             const float* code2, int64_t n_qblocks, void* out_f16, void* stream) {
  using namespace nf4ll;
  if (n_qblocks == 0) return NF4LL_OK;
  if (!nib || !qabs || !scale2 || !offset2 || !code2 || !out_f16) {
    set_detail("nf4ll_dequant: null pointer");
    return NF4LL_ERR_NULL;
  }
  if (n_qblocks < 0) {
    set_detail("nf4ll_dequant: n_qblocks=%lld", static_cast<long long>(n_qblocks));
    return NF4LL_ERR_SHAPE;
  }
  if ((reinterpret_cast<uintptr_t>(nib) & 15) || (reinterpret_cast<uintptr_t>(out_f16) & 15) ||
      (reinterpret_cast<uintptr_t>(scale2) & 3) || (reinterpret_cast<uintptr_t>(offset2) & 3)) {
    set_detail("nf4ll_dequant: nib/out must be 16-byte aligned, scale2/offset2 4-byte aligned");
    return NF4LL_ERR_ALIGN;
  }
  if (int rc = require_sm100()) return rc;
  return dequant_launch(nib, qabs, scale2, offset2, code2, n_qblocks, out_f16, DequantSide{}, static_cast<cudaStream_t>(stream));
}
