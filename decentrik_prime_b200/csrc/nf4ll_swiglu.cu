// SiLU-gated product between the up and down projections, forward and backward, fp32 math on fp16
// tensors: the step that sits between two calls of the fused linear in an MLP block.
// Same arithmetic as the reference's gated_silu_fwd/bwd kernels (solution/k_mlp.py:21-47):
//   h      = fp16( g / (1 + exp(-g)) * u )
//   d up   = dh * silu(g),   d gate = (dh * u) * sig * (1 + g * (1 - sig))
// Bandwidth-bound: 8 fp16 per thread per 128-bit access, grid-stride over [M, I].
#include "nf4ll_lora.cuh"

namespace nf4ll {

// Both kernels are one pass at memory speed: a thread takes several 16-byte chunks per trip, all loads of the trip issued before the
// arithmetic, so that every SM keeps enough bytes in flight. T: how wide a chunk's number is (its row comes out of a division, which
// took a good part of a trip in 64 bits). us at 16384 x 18944 / 2048 x 8960 / 951 x 8960 / 187 x 8960, operands
// out of HBM, with two chunks per trip and 64-bit divisions for all and now: backward 479 / 30.9 / 15.5 / 4.6 and 480 / 30.0 / 15.1 / 4.1, forward 347 /
// 22.8 / 11.4 / 3.3 and 305 / 19.9 / 9.8 / 3.0.
template <typename T, int U>
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __half* __restrict__ g, int64_t ldg, const __half* __restrict__ u, int64_t ldu,
                  __half* __restrict__ h, int64_t ldh, T total, T chunks_per_row) {
  pdl_wait();
  pdl_launch_dependents();
  const T stride = static_cast<T>(gridDim.x) * 256;
  for (T i = static_cast<T>(blockIdx.x) * 256 + threadIdx.x; i < total; i += U * stride) {
    uint4 gv[U], uv[U];
    int64_t at[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const T j = i + k * stride < total ? i + k * stride : i;
      const T row = j / chunks_per_row;
      const int64_t col = static_cast<int64_t>(j - row * chunks_per_row) * 8;
      gv[k] = __ldcs(reinterpret_cast<const uint4*>(g + row * ldg + col));
      uv[k] = __ldcs(reinterpret_cast<const uint4*>(u + row * ldu + col));
      at[k] = row * ldh + col;
    }
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (k == 0 || i + k * stride < total) *reinterpret_cast<uint4*>(h + at[k]) = swiglu_fwd8(gv[k], uv[k]);
  }
}

// dg / du may alias g / u (in-place, as the reference overwrites [gate | up]): a chunk is read in
// full before it is written, by the same thread.
template <typename T, int U>
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __half* g, int64_t ldg, const __half* u, int64_t ldu, const __half* __restrict__ dh, int64_t lddh,
                  __half* dg, int64_t lddg, __half* du, int64_t lddu, T total, T chunks_per_row) {
  pdl_wait();
  pdl_launch_dependents();
  const T stride = static_cast<T>(gridDim.x) * 256;
  for (T i = static_cast<T>(blockIdx.x) * 256 + threadIdx.x; i < total; i += U * stride) {
    uint4 gv[U], uv[U], dv[U];
    int64_t row[U], col[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const T j = i + k * stride < total ? i + k * stride : i;
      const T r = j / chunks_per_row;
      row[k] = r;
      col[k] = static_cast<int64_t>(j - r * chunks_per_row) * 8;
      gv[k] = *reinterpret_cast<const uint4*>(g + row[k] * ldg + col[k]);
      uv[k] = *reinterpret_cast<const uint4*>(u + row[k] * ldu + col[k]);
      dv[k] = __ldcs(reinterpret_cast<const uint4*>(dh + row[k] * lddh + col[k]));
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (k > 0 && i + k * stride >= total) break;
      uint4 og, ou, oh;
      swiglu_bwd8(gv[k], uv[k], dv[k], og, ou, oh);
      *reinterpret_cast<uint4*>(dg + row[k] * lddg + col[k]) = og;
      *reinterpret_cast<uint4*>(du + row[k] * lddu + col[k]) = ou;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The backward with what LoRA branches on gate, up and down take from [M, I] matrices: the rank-16 products of dg and du with
// lora_B (a sum over columns) and the gradients dB_gate, dB_up and dA_down (sums over rows of dg, du and drop(h), h formed anew from g
// and u, bit for bit as the forward forms it). Each of these as a kernel of its own reads its matrix again: 6 B per element
// for the gradients and 4 B for the products, against the 11 B that this pass moves at all (mask included).
// A CTA is four warps of 32 columns each and goes down a range of rows in stages of sixteen; g, u, dh and the mask come through a
// ring of two stages (cp.async, a warp its own part), the three rank-16 sides in two fp16 parts that the CTA's threads make once per
// stage. A warp forms dg, du and h from shared memory, stores dg and du, feeds them to the product's MMAs as they are (a lane's eight
// columns are the same k slots on both operands) and puts dg, du and h back in place, from where ldmatrix.trans reads them with the
// rows as k: side^T . d. The gradients stay in registers (48 per lane) for all of the range and are added to memory once, by atomics:
// their order is not fixed. The products of the four warps meet in shared memory (one barrier per stage) and go to a part per CTA
// column, which a second kernel adds up in order.
// Four CTAs of 128 registers per SM. No unit is full (at 2048 rows of 8960: shared memory 60 %, issue 43 %, HBM 35 %): what counts is how many
// warps stand in for each other, and how few meet at a barrier. Both kernels, 2048 / 512 rows of 8960: 63.7 / 24.2 us with 64 columns per
// warp (eight warps per SM, 244 registers), 65.7 / 23.3 with eight warps of 32 columns per CTA, 57.3 / 21.4 so; the kernels that it
// replaces (the gated backward, two products and the three reductions) took 115 in the step of an MLP block. The whole step, 1536 x 8960:
// 88.5 -> 69.9 us with 8 tokens, 168 -> 139 with 333, 535 -> 459 with 2048.
// ---------------------------------------------------------------------------------------------
constexpr int kGatedWarps = 4;
constexpr int kGatedThreads = kGatedWarps * 32;
constexpr int kGatedCols = kGatedWarps * 32;       // per CTA
constexpr int kGatedRows = 16;
constexpr int kGatedAct = kGatedRows * 64;         // a warp's part of g, u or dh: rows of 64 B, 16-byte pieces XORed with the row pair
constexpr int kGatedWarpStage = 3 * kGatedAct + kGatedRows * 32;
constexpr int kGatedStage = kGatedWarps * kGatedWarpStage;
constexpr int kGatedSideRow = 48;                  // sixteen ranks in fp16, rows apart so that ldmatrix finds eight of them on distinct banks
constexpr int kGatedSide = kGatedRows * kGatedSideRow;
constexpr int kGatedSides = 6 * kGatedSide;        // three sides in two parts each
constexpr int kGatedPartRow = 36;                  // a fragment's writes fall on distinct banks
constexpr int kGatedPart = kGatedRows * kGatedPartRow;
constexpr int kGatedSmem = 2 * (kGatedStage + kGatedSides + kGatedWarps * kGatedPart * 4);
static_assert(4 * (kGatedSmem + 1024) <= 228 * 1024, "four CTAs per SM");

struct GatedParams {
  const __half *g, *u, *dh;
  __half *dg, *du;
  int64_t ldg, ldu, lddh, lddg, lddu;
  const uint8_t* mask;
  int64_t ld_mask;
  float keep_scale;
  const float* side[3];                            // t_gate, t_up, u_down
  const __half* Rt[2];                             // lora_B of gate and of up transposed
  float* grad[3];                                  // dB_gate, dB_up, dA_down
  float scale[2];
  float* part;                                     // [CTA columns, M, 32]
  int64_t M, I, rows_per;
};

__global__ void __launch_bounds__(kGatedThreads, 4)
gated_bwd_kernel(const __grid_constant__ GatedParams p) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(16) uint8_t g_smem[];
  const uint32_t base = smem_u32(g_smem);
  uint8_t* const side_smem = g_smem + 2 * kGatedStage;
  float* const part = reinterpret_cast<float*>(side_smem + 2 * kGatedSides);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane >> 2, t = lane & 3;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * kGatedCols + warp * 32;
  const int64_t c = c0 + t * 8;                    // this lane's eight columns, of rows r and r + 8
  const int64_t r_begin = static_cast<int64_t>(blockIdx.y) * p.rows_per;
  const int64_t r_end = r_begin + p.rows_per < p.M ? r_begin + p.rows_per : p.M;
  const bool in = c < p.I;
  const uint32_t piece = warp * kGatedWarpStage + r * 64 + ((t ^ (r >> 1)) << 4);      // of row r; 512 B on, of row r + 8

  // rows r0 .. r0 + 15 of g, u, dh and the mask: a warp its own columns
  auto issue = [&](int64_t r0, int slot) {
    const uint32_t to = base + slot * kGatedStage + piece;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t m = r0 + r + 8 * h;
      const bool ok = in && m < r_end;
      cp_async16(to + h * 512, ok ? p.g + m * p.ldg + c : p.g, ok);
      cp_async16(to + h * 512 + kGatedAct, ok ? p.u + m * p.ldu + c : p.u, ok);
      cp_async16(to + h * 512 + 2 * kGatedAct, ok ? p.dh + m * p.lddh + c : p.dh, ok);
    }
    if (p.mask) {
      const int64_t m = r0 + (lane >> 1), cm = c0 + (lane & 1) * 16;
      const bool ok = cm < p.I && m < r_end;
      cp_async16(base + slot * kGatedStage + warp * kGatedWarpStage + 3 * kGatedAct + lane * 16, ok ? p.mask + m * p.ld_mask + cm : p.mask, ok);
    }
    cp_async_commit();
  };
  // the sides of rows r0 .. r0 + 15, a piece of four ranks at a time: t_gate in threads 0 .. 63, t_up in the others, u_down in the first again
  const int half = threadIdx.x >> 6, side_row = threadIdx.x >> 2 & 15, side_rank = (threadIdx.x & 3) * 4;
  struct Pieces { float4 a, b; };
  auto fetch = [&](int64_t r0) {
    const int64_t m = r0 + side_row, at = m * 16 + side_rank;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    return Pieces{m < r_end ? __ldcg(reinterpret_cast<const float4*>((half ? p.side[1] : p.side[0]) + at)) : zero,
                  m < r_end && half == 0 ? __ldcg(reinterpret_cast<const float4*>(p.side[2] + at)) : zero};
  };
  auto put_piece = [&](const float4& f, int buf, int which) {
    uint8_t* const to = side_smem + buf * kGatedSides + which * 2 * kGatedSide + side_row * kGatedSideRow + side_rank * 2;
    uint2 hi, lo;
    split_half2(f.x, f.y, hi.x, lo.x);
    split_half2(f.z, f.w, hi.y, lo.y);
    *reinterpret_cast<uint2*>(to) = hi;
    *reinterpret_cast<uint2*>(to + kGatedSide) = lo;
  };
  auto put = [&](const Pieces& f, int buf) {
    put_piece(f.a, buf, half);
    if (half == 0) put_piece(f.b, buf, 2);
  };

  issue(r_begin, 0);
  put(fetch(r_begin), 0);
  // lora_B of this lane's columns: ranks r and r + 8
  uint4 ra[2], rb[2];
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
    ra[b] = in ? __ldg(reinterpret_cast<const uint4*>(p.Rt[b] + r * p.I + c)) : zero;
    rb[b] = in ? __ldg(reinterpret_cast<const uint4*>(p.Rt[b] + (r + 8) * p.I + c)) : zero;
  }
  float acc[3][4][4];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int n = 0; n < 4; ++n) acc[a][n][0] = acc[a][n][1] = acc[a][n][2] = acc[a][n][3] = 0.f;
  cp_async_wait<0>();
  __syncthreads();
  int buf = 0;
  for (int64_t r0 = r_begin; r0 < r_end; r0 += kGatedRows) {
    issue(r0 + kGatedRows, buf ^ 1);               // past the range: empty, zero-filled
    const Pieces side = fetch(r0 + kGatedRows);
    uint8_t* const st = g_smem + buf * kGatedStage;
    float prod[2][2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {                  // rows 8 h + r
#pragma unroll
      for (int b = 0; b < 2; ++b) prod[b][h][0] = prod[b][h][1] = prod[b][h][2] = prod[b][h][3] = 0.f;
      const int64_t m = r0 + 8 * h + r;
      uint4* const at = reinterpret_cast<uint4*>(st + piece + h * 512);
      const uint4 gv = at[0], uv = at[kGatedAct / 16], dv = at[2 * kGatedAct / 16];
      uint4 og, ou, oh;
      swiglu_bwd8(gv, uv, dv, og, ou, oh);
      if (p.mask) oh = drop8(oh, *reinterpret_cast<const uint2*>(st + warp * kGatedWarpStage + 3 * kGatedAct + h * 256 + lane * 8), p.keep_scale);
      if (in && m < r_end) {
        *reinterpret_cast<uint4*>(p.dg + m * p.lddg + c) = og;
        *reinterpret_cast<uint4*>(p.du + m * p.lddu + c) = ou;
      }
      at[0] = og;
      at[kGatedAct / 16] = ou;
      at[2 * kGatedAct / 16] = oh;
      mma16816(prod[0][h], ra[0].x, rb[0].x, ra[0].y, rb[0].y, og.x, og.y);
      mma16816(prod[1][h], ra[1].x, rb[1].x, ra[1].y, rb[1].y, ou.x, ou.y);
      mma16816(prod[0][h], ra[0].z, rb[0].z, ra[0].w, rb[0].w, og.z, og.w);
      mma16816(prod[1][h], ra[1].z, rb[1].z, ra[1].w, rb[1].w, ou.z, ou.w);
    }
    __syncwarp();
    const uint32_t acts = base + buf * kGatedStage + warp * kGatedWarpStage;
    // side^T as the left operand: (ranks 0-7, rows 0-7), (ranks 8-15, rows 0-7), (ranks 0-7, rows 8-15), (ranks 8-15, rows 8-15)
    const uint32_t sd = smem_u32(side_smem) + buf * kGatedSides + ((lane & 7) + 8 * (lane >> 4)) * kGatedSideRow + (lane >> 3 & 1) * 16;
    const int arow = ((lane >> 3) & 1) * 8 + (lane & 7);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      uint32_t hi[4], lo[4], b[4][2];
      ldmatrix_x4_trans(sd + 2 * a * kGatedSide, hi[0], hi[1], hi[2], hi[3]);
      ldmatrix_x4_trans(sd + (2 * a + 1) * kGatedSide, lo[0], lo[1], lo[2], lo[3]);
#pragma unroll
      for (int np = 0; np < 2; ++np)
        ldmatrix_x4_trans(acts + a * kGatedAct + arow * 64 + (((2 * np + (lane >> 4)) ^ (arow >> 1 & 3)) << 4), b[2 * np][0], b[2 * np][1], b[2 * np + 1][0], b[2 * np + 1][1]);
#pragma unroll
      for (int n = 0; n < 4; ++n) mma16816(acc[a][n], hi[0], hi[1], hi[2], hi[3], b[n][0], b[n][1]);
#pragma unroll
      for (int n = 0; n < 4; ++n) mma16816(acc[a][n], lo[0], lo[1], lo[2], lo[3], b[n][0], b[n][1]);
    }
    // prod[b][h]: ranks r (and r + 8) of rows 8 h + 2 t and + 1
    float* const all = part + buf * (kGatedWarps * kGatedPart);
    float* const mine = all + warp * kGatedPart + 2 * t * kGatedPartRow + r;
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 4; ++i) mine[(8 * h + (i & 1)) * kGatedPartRow + 16 * b + 8 * (i >> 1)] = prod[b][h][i];
    put(side, buf ^ 1);
    cp_async_wait<0>();                            // this thread's part of the next stage
    __syncthreads();                               // everyone's; and the products of this one
#pragma unroll
    for (int i = 0; i < kGatedRows / kGatedWarps; ++i) {
      const int row = warp + kGatedWarps * i;
      const float* q = all + row * kGatedPartRow + lane;
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kGatedWarps; ++w) v += q[w * kGatedPart];
      if (r0 + row < r_end) p.part[(static_cast<int64_t>(blockIdx.x) * p.M + r0 + row) * 32 + lane] = v;
    }
    buf ^= 1;                                      // the exchange is written again only after the next barrier
  }
  // acc[a][n]: rank r (and r + 8) of columns 8 n + 2 t and + 1
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float* const out = a == 0 ? p.grad[0] : a == 1 ? p.grad[1] : p.grad[2];
    const float scale = a < 2 ? p.scale[a & 1] : 1.0f;
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t col = c0 + 8 * n + 2 * t + (i & 1);
        const int rank = r + 8 * (i >> 1);
        if (col < p.I) atomicAdd(a < 2 ? out + col * 16 + rank : out + rank * p.I + col, acc[a][n][i] * scale);
      }
  }
}

// A CTA per row: 32 columns of the parts, eight warps with every eighth part each
__global__ void __launch_bounds__(256)
gated_sum_kernel(const float* __restrict__ part, int parts, int64_t M, float scale_gate, float scale_up, float* __restrict__ u_gate, float* __restrict__ u_up) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float sum[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x;
  float v = 0.f;
#pragma unroll 8
  for (int c = warp; c < parts; c += 8) v += __ldcg(part + (c * M + row) * 32 + lane);
  sum[warp][lane] = v;
  __syncthreads();
  if (warp == 0) {
    v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += sum[w][lane];
    if (lane < 16) u_gate[row * 16 + lane] = v * scale_gate;
    else u_up[row * 16 + lane - 16] = v * scale_up;
  }
}

static int check_mat16(const void* p, int64_t ld, int64_t cols, const char* who, const char* what) {
  if (!p) { set_detail("%s: %s is null", who, what); return NF4LL_ERR_NULL; }
  if ((reinterpret_cast<uintptr_t>(p) & 15) || ld % 8 || ld < cols) {
    set_detail("%s: %s must be 16-byte aligned with a leading dimension multiple of 8 and >= the row length", who, what);
    return NF4LL_ERR_ALIGN;
  }
  return NF4LL_OK;
}

// `shortish`: so few chunks that one per thread and trip serves them best (with two or four some threads of a trip have none): up to four
// trips of all resident threads; 951 x 8960 backward 15.5 us with one, 16.6 with two, 2048 x 8960 31.6 and 30.8
static int grid_for(int64_t total, unsigned* blocks, bool* shortish) {
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int64_t b = (total + 255) / 256;
  const int64_t cap = static_cast<int64_t>(sms) * 8;
  *shortish = total <= 4 * cap * 256;
  *blocks = static_cast<unsigned>(b < cap ? b : cap);
  return NF4LL_OK;
}

}  // namespace nf4ll

extern "C" int nf4ll_swiglu_forward(const void* g, int64_t ldg, const void* u, int64_t ldu, void* h, int64_t ldh, int64_t M,
                                    int64_t I, void* stream) {
  using namespace nf4ll;
  if (M < 0 || I <= 0 || I % 8) { set_detail("nf4ll_swiglu_forward: M=%lld I=%lld", (long long)M, (long long)I); return NF4LL_ERR_SHAPE; }
  if (M == 0) return NF4LL_OK;
  if (int rc = check_mat16(g, ldg, I, "nf4ll_swiglu_forward", "g")) return rc;
  if (int rc = check_mat16(u, ldu, I, "nf4ll_swiglu_forward", "u")) return rc;
  if (int rc = check_mat16(h, ldh, I, "nf4ll_swiglu_forward", "h")) return rc;
  if (int rc = require_sm100()) return rc;
  unsigned blocks = 1;
  const int64_t total = M * (I / 8);
  bool shortish = false;
  if (int rc = grid_for(total, &blocks, &shortish)) return rc;
  PdlLaunch lc(dim3(blocks), dim3(256), 0, static_cast<cudaStream_t>(stream));
  const __half *gp = static_cast<const __half*>(g), *up = static_cast<const __half*>(u);
  __half* hp = static_cast<__half*>(h);
  if (total < (int64_t(1) << 30)) {
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, shortish ? swiglu_fwd_kernel<uint32_t, 1> : swiglu_fwd_kernel<uint32_t, 4>, gp, ldg, up, ldu, hp, ldh,
                                  static_cast<uint32_t>(total), static_cast<uint32_t>(I / 8)));
  } else {
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, swiglu_fwd_kernel<int64_t, 4>, gp, ldg, up, ldu, hp, ldh, total, I / 8));
  }
  return NF4LL_OK;
}

extern "C" int nf4ll_swiglu_backward(const void* g, int64_t ldg, const void* u, int64_t ldu, const void* dh, int64_t lddh,
                                     void* dg, int64_t lddg, void* du, int64_t lddu, int64_t M, int64_t I, void* stream) {
  using namespace nf4ll;
  if (M < 0 || I <= 0 || I % 8) { set_detail("nf4ll_swiglu_backward: M=%lld I=%lld", (long long)M, (long long)I); return NF4LL_ERR_SHAPE; }
  if (M == 0) return NF4LL_OK;
  if (int rc = check_mat16(g, ldg, I, "nf4ll_swiglu_backward", "g")) return rc;
  if (int rc = check_mat16(u, ldu, I, "nf4ll_swiglu_backward", "u")) return rc;
  if (int rc = check_mat16(dh, lddh, I, "nf4ll_swiglu_backward", "dh")) return rc;
  if (int rc = check_mat16(dg, lddg, I, "nf4ll_swiglu_backward", "dg")) return rc;
  if (int rc = check_mat16(du, lddu, I, "nf4ll_swiglu_backward", "du")) return rc;
  if (int rc = require_sm100()) return rc;
  unsigned blocks = 1;
  const int64_t total = M * (I / 8);
  bool shortish = false;
  if (int rc = grid_for(total, &blocks, &shortish)) return rc;
  PdlLaunch lc(dim3(blocks), dim3(256), 0, static_cast<cudaStream_t>(stream));
  const __half *gp = static_cast<const __half*>(g), *up = static_cast<const __half*>(u), *dp = static_cast<const __half*>(dh);
  __half *dgp = static_cast<__half*>(dg), *dup = static_cast<__half*>(du);
  if (total < (int64_t(1) << 30)) {
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, shortish ? swiglu_bwd_kernel<uint32_t, 1> : swiglu_bwd_kernel<uint32_t, 2>, gp, ldg, up, ldu, dp, lddh, dgp, lddg,
                                  dup, lddu, static_cast<uint32_t>(total), static_cast<uint32_t>(I / 8)));
  } else {
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, swiglu_bwd_kernel<int64_t, 2>, gp, ldg, up, ldu, dp, lddh, dgp, lddg, dup, lddu, total, I / 8));
  }
  return NF4LL_OK;
}

// rows per pair of launches at most: bounds the parts of the products (128 B per row and CTA column, half of what a row of dg takes there)
constexpr int64_t kGatedSlab = 4096;

extern "C" int64_t nf4ll_gated_backward_bytes(int64_t M, int64_t I) {
  return M <= 0 || I <= 0 ? 0 : (I + nf4ll::kGatedCols - 1) / nf4ll::kGatedCols * (M < kGatedSlab ? M : kGatedSlab) * 32 * 4;
}

extern "C" int nf4ll_gated_backward(const nf4ll_gated* q, int64_t M, int64_t I, int32_t accumulate, void* scratch, int64_t scratch_bytes, void* stream_v) {
  using namespace nf4ll;
  const char* who = "nf4ll_gated_backward";
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (!q) { set_detail("%s: null pointer", who); return NF4LL_ERR_NULL; }
  if (M < 0 || I <= 0 || I % 8) { set_detail("%s: M=%lld I=%lld", who, (long long)M, (long long)I); return NF4LL_ERR_SHAPE; }
  for (const void* d : {q->dB_gate, q->dB_up, q->dA_down})
    if (!d) { set_detail("%s: null gradient", who); return NF4LL_ERR_NULL; }
  if (M > 0) {
    if (int rc = check_mat16(q->g, q->ldg, I, who, "g")) return rc;
    if (int rc = check_mat16(q->u, q->ldu, I, who, "u")) return rc;
    if (int rc = check_mat16(q->dh, q->lddh, I, who, "dh")) return rc;
    if (int rc = check_mat16(q->dg, q->lddg, I, who, "dg")) return rc;
    if (int rc = check_mat16(q->du, q->lddu, I, who, "du")) return rc;
    for (const void* s : {q->t_gate, q->t_up, q->u_down, q->Bt_gate, q->Bt_up, static_cast<const void*>(q->u_gate), static_cast<const void*>(q->u_up),
                          static_cast<const void*>(scratch)}) {
      if (!s) { set_detail("%s: null pointer", who); return NF4LL_ERR_NULL; }
      if (reinterpret_cast<uintptr_t>(s) & 15) { set_detail("%s: t, u, Bt and scratch must be 16-byte aligned", who); return NF4LL_ERR_ALIGN; }
    }
    if (q->mask && ((reinterpret_cast<uintptr_t>(q->mask) & 15) || q->ld_mask % 16 || q->ld_mask < I)) {
      set_detail("%s: mask 16-byte aligned, ld_mask a multiple of 16 and >= I", who);
      return NF4LL_ERR_ALIGN;
    }
    if (scratch_bytes < nf4ll_gated_backward_bytes(M < kGatedRows ? M : kGatedRows, I)) { set_detail("%s: scratch of %lld bytes", who, (long long)scratch_bytes); return NF4LL_ERR_WORKSPACE; }
  }
  if (int rc = require_sm100()) return rc;
  if (!accumulate)
    for (void* d : {q->dB_gate, q->dB_up, q->dA_down}) NF4LL_CUDA(cudaMemsetAsync(d, 0, sizeof(float) * 16 * I, stream));
  if (M == 0) return NF4LL_OK;
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  NF4LL_CUDA(cudaFuncSetAttribute(gated_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGatedSmem));
  const int64_t cols = (I + kGatedCols - 1) / kGatedCols;
  // as many rows at a time as the scratch has room for, in whole stages
  const int64_t room = scratch_bytes / (cols * 32 * 4), slab = room >= (M < kGatedSlab ? M : kGatedSlab) ? kGatedSlab : room / kGatedRows * kGatedRows;
  for (int64_t m0 = 0; m0 < M; m0 += slab) {
    const int64_t rows = M - m0 < slab ? M - m0 : slab;
    // as many row ranges as one wave of four CTAs per SM holds
    const int64_t steps = (rows + kGatedRows - 1) / kGatedRows;
    int64_t ranges = 4 * static_cast<int64_t>(sms) / cols;
    ranges = ranges < 1 ? 1 : ranges > steps ? steps : ranges;
    const int64_t rows_per = (steps + ranges - 1) / ranges * kGatedRows;
    ranges = (rows + rows_per - 1) / rows_per;
    const GatedParams p{static_cast<const __half*>(q->g) + m0 * q->ldg, static_cast<const __half*>(q->u) + m0 * q->ldu,
                        static_cast<const __half*>(q->dh) + m0 * q->lddh, static_cast<__half*>(q->dg) + m0 * q->lddg,
                        static_cast<__half*>(q->du) + m0 * q->lddu, q->ldg, q->ldu, q->lddh, q->lddg, q->lddu,
                        q->mask ? q->mask + m0 * q->ld_mask : nullptr, q->ld_mask, q->keep_scale,
                        {static_cast<const float*>(q->t_gate) + m0 * 16, static_cast<const float*>(q->t_up) + m0 * 16, static_cast<const float*>(q->u_down) + m0 * 16},
                        {static_cast<const __half*>(q->Bt_gate), static_cast<const __half*>(q->Bt_up)},
                        {static_cast<float*>(q->dB_gate), static_cast<float*>(q->dB_up), static_cast<float*>(q->dA_down)}, {q->scale_gate, q->scale_up},
                        static_cast<float*>(scratch), rows, I, rows_per};
    PdlLaunch lc(dim3(static_cast<unsigned>(cols), static_cast<unsigned>(ranges)), dim3(kGatedThreads), kGatedSmem, stream);
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, gated_bwd_kernel, p));
    PdlLaunch sum(dim3(static_cast<unsigned>(rows)), dim3(256), 0, stream);
    NF4LL_CUDA(cudaLaunchKernelEx(&sum.cfg, gated_sum_kernel, static_cast<const float*>(p.part), static_cast<int>(cols), rows, q->scale_gate, q->scale_up,
                                  static_cast<float*>(q->u_gate) + m0 * 16, static_cast<float*>(q->u_up) + m0 * 16));
  }
  return NF4LL_OK;
}
