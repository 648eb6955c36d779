// Fused residual add + RMSNorm producer of the NF4 + LoRA linear's inputs, and its backward.
//
// Forward (replaces the reference's rms_fwd_kernel, solution/k_norm.py:29-53, and the two LoRA-A GEMMs that
// read its xq / xv outputs, solution/fast_qwen.py:943-944; call sites fast_qwen.py:1021-1027):
//     x    = x_prev (fp32) [+ delta (fp16 GEMM output)]        residual stream, kept in fp32
//     rstd = rsqrt(mean(x^2) + eps)
//     y    = w * (x * rstd);   y16 = fp16(y)                    the A operand of the projections that follow
//     T_i  = fp16(keep_i ? y * keep_scale : 0) . A_i^T          for up to two LoRA branches (q and v), fp32 [M,16]
// The reference writes the dropped-out copies xq, xv ([M, D] fp16 each) and multiplies them by lora_A in
// separate GEMMs; here the rank-16 products are formed on the tensor cores while y is still in registers, so
// neither the copies nor a second pass over y exist, and the projections get their rank-16 operand ready-made.
//
// Backward (replaces rms_bwd_kernel, solution/k_norm.py:56-87, and the two GEMMs lqx = daq . A_q,
// lvx = dav . A_v that feed it, solution/fast_qwen.py:1376-1380):
//     dy   = fp16 grad * gscale + sum_i keep_i * keep_scale * (u_i . A_i)     u_i fp32 [M,16] = scale * d(out_i) . B_i
//     dx   = rstd * (w*dy - xhat * mean(w*dy*xhat)),  xhat = x * rstd
//     out  = dres + dx  (fp32)  and its fp16 copy
// The [M, D] LoRA input gradients of the reference never exist: the rank-16 factors are expanded per element.
//
// A group of 8 token rows (16 in the forward of a long batch) belongs to a CTA or, where the groups would leave SMs idle, to a cluster
// whose CTAs share out the hidden dimension; a lane's values stay in registers between the row reduction and the second phase.
#include "nf4ll_lora.cuh"
#include "nf4ll_pair.cuh"

namespace nf4ll {

constexpr int kNormWarps = 16;

struct NormBranch {
  const __half* A;        // lora_A fp16 [16, D]; null = branch absent
  const uint8_t* mask;    // keep-mask [M, ld_mask] or null (no dropout)
  int64_t ld_mask;
  float keep_scale;
  float* t;               // forward: out fp32 [M,16]
  const float* u;         // backward: in fp32 [M,16]
};

__device__ __forceinline__ void load8_f32(const float* p, float (&v)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// of memory that the kernel writes too
__device__ __forceinline__ void load8_f32_rw(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store8_f32(float* p, const float (&v)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ bool keep_bit(const uint2& m, int j) {
  return (((j < 4 ? m.x : m.y) >> ((j & 3) * 8)) & 0xffu) != 0;
}

// RG row groups of 8 rows per CTA, CPW 32-column chunks per warp (D <= kNormWarps * 32 * CPW)
template <int RG, int CPW>
__global__ void __launch_bounds__(kNormWarps * 32)
rms_fwd_kernel(const float* __restrict__ x, const __half* __restrict__ delta, float* __restrict__ xout,
               const float* __restrict__ w, float eps, int64_t M, int64_t D, __half* __restrict__ y16, int64_t ldy,
               float* __restrict__ rstd_out, const NormBranch ba, const NormBranch bb) {
  pdl_wait();
  pdl_launch_dependents();
  constexpr int ROWS = 8 * RG;
  __shared__ float s_part[kNormWarps][ROWS];
  __shared__ float s_rstd[ROWS];
  __shared__ float s_t[kNormWarps][ROWS][17];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int64_t m0 = static_cast<int64_t>(blockIdx.x) * ROWS;
  int64_t row[RG];
  bool ok[RG];
#pragma unroll
  for (int i = 0; i < RG; ++i) {
    row[i] = m0 + g + 8 * i;
    ok[i] = row[i] < M;
    if (!ok[i]) row[i] = 0;
  }
  // phase 1: load (x + delta), write the residual stream, sum of squares
  float xv[CPW][RG][8];
  float ss[RG];
#pragma unroll
  for (int i = 0; i < RG; ++i) ss[i] = 0.f;
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int64_t k = (static_cast<int64_t>(c) * kNormWarps + warp) * 32 + t * 8;
#pragma unroll
    for (int i = 0; i < RG; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) xv[c][i][j] = 0.f;
      if (k < D && ok[i]) {
        load8_f32(x + row[i] * D + k, xv[c][i]);
        if (delta) {
          float dv[8];
          unpack8(__ldg(reinterpret_cast<const uint4*>(delta + row[i] * D + k)), dv);
#pragma unroll
          for (int j = 0; j < 8; ++j) xv[c][i][j] += dv[j];
        }
        if (xout) store8_f32(xout + row[i] * D + k, xv[c][i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss[i] = fmaf(xv[c][i][j], xv[c][i][j], ss[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RG; ++i) {
    ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 1);
    ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 2);
    if (t == 0) s_part[warp][g + 8 * i] = ss[i];
  }
  __syncthreads();
  if (threadIdx.x < ROWS) {
    float v = 0.f;
#pragma unroll
    for (int wq = 0; wq < kNormWarps; ++wq) v += s_part[wq][threadIdx.x];
    const float r = rsqrtf(v * (1.0f / static_cast<float>(D)) + eps);
    s_rstd[threadIdx.x] = r;
    if (m0 + threadIdx.x < M) rstd_out[m0 + threadIdx.x] = r;
  }
  __syncthreads();
  // phase 2: y, its fp16 copy, and the rank-16 products of the dropped-out copies
  float ca[RG][4], cb[RG][4];
#pragma unroll
  for (int i = 0; i < RG; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) { ca[i][j] = 0.f; cb[i][j] = 0.f; }
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int64_t kc = (static_cast<int64_t>(c) * kNormWarps + warp) * 32;      // first column of the warp's chunk
    const int64_t k = kc + t * 8;
    // the MMAs below are warp-wide instructions: the whole warp takes part in a chunk that starts inside the
    // row, and lanes whose eight columns lie past its end (D need not be a multiple of 32) contribute zeros
    if (kc < D) {
      const bool in = k < D;
      float wv[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) wv[j] = 0.f;
      if (in) load8_f32(w + k, wv);
      uint4 ra = make_uint4(0, 0, 0, 0), rb = ra, sa = ra, sb = ra;
      if (ba.A && in) { ra = __ldg(reinterpret_cast<const uint4*>(ba.A + static_cast<int64_t>(g) * D + k));
                        rb = __ldg(reinterpret_cast<const uint4*>(ba.A + static_cast<int64_t>(g + 8) * D + k)); }
      if (bb.A && in) { sa = __ldg(reinterpret_cast<const uint4*>(bb.A + static_cast<int64_t>(g) * D + k));
                        sb = __ldg(reinterpret_cast<const uint4*>(bb.A + static_cast<int64_t>(g + 8) * D + k)); }
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        const float r = s_rstd[g + 8 * i];
        const bool live = in && ok[i];
        float y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = wv[j] * (xv[c][i][j] * r);
        if (y16 && live) *reinterpret_cast<uint4*>(y16 + row[i] * ldy + k) = pack8(y);
        if (ba.A) {
          float d[8];
          const uint2 m = (ba.mask && live) ? __ldg(reinterpret_cast<const uint2*>(ba.mask + row[i] * ba.ld_mask + k)) : make_uint2(0, 0);
#pragma unroll
          for (int j = 0; j < 8; ++j) d[j] = live ? (ba.mask ? (keep_bit(m, j) ? y[j] * ba.keep_scale : 0.f) : y[j]) : 0.f;
          const uint4 q = pack8(d);
          mma16816(ca[i], ra.x, rb.x, ra.y, rb.y, q.x, q.y);
          mma16816(ca[i], ra.z, rb.z, ra.w, rb.w, q.z, q.w);
        }
        if (bb.A) {
          float d[8];
          const uint2 m = (bb.mask && live) ? __ldg(reinterpret_cast<const uint2*>(bb.mask + row[i] * bb.ld_mask + k)) : make_uint2(0, 0);
#pragma unroll
          for (int j = 0; j < 8; ++j) d[j] = live ? (bb.mask ? (keep_bit(m, j) ? y[j] * bb.keep_scale : 0.f) : y[j]) : 0.f;
          const uint4 q = pack8(d);
          mma16816(cb[i], sa.x, sb.x, sa.y, sb.y, q.x, q.y);
          mma16816(cb[i], sa.z, sb.z, sa.w, sb.w, q.z, q.w);
        }
      }
    }
  }
  // accumulator layout: c[.][0], c[.][1] = (rank g, rows 2t, 2t+1); c[.][2], c[.][3] = (rank g+8, same rows)
#pragma unroll
  for (int br = 0; br < 2; ++br) {
    const NormBranch& b = br ? bb : ba;
    if (!b.A) continue;               // uniform over the CTA
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RG; ++i) {
      const float* c = br ? cb[i] : ca[i];
      s_t[warp][8 * i + 2 * t][g] = c[0];      s_t[warp][8 * i + 2 * t + 1][g] = c[1];
      s_t[warp][8 * i + 2 * t][g + 8] = c[2];  s_t[warp][8 * i + 2 * t + 1][g + 8] = c[3];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < ROWS * 16; idx += kNormWarps * 32) {
      const int rr = idx >> 4, j = idx & 15;
      if (m0 + rr < M) {
        float v = 0.f;
#pragma unroll
        for (int wq = 0; wq < kNormWarps; ++wq) v += s_t[wq][rr][j];
        b.t[(m0 + rr) * 16 + j] = v;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The forward for batches whose groups of rows do not fill the SMs: eight rows per cluster of up to eight CTAs (eight warps each),
// which share out the columns. The row sums meet through distributed shared memory, every CTA adding them up in rank order, and the
// rank-16 products in the first CTA likewise. Such a batch is bound by the chain load - sum - products - store of one CTA, so what
// counts is how little of a row a CTA has, and that the loads of the second phase are on their way before the sum: one CTA of sixteen
// warps per 16 (D > 2048: 8) rows against this, us, with two branches / without, three sets of operands in turn: 1536 columns, 8 rows 9.3 / 4.7 ->
// 4.4 / 2.7, 333 rows 12.3 / 7.1 -> 6.0 / 3.7, 951 rows 12.5 / 7.2 -> 9.0 / 5.5; 3584 columns, 8 rows 14.3 / 8.6 -> 5.3 / 3.2, 333 rows 14.6 / 8.8 -> 8.4 / 5.1.
// ---------------------------------------------------------------------------------------------
constexpr int kSplitWarps = 8;

__device__ __forceinline__ float peer_f32(const float* local, uint32_t rank) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_cta(smem_u32(local), rank)) : "memory");
  return v;
}

// total over the cluster of every row's sum, for row g: part[warp][row] of each CTA; s_sum is read by the others until the next cluster barrier
template <int NW>
__device__ __forceinline__ float split_row_total(const float (&part)[NW][8], float (&s_sum)[8], int g) {
  __syncthreads();
  if (threadIdx.x < 8) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) v += part[w][threadIdx.x];
    s_sum[threadIdx.x] = v;
  }
  if (gridDim.y == 1) {
    __syncthreads();
    return s_sum[g];
  }
  cluster_sync_all();
  float peer[8], v = 0.f;
#pragma unroll
  for (uint32_t r = 0; r < 8; ++r) peer[r] = r < gridDim.y ? peer_f32(&s_sum[g], r) : 0.f;      // all in flight at once
#pragma unroll
  for (uint32_t r = 0; r < 8; ++r) v += peer[r];
  return v;
}

// CPW chunks of 32 columns per warp; `chunks` of them per CTA
template <int CPW>
__global__ void __launch_bounds__(kSplitWarps * 32, 2)
rms_fwd_split_kernel(const float* __restrict__ x, const __half* __restrict__ delta, float* __restrict__ xout, const float* __restrict__ w, float eps,
                     int64_t M, int64_t D, __half* __restrict__ y16, int64_t ldy, float* __restrict__ rstd_out, const NormBranch ba, const NormBranch bb,
                     int chunks) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float s_part[kSplitWarps][8];
  __shared__ float s_sum[8];
  __shared__ float s_t[2][kSplitWarps][8][17];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * 8 + g;
  const bool ok = row < M;
  const int64_t col0 = static_cast<int64_t>(blockIdx.y) * chunks * 32;
  const int64_t col1 = col0 + chunks * 32 < D ? col0 + chunks * 32 : D;
  float xv[CPW][8], wv[CPW][8], ss = 0.f;
  constexpr bool kEarly = CPW <= 2;                // lora_A of both branches, ranks g and g + 8, before the sums where registers allow
  uint4 fr[kEarly ? CPW : 1][4];
  auto load_fr = [&](int64_t k, uint4 (&f)[4]) {
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const __half* A = b ? bb.A : ba.A;
      const uint4 zero = make_uint4(0, 0, 0, 0);
      f[2 * b] = A && k < col1 ? __ldg(reinterpret_cast<const uint4*>(A + static_cast<int64_t>(g) * D + k)) : zero;
      f[2 * b + 1] = A && k < col1 ? __ldg(reinterpret_cast<const uint4*>(A + static_cast<int64_t>(g + 8) * D + k)) : zero;
    }
  };
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int64_t k = col0 + (c * kSplitWarps + warp) * 32 + t * 8;
    const bool in = k < col1;
#pragma unroll
    for (int j = 0; j < 8; ++j) xv[c][j] = wv[c][j] = 0.f;
    if (in && ok) {
      load8_f32(x + row * D + k, xv[c]);
      if (delta) {
        float dv[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(delta + row * D + k)), dv);
#pragma unroll
        for (int j = 0; j < 8; ++j) xv[c][j] += dv[j];
      }
    }
    if (in) load8_f32(w + k, wv[c]);
    if (kEarly) load_fr(k, fr[c]);
  }
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int64_t k = col0 + (c * kSplitWarps + warp) * 32 + t * 8;
    if (xout && k < col1 && ok) store8_f32(xout + row * D + k, xv[c]);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss = fmaf(xv[c][j], xv[c][j], ss);
  }
  ss += __shfl_xor_sync(0xffffffffu, ss, 1);
  ss += __shfl_xor_sync(0xffffffffu, ss, 2);
  if (t == 0) s_part[warp][g] = ss;
  const float r = rsqrtf(split_row_total(s_part, s_sum, g) * (1.0f / static_cast<float>(D)) + eps);
  if (blockIdx.y == 0 && warp == 0 && t == 0 && ok) rstd_out[row] = r;
  float acc[2][4];
#pragma unroll
  for (int b = 0; b < 2; ++b) acc[b][0] = acc[b][1] = acc[b][2] = acc[b][3] = 0.f;
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int64_t k = col0 + (c * kSplitWarps + warp) * 32 + t * 8;
    const bool live = k < col1 && ok;
    uint4 (&f)[4] = fr[kEarly ? c : 0];
    if (!kEarly) load_fr(k, f);
    float y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) y[j] = wv[c][j] * (xv[c][j] * r);
    if (y16 && live) *reinterpret_cast<uint4*>(y16 + row * ldy + k) = pack8(y);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const NormBranch& br = b ? bb : ba;
      if (!br.A) continue;
      float d[8];
      const uint2 m = br.mask && live ? __ldg(reinterpret_cast<const uint2*>(br.mask + row * br.ld_mask + k)) : make_uint2(0, 0);
#pragma unroll
      for (int j = 0; j < 8; ++j) d[j] = live ? (br.mask ? (keep_bit(m, j) ? y[j] * br.keep_scale : 0.f) : y[j]) : 0.f;
      const uint4 q = pack8(d);
      mma16816(acc[b], f[2 * b].x, f[2 * b + 1].x, f[2 * b].y, f[2 * b + 1].y, q.x, q.y);
      mma16816(acc[b], f[2 * b].z, f[2 * b + 1].z, f[2 * b].w, f[2 * b + 1].w, q.z, q.w);
    }
  }
  if (ba.A || bb.A) {
    // acc[b][0], [1] = (rank g, rows 2t, 2t+1); [2], [3] = (rank g+8, same rows)
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int i = 0; i < 4; ++i) s_t[b][warp][2 * t + (i & 1)][g + 8 * (i >> 1)] = acc[b][i];
    __syncthreads();
    const int b = threadIdx.x >> 7, rr = threadIdx.x >> 4 & 7, j = threadIdx.x & 15;
    float v = 0.f;
#pragma unroll
    for (int wq = 0; wq < kSplitWarps; ++wq) v += s_t[b][wq][rr][j];
    if (gridDim.y > 1) {
      s_t[b][0][rr][j] = v;                        // read and written by this thread only
      cluster_sync_all();
      if (blockIdx.y == 0) {
        float peer[8];
#pragma unroll
        for (uint32_t q = 1; q < 8; ++q) peer[q] = q < gridDim.y ? peer_f32(&s_t[b][0][rr][j], q) : 0.f;
#pragma unroll
        for (uint32_t q = 1; q < 8; ++q) v += peer[q];
      }
    }
    const NormBranch& br = b ? bb : ba;
    const int64_t m = static_cast<int64_t>(blockIdx.x) * 8 + rr;
    if (blockIdx.y == 0 && br.A && m < M) br.t[m * 16 + j] = v;
  }
  if (gridDim.y > 1) cluster_sync_all();           // shared memory stays until the others have read it
}

// The expansion u . A on the tensor cores: a lane's sixteen bytes of a rank's row are four 2-column pieces, which movmatrix turns into the
// right operand for columns 8 i + 2 w, + 1 (i = 0..3), so that over w = 0..3 lane (g, t) ends with its own columns 8 t .. + 7 of row g. u
// goes in three fp16 parts under a power of two per row that brings its largest rank to [2^14, 2^15): all 24 bits of every rank down to
// 2^-15 of the largest; of smaller ones what is above 2^-40 of the largest.
// With fp32 FMAs it was 32 loads, 256 conversions and 256 FMAs per lane and chunk, and the larger error against fp64 (8.6e-8 of the
// result's norm at u of 1 with 1536 columns, 6.6e-8 so). us with two branches / without, one CTA and FMAs before, three sets of operands in turn: 1536
// columns, 8 rows 12.6 / 5.8 -> 4.4 / 2.9, 951 rows 16.7 / 8.6 -> 12.7 / 8.3, 2048 rows (a CTA per group) 39.0 / 20.6 -> 31.1 / 20.1; 3584 columns,
// 333 rows 33.7 / 13.4 -> 10.8 / 6.9, 2048 rows 117 / 45 -> 68 / 42.
template <int CPW, int NW, bool KEEP>
__global__ void __launch_bounds__(NW * 32, NW == kSplitWarps ? 2 : 1)
rms_bwd_kernel(const __half* __restrict__ dy16, int64_t lddy, float gscale, const float* __restrict__ x, const __half* __restrict__ delta,
                     const float* __restrict__ w, const float* __restrict__ rstd, const float* dres, float* out, __half* __restrict__ out16, int64_t M,
                     int64_t D, const NormBranch ba, const NormBranch bb, int chunks) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ float s_part[NW][8];
  __shared__ float s_sum[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * 8 + g;
  const bool ok = row < M;
  const int64_t col0 = static_cast<int64_t>(blockIdx.y) * chunks * 32;
  const int64_t col1 = col0 + chunks * 32 < D ? col0 + chunks * 32 : D;
  const float r = ok ? __ldg(rstd + row) : 0.f;
  auto load_x = [&](int64_t k, float (&v)[8]) {
    load8_f32(x + row * D + k, v);
    if (delta) {
      float dv[8];
      unpack8(__ldg(reinterpret_cast<const uint4*>(delta + row * D + k)), dv);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += dv[j];
    }
  };
  // left operand: row g, ranks 2t, 2t+1 and + 8 (rows g + 8 are zeros)
  uint32_t ul[2][3], uh[2][3];
  float back[2] = {1.f, 1.f};
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const NormBranch& br = b ? bb : ba;
    if (!br.A) continue;
    const float2 zero = make_float2(0.f, 0.f);
    float2 lo = ok ? __ldg(reinterpret_cast<const float2*>(br.u + row * 16 + 2 * t)) : zero;
    float2 hi = ok ? __ldg(reinterpret_cast<const float2*>(br.u + row * 16 + 2 * t + 8)) : zero;
    lo.x *= br.keep_scale; lo.y *= br.keep_scale; hi.x *= br.keep_scale; hi.y *= br.keep_scale;
    const RowScale f = row_scale(fmaxf(fmaxf(fabsf(lo.x), fabsf(lo.y)), fmaxf(fabsf(hi.x), fabsf(hi.y))));
    back[b] = f.back;
    split_parts(lo.x * f.to, lo.y * f.to, ul[b]);
    split_parts(hi.x * f.to, hi.y * f.to, uh[b]);
  }
  constexpr int KC = KEEP ? CPW : 1;               // chunks whose x and dres stay in registers
  float gv[CPW][8], xh[KC][8], dr[KC][8], cs = 0.f;
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int64_t k = col0 + (c * NW + warp) * 32 + t * 8;
    const bool in = k < col1, live = in && ok;
    const int kc = KEEP ? c : 0;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    float dy[8], wv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) xh[kc][j] = dr[kc][j] = wv[j] = 0.f;
    unpack8(live ? __ldg(reinterpret_cast<const uint4*>(dy16 + row * lddy + k)) : zero, dy);
    if (live) {
      load_x(k, xh[kc]);
      if (KEEP && dres) load8_f32_rw(dres + row * D + k, dr[kc]);
    }
    if (in) load8_f32(w + k, wv);
#pragma unroll
    for (int j = 0; j < 8; ++j) dy[j] *= gscale;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const NormBranch& br = b ? bb : ba;
      if (!br.A) continue;
      const uint4 f0 = in ? __ldg(reinterpret_cast<const uint4*>(br.A + static_cast<int64_t>(g) * D + k)) : zero;
      const uint4 f1 = in ? __ldg(reinterpret_cast<const uint4*>(br.A + static_cast<int64_t>(g + 8) * D + k)) : zero;
      const uint2 m = br.mask && live ? __ldg(reinterpret_cast<const uint2*>(br.mask + row * br.ld_mask + k)) : make_uint2(0, 0);
      const uint32_t p0[4] = {f0.x, f0.y, f0.z, f0.w}, p1[4] = {f1.x, f1.y, f1.z, f1.w};
      uint32_t b0[4], b1[4];
      float l[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        b0[q] = transpose8x8(p0[q]);
        b1[q] = transpose8x8(p1[q]);
        l[q][0] = l[q][1] = l[q][2] = l[q][3] = 0.f;
      }
#pragma unroll
      for (int i = 2; i >= 0; --i)                 // the smallest part first
#pragma unroll
        for (int q = 0; q < 4; ++q) mma16816(l[q], ul[b][i], 0u, uh[b][i], 0u, b0[q], b1[q]);
#pragma unroll
      for (int j = 0; j < 8; ++j) dy[j] += !br.mask || keep_bit(m, j) ? l[j >> 1][j & 1] * back[b] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      xh[kc][j] *= r;
      gv[c][j] = dy[j] * wv[j];
      cs = fmaf(gv[c][j], xh[kc][j], cs);
    }
  }
  cs += __shfl_xor_sync(0xffffffffu, cs, 1);
  cs += __shfl_xor_sync(0xffffffffu, cs, 2);
  if (t == 0) s_part[warp][g] = cs;
  const float cm = split_row_total(s_part, s_sum, g) * (1.0f / static_cast<float>(D));
#pragma unroll
  for (int c = 0; c < CPW; ++c) {
    const int64_t k = col0 + (c * NW + warp) * 32 + t * 8;
    if (k < col1 && ok) {
      float o[8];
      const int kc = KEEP ? c : 0;
      if (!KEEP) {                                 // second read of x: from L1 / L2
        load_x(k, xh[0]);
#pragma unroll
        for (int j = 0; j < 8; ++j) xh[0][j] *= r, dr[0][j] = 0.f;
        if (dres) load8_f32_rw(dres + row * D + k, dr[0]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = (gv[c][j] - xh[kc][j] * cm) * r + dr[kc][j];
      store8_f32(out + row * D + k, o);
      if (out16) *reinterpret_cast<uint4*>(out16 + row * D + k) = pack8(o);
    }
  }
  if (gridDim.y > 1) cluster_sync_all();
}

// How many clusters of `parts` CTAs of eight warps the current device holds at once. They lie in a GPC each, so not as many as its SMs hold
// CTAs (two each): 74 clusters of four would, and took two waves (590 rows of 1536 backward 8.3 us, in threes 5.4).
static int split_clusters(int parts) {
  constexpr int kDevices = 64;
  static int known[kDevices][9];               // 0: not asked yet; written with the same value by any thread
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
  int n = __atomic_load_n(&known[dev][parts], __ATOMIC_RELAXED);
  if (n > 0) return n;
  const void* kernel = reinterpret_cast<const void*>(rms_bwd_kernel<4, kSplitWarps, true>);
  PdlLaunch probe(dim3(1, static_cast<unsigned>(parts)), dim3(kSplitWarps * 32), 0, nullptr, 1, static_cast<unsigned>(parts), false, false);
  probe.cfg.numAttrs = 1;                      // the cluster dimension only
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &probe.cfg) != cudaSuccess) n = 0;
  if (n > 0) __atomic_store_n(&known[dev][parts], n, __ATOMIC_RELAXED);
  else (void)cudaGetLastError();
  return n;
}

// CTAs per group of eight rows and 32-column chunks per CTA: as many CTAs as find room at once, behind another kernel, each warp with a chunk at
// least. Backward in a row of calls without branches and with two, us: 54 groups of 1536 columns, two chunks to a warp either way, by fives, of which
// the device holds 56, 5.7 and 8.8, by fours 4.9 and 7.2; 36 of 3584 columns by sevens, of which it holds 37, two chunks, 5.6 and 8.5, by sixes,
// three chunks, 6.8 and 10.4. parts = 0: a
// second wave would be needed (951 rows of 1536 in two waves of clusters: 23.7 us against 20.3), or a row is too long for what is free; then
// a CTA of sixteen warps takes the whole row. So it does in the backward where pairs would share SMs, unevenly, without the factors' products
// to keep them busy, or with all of a warp's registers taken: with / without two branches, us, in pairs and by whole rows, 951 rows of 896
// columns 7.6, 5.1 and 8.8, 4.7; of 1536 13.6, 8.8 and 14.7, 8.8 (700 rows 11.1, 7.3 and 11.5, 7.0); of 2048 19.7, 13.4 and 18.3, 12.4. parts = 1 is
// worth it in the backward only (2048 rows of 1024: 12.6 us against 15.1; forward 9.1 against 8.4).
struct NormSplit {
  unsigned groups, parts;
  int chunks, cpw;
};
static int norm_split(NormSplit* s, int64_t M, int64_t D, bool backward, bool branches) {
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t groups = (M + 7) / 8, all = (D + 31) / 32;
  int64_t parts = 8;
  // Clusters that find no room while the kernel before this one still holds SMs come a wave later: the last two of most sizes, of fives and
  // threes more. That costs more than a CTA less to a row would, unless its warps then had another chunk to go through (second line).
  constexpr int kWait[2][9] = {{0, 0, 0, 3, 2, 5, 2, 2, 2}, {0, 0, 0, 1, 0, 1, 0, 0, 0}};
  auto warp_chunks = [&](int64_t n) { return ((all + n - 1) / n + kSplitWarps - 1) / kSplitWarps; };
  auto fits = [&](int64_t n) {
    if (n == 1) return groups <= 2 * static_cast<int64_t>(sms);
    return groups <= split_clusters(static_cast<int>(n)) - kWait[warp_chunks(n) < warp_chunks(n - 1)][n];
  };
  while (parts > 1 && (!fits(parts) || all < parts * kSplitWarps)) --parts;
  *s = NormSplit{static_cast<unsigned>(groups), 0, 0, 0};
  const int64_t chunks = (all + parts - 1) / parts;
  if (!fits(parts) || chunks > 4 * kSplitWarps) return NF4LL_OK;
  if (backward && parts == 2 && 2 * groups > sms && !(branches && chunks <= 3 * kSplitWarps)) return NF4LL_OK;
  s->chunks = static_cast<int>(chunks);
  s->parts = static_cast<unsigned>((all + chunks - 1) / chunks);
  s->cpw = static_cast<int>((chunks + kSplitWarps - 1) / kSplitWarps);
  return NF4LL_OK;
}

static int check_branch(const nf4ll_lora* l, const void* side, const char* who, int64_t D, NormBranch* out, bool forward) {
  *out = NormBranch{};
  if (!l) return NF4LL_OK;
  if (l->r != 16) { set_detail("%s: LoRA rank %d", who, l->r); return NF4LL_ERR_RANK; }
  if (!l->A || !side) { set_detail("%s: a LoRA branch needs lora_A and its [M,16] %s", who, forward ? "output t" : "input u"); return NF4LL_ERR_NULL; }
  if ((reinterpret_cast<uintptr_t>(l->A) & 15) || (reinterpret_cast<uintptr_t>(side) & 15)) { set_detail("%s: LoRA operands must be 16-byte aligned", who); return NF4LL_ERR_ALIGN; }
  if (l->mask && ((reinterpret_cast<uintptr_t>(l->mask) & 7) || l->ld_mask % 8 || l->ld_mask < D)) {
    set_detail("%s: mask must be 8-byte aligned with ld_mask a multiple of 8 and >= D", who);
    return NF4LL_ERR_ALIGN;
  }
  out->A = static_cast<const __half*>(l->A);
  out->mask = l->mask; out->ld_mask = l->ld_mask; out->keep_scale = l->mask ? l->keep_scale : 1.0f;
  if (forward) out->t = static_cast<float*>(const_cast<void*>(side)); else out->u = static_cast<const float*>(side);
  return NF4LL_OK;
}

static int check_norm_shape(const char* who, int64_t M, int64_t D) {
  if (M < 0 || D <= 0 || D % 8 || D > kNormWarps * 32 * 8) {
    set_detail("%s: M=%lld, D=%lld (D a multiple of 8, at most %d)", who, static_cast<long long>(M), static_cast<long long>(D), kNormWarps * 32 * 8);
    return NF4LL_ERR_SHAPE;
  }
  return NF4LL_OK;
}

}  // namespace nf4ll

extern "C" int nf4ll_rms_forward(const float* x, const void* delta16, float* xout, const float* w, float eps, int64_t M,
                                 int64_t D, void* y16, int64_t ldy, float* rstd, const nf4ll_lora* lora_a, void* t_a,
                                 const nf4ll_lora* lora_b, void* t_b, void* stream) {
  using namespace nf4ll;
  const char* who = "nf4ll_rms_forward";
  if (int rc = check_norm_shape(who, M, D)) return rc;
  if (M == 0) return NF4LL_OK;
  if (!x || !w || !rstd) { set_detail("%s: x, w and rstd are required", who); return NF4LL_ERR_NULL; }
  for (const void* p : {static_cast<const void*>(x), delta16, static_cast<const void*>(xout), static_cast<const void*>(w), static_cast<const void*>(y16)})
    if (reinterpret_cast<uintptr_t>(p) & 15) { set_detail("%s: pointers must be 16-byte aligned", who); return NF4LL_ERR_ALIGN; }
  if (y16 && (ldy % 8 || ldy < D)) { set_detail("%s: ldy must be a multiple of 8 and >= D", who); return NF4LL_ERR_ALIGN; }
  NormBranch ba, bb;
  if (int rc = check_branch(lora_a, t_a, who, D, &ba, true)) return rc;
  if (int rc = check_branch(lora_b, t_b, who, D, &bb, true)) return rc;
  if (int rc = require_sm100()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int cpw = static_cast<int>((D + kNormWarps * 32 - 1) / (kNormWarps * 32));
  const __half* dl = static_cast<const __half*>(delta16);
  __half* y = static_cast<__half*>(y16);
  NormSplit s;
  if (int rc = norm_split(&s, M, D, false, false)) return rc;
  if (s.parts > 1) {
    PdlLaunch lc(dim3(s.groups, s.parts), dim3(kSplitWarps * 32), 0, st, 1, s.parts);
    const auto kernel = s.cpw <= 1 ? rms_fwd_split_kernel<1> : s.cpw <= 2 ? rms_fwd_split_kernel<2> : s.cpw <= 3 ? rms_fwd_split_kernel<3> : rms_fwd_split_kernel<4>;
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, kernel, x, dl, xout, w, eps, M, D, y, ldy, rstd, ba, bb, s.chunks));
    return NF4LL_OK;
  }
  if (cpw <= 4) {
    PdlLaunch lc(dim3(static_cast<unsigned>((M + 15) / 16)), dim3(kNormWarps * 32), 0, st);
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, rms_fwd_kernel<2, 4>, x, dl, xout, w, eps, M, D, y, ldy, rstd, ba, bb));
  } else {
    PdlLaunch lc(dim3(static_cast<unsigned>((M + 7) / 8)), dim3(kNormWarps * 32), 0, st);
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, rms_fwd_kernel<1, 8>, x, dl, xout, w, eps, M, D, y, ldy, rstd, ba, bb));
  }
  return NF4LL_OK;
}

extern "C" int nf4ll_rms_backward(const void* dy16, int64_t lddy, float gscale, const float* x, const void* delta16,
                                  const float* w, const float* rstd, const float* dres, float* out, void* out16, int64_t M,
                                  int64_t D, const nf4ll_lora* lora_a, const void* u_a, const nf4ll_lora* lora_b,
                                  const void* u_b, void* stream) {
  using namespace nf4ll;
  const char* who = "nf4ll_rms_backward";
  if (int rc = check_norm_shape(who, M, D)) return rc;
  if (M == 0) return NF4LL_OK;
  if (!dy16 || !x || !w || !rstd || !out) { set_detail("%s: dy, x, w, rstd and out are required", who); return NF4LL_ERR_NULL; }
  for (const void* p : {dy16, static_cast<const void*>(x), delta16, static_cast<const void*>(w), static_cast<const void*>(dres),
                        static_cast<const void*>(out), static_cast<const void*>(out16)})
    if (reinterpret_cast<uintptr_t>(p) & 15) { set_detail("%s: pointers must be 16-byte aligned", who); return NF4LL_ERR_ALIGN; }
  if (lddy % 8 || lddy < D) { set_detail("%s: lddy must be a multiple of 8 and >= D", who); return NF4LL_ERR_ALIGN; }
  NormBranch ba, bb;
  if (int rc = check_branch(lora_a, u_a, who, D, &ba, false)) return rc;
  if (int rc = check_branch(lora_b, u_b, who, D, &bb, false)) return rc;
  if (int rc = require_sm100()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* dyp = static_cast<const __half*>(dy16);
  const __half* dl = static_cast<const __half*>(delta16);
  __half* o16 = static_cast<__half*>(out16);
  NormSplit s;
  if (int rc = norm_split(&s, M, D, true, ba.A || bb.A)) return rc;
  const auto kernel = !s.parts ? (D <= kNormWarps * 32 * 4 ? rms_bwd_kernel<4, kNormWarps, false> : rms_bwd_kernel<8, kNormWarps, false>)
                      : s.cpw <= 1 ? rms_bwd_kernel<1, kSplitWarps, true> : s.cpw <= 2 ? rms_bwd_kernel<2, kSplitWarps, true>
                      : s.cpw <= 3 ? rms_bwd_kernel<3, kSplitWarps, true> : rms_bwd_kernel<4, kSplitWarps, true>;
  PdlLaunch lc(dim3(s.groups, s.parts ? s.parts : 1), dim3((s.parts ? kSplitWarps : kNormWarps) * 32), 0, st, s.parts > 1 ? 1 : 0, s.parts > 1 ? s.parts : 0);
  NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, kernel, dyp, lddy, gscale, x, dl, w, rstd, dres, out, o16, M, D, ba, bb, s.parts ? s.chunks : static_cast<int>((D + 31) / 32)));
  return NF4LL_OK;
}
