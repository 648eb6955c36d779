// The skinny (rank-16) LoRA products around the fused linear, as small tensor-core GEMMs:
//   lora_down   t[M,16]  = drop(x)[M,C] . R^T,  R = lora_A [16,C]      (forward: T)
//                                               R = lora_B^T [16,C]    (backward: U = dy . B)
//   lora_grads  dA[16,K] (+)= u^T . drop(x),  dB[N,16] (+)= scale * dy^T . t
// Replaces solution/fast_qwen.py:943-944 and 1369-1374 of the reference. Accumulation is fp32 and
// t / u stay fp32 between the passes (split into fp16 hi + lo parts where they feed a tensor-core
// operand): the reference rounds them (and dA/dB) to fp16, which costs up to 0.08 absolute error on
// gradients of magnitude ~100.
//
// Both kernels are bandwidth-bound passes over x / dy (32 multiply-adds per fp16 element read), so
// they use warp-level mma.sync.m16n8k16 with operands loaded straight from global memory with
// 128-bit loads; there is nothing for TMA staging or tensor memory to win here.
#include "nf4ll_lora.cuh"

namespace nf4ll {

// ---------------------------------------------------------------------------------------------
// Row reduction: t[M,16] = scale * drop(act)[M,C] . R^T with R [16,C] row-major fp16.
// One CTA = 8*RG rows x a range of the contraction, 8 warps; warp w takes the 32-column chunks
// w, w+8, ... of the range. Per chunk a lane issues RG 128-bit loads of act (rows g, g+8, ...) and
// two of R (rank rows g and g+8); a lane's 8 consecutive columns feed two MMAs with the SAME
// column-to-slot assignment on both operands, so no shuffle or shared-memory transpose is needed:
// out^T[16 ranks, 8 rows] = R[16, k] . act^T[k, 8 rows]. The warps' partial results are summed
// through shared memory. The contraction is split over grid.y so that every SM has loads in
// flight; how the parts of one row block meet depends on COMBINE:
//   kDownDirect   grid.y == 1, plain stores;
//   kDownCluster  the grid.y CTAs of a row block form one thread-block cluster (at most 8); after a
//                 cluster barrier rank 0 adds the others' partial sums out of their shared memory in
//                 rank order and stores: no zero-fill, no atomics, bit-reproducible;
//   kDownAtomic   more than 8 parts (few rows, long contraction): fp32 atomics into t, which the
//                 launcher zeroes first.
// `zero_words` 32-bit words at `zero_ptr` are cleared by CTA (0,0): the caller's next kernel (the
// split-K GEMM this product feeds) finds its tile counters reset without a separate memset.
// ---------------------------------------------------------------------------------------------
constexpr int kDownWarps = 8;
constexpr int kDownDirect = 0, kDownCluster = 1, kDownAtomic = 2;

__device__ __forceinline__ uint32_t down_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ float down_peer_load(const float* local, uint32_t rank) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(local)), r;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(r) : "memory");
  return v;
}

// drop8 value by value. The kernel of short batches, all latency, is the faster one with it even without a mask (the code around the loads
// comes out otherwise): with drop8 1 x 27648 under a mask takes 5.4 us, so 5.0, 16 x 5120 2.95 / 2.75, 1 x 1024 without a mask 2.15 /
// 2.03; with 32 rows per CTA and from one CTA per SM on drop8 is (64 x 27648 7.0 / 7.6, 1900 x 8960 14.9 / 16.8).
__device__ __forceinline__ uint4 drop8_short(uint4 raw, uint2 m, float keep_scale) {
  uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  const uint32_t mw[2] = {m.x, m.y};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
    const uint32_t pair = mw[j >> 1] >> (16 * (j & 1));
    w[j] = pack_half2_rn(pair & 0xffu ? v.x * keep_scale : 0.f, pair & 0xff00u ? v.y * keep_scale : 0.f);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <int RG, int COMBINE, int NW>
__global__ void __launch_bounds__(NW * 32)
lora_down_kernel(const __half* __restrict__ act, int64_t ldact, const DownBranch first, const DownBranch second, float scale, int64_t M, int64_t C,
                 int64_t c_per_cta, int* __restrict__ zero_ptr, int zero_words) {
  pdl_wait();
  pdl_launch_dependents();
  // Two branches in one launch only where a row's sum is cut up (short batches). The choice costs registers that the direct variant's
  // loads need: with it 2048 x 8960 / 16384 x 18944 under a mask take 21.0 / 230 us, without 16.0 / 178.
  const DownBranch& br = COMBINE != kDownDirect && blockIdx.z ? second : first;
  const uint8_t* __restrict__ mask = br.mask;
  const __half* __restrict__ R = br.R;
  float* __restrict__ t32 = br.t32;
  const int64_t ld_mask = br.ld_mask;
  const float keep_scale = br.keep_scale;
  constexpr int ROWS = 8 * RG;
  __shared__ float part[NW][ROWS][17];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
    for (int i = threadIdx.x; i < zero_words; i += NW * 32) zero_ptr[i] = 0;
  }
  const int64_t m0 = static_cast<int64_t>(blockIdx.x) * ROWS;
  const int64_t c_begin = static_cast<int64_t>(blockIdx.y) * c_per_cta;
  const int64_t c_end = (c_begin + c_per_cta < C) ? c_begin + c_per_cta : C;
  const __half* ap[RG];
  const uint8_t* mp[RG];
  bool ok[RG];
#pragma unroll
  for (int i = 0; i < RG; ++i) {
    const int64_t row = m0 + g + 8 * i;
    ok[i] = row < M;
    ap[i] = act + (ok[i] ? row : 0) * ldact;
    mp[i] = mask ? mask + (ok[i] ? row : 0) * ld_mask : nullptr;
  }
  const __half* r0p = R + static_cast<int64_t>(g) * C;
  const __half* r1p = R + static_cast<int64_t>(g + 8) * C;
  float c[RG][4];
#pragma unroll
  for (int i = 0; i < RG; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) c[i][j] = 0.f;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  // U chunks per trip, every load of the trip issued before the first use: the loop is bound by the
  // number of bytes a warp keeps in flight, not by arithmetic
  constexpr int U = RG <= 2 ? 4 : 2;
  for (int64_t k0 = c_begin + static_cast<int64_t>(warp) * 32 + t * 8; k0 < c_end; k0 += U * NW * 32) {
    uint4 x[U][RG], ra[U], rb[U];
    uint2 mk[U][RG];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t k = k0 + u * NW * 32;
      const bool in = k < c_end;
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        x[u][i] = (in && ok[i]) ? __ldg(reinterpret_cast<const uint4*>(ap[i] + k)) : zero;
        mk[u][i] = (in && mask) ? __ldg(reinterpret_cast<const uint2*>(mp[i] + k)) : make_uint2(0, 0);
      }
      ra[u] = in ? __ldg(reinterpret_cast<const uint4*>(r0p + k)) : zero;
      rb[u] = in ? __ldg(reinterpret_cast<const uint4*>(r1p + k)) : zero;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (mask) {
#pragma unroll
        for (int i = 0; i < RG; ++i) x[u][i] = COMBINE == kDownDirect || RG == 4 ? drop8(x[u][i], mk[u][i], keep_scale) : drop8_short(x[u][i], mk[u][i], keep_scale);
      }
      // columns k..k+3 -> MMA slots (2t, 2t+1, 2t+8, 2t+9) of the first MMA, k+4..k+7 of the second
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        mma16816(c[i], ra[u].x, rb[u].x, ra[u].y, rb[u].y, x[u][i].x, x[u][i].y);
        mma16816(c[i], ra[u].z, rb[u].z, ra[u].w, rb[u].w, x[u][i].z, x[u][i].w);
      }
    }
  }
  // accumulator layout: c[.][0], c[.][1] = (rank g, rows 2t, 2t+1); c[.][2], c[.][3] = (rank g+8, same rows)
#pragma unroll
  for (int i = 0; i < RG; ++i) {
    part[warp][8 * i + 2 * t][g] = c[i][0];      part[warp][8 * i + 2 * t + 1][g] = c[i][1];
    part[warp][8 * i + 2 * t][g + 8] = c[i][2];  part[warp][8 * i + 2 * t + 1][g + 8] = c[i][3];
  }
  __syncthreads();
  if (COMBINE == kDownCluster) {
    // every CTA folds its warps' parts into part[0]; rank 0 then gathers the cluster's
    for (int idx = threadIdx.x; idx < ROWS * 16; idx += NW * 32) {
      const int row = idx >> 4, j = idx & 15;
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < NW; ++w) v += part[w][row][j];
      part[0][row][j] = v;                       // read and written by this thread only
    }
    cluster_sync_all();
    if (down_cluster_rank() == 0) {
      for (int idx = threadIdx.x; idx < ROWS * 16; idx += NW * 32) {
        const int row = idx >> 4, j = idx & 15;
        if (m0 + row < M) {
          float v = part[0][row][j], peer[8];
#pragma unroll
          for (uint32_t r = 1; r < 8; ++r) peer[r] = r < gridDim.y ? down_peer_load(&part[0][row][j], r) : 0.f;      // all in flight at once
#pragma unroll
          for (uint32_t r = 1; r < 8; ++r)
            if (r < gridDim.y) v += peer[r];
          t32[(m0 + row) * 16 + j] = v * scale;
        }
      }
    }
    cluster_sync_all();                         // peers keep their shared memory until rank 0 has read it
  } else {
    for (int idx = threadIdx.x; idx < ROWS * 16; idx += NW * 32) {
      const int row = idx >> 4, j = idx & 15;
      if (m0 + row < M) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < NW; ++w) v += part[w][row][j];
        if (COMBINE == kDownAtomic) atomicAdd(t32 + (m0 + row) * 16 + j, v * scale);
        else t32[(m0 + row) * 16 + j] = v * scale;
      }
    }
  }
}

// t16 = fp16(scale * t32), for callers of the stand-alone projection that want the fp16 copy
__global__ void scale_to_half_kernel(const float* __restrict__ t32, __half* __restrict__ t16, float scale, int64_t n) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) t16[i] = __float2half_rn(t32[i] * scale);
}

// B[N,16] -> Bt[16,N] (fp16), for callers that do not keep a transposed shadow of lora_B.
__global__ void transpose_n16_kernel(const __half* __restrict__ B, __half* __restrict__ Bt, int64_t N) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < N * 16) {
    const int64_t n = i >> 4;
    const int j = static_cast<int>(i & 15);
    Bt[j * N + n] = B[i];
  }
}

// fp16 shadows of fp32 masters: A [16,K] and B [N,16] rounded, B also transposed to [16,N]
__global__ void __launch_bounds__(256)
lora_shadow_kernel(const float* __restrict__ A, const float* __restrict__ B, int64_t K, int64_t N, __half* __restrict__ A16, __half* __restrict__ B16,
                   __half* __restrict__ Bt16) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x, first = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (int64_t i = first; i < K * 16; i += stride) A16[i] = __float2half_rn(A[i]);
  for (int64_t n = first; n < N; n += stride) {
    const float4* src = reinterpret_cast<const float4*>(B + n * 16);
    float v[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) { const float4 f = src[j]; v[4 * j] = f.x; v[4 * j + 1] = f.y; v[4 * j + 2] = f.z; v[4 * j + 3] = f.w; }
#pragma unroll
    for (int j = 0; j < 16; ++j) Bt16[j * N + n] = __float2half_rn(v[j]);
    uint4* dst = reinterpret_cast<uint4*>(B16 + n * 16);
    dst[0] = make_uint4(pack_half2_rn(v[0], v[1]), pack_half2_rn(v[2], v[3]), pack_half2_rn(v[4], v[5]), pack_half2_rn(v[6], v[7]));
    dst[1] = make_uint4(pack_half2_rn(v[8], v[9]), pack_half2_rn(v[10], v[11]), pack_half2_rn(v[12], v[13]), pack_half2_rn(v[14], v[15]));
  }
}

int transpose_n16_launch(const void* B, void* Bt, int64_t N, cudaStream_t stream) {
  const int64_t total = N * 16;
  count_launch();
  transpose_n16_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(
      static_cast<const __half*>(B), static_cast<__half*>(Bt), N);
  NF4LL_CUDA(cudaGetLastError());
  return NF4LL_OK;
}

// Clears 32-bit words that the next kernel counts in. A kernel and not a memset: it is launched while the kernel before it
// drains and the one after it while it runs (a split-K GEMM of 951 rows starts 3 us earlier).
__global__ void __launch_bounds__(256) zero_words_kernel(int* words, int n) {
  pdl_wait();
  pdl_launch_dependents();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) words[i] = 0;
}

int zero_words_launch(int* words, int n, cudaStream_t stream) {
  const int blocks = (n + 1023) / 1024;
  PdlLaunch lc(dim3(static_cast<unsigned>(blocks < 1 ? 1 : (blocks > 148 ? 148 : blocks))), dim3(256), 0, stream);
  NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, zero_words_kernel, words, n));
  return NF4LL_OK;
}

template <int RG, int COMBINE, int NW>
static int down_run(dim3 grid, unsigned cluster_y, const __half* a, int64_t ldact, const DownBranch* br, int n, float scale, int64_t M, int64_t C,
                    int64_t c_per_cta, int* zero_ptr, int zero_words, cudaStream_t stream) {
  const int launches = COMBINE == kDownDirect ? n : 1;
  grid.z = static_cast<unsigned>(n / launches);
  for (int i = 0; i < launches; ++i) {
    PdlLaunch lc(grid, dim3(NW * 32), 0, stream, cluster_y ? 1 : 0, cluster_y);
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, lora_down_kernel<RG, COMBINE, NW>, a, ldact, br[i], br[n - 1], scale, M, C, c_per_cta, zero_ptr,
                                  i == 0 ? zero_words : 0));
  }
  return NF4LL_OK;
}

// t32 (fp32 [M,16]) = scale * (drop(act) . R^T), R [16,C] row-major, for one branch or for two over the same rows, in one launch
// where the rows are few (q and v of a layer, gate and up: a second launch cost a decoded layer 4 us). `zero_ptr` / `zero_words`: optional 32-bit words
// the kernel clears on the way (see the kernel).
// How many parts of the contraction a batch that does not fill the SMs with rows is cut into, and columns of a part
static int64_t down_parts(int64_t M, int64_t C, int n, int sms, int64_t* c_per_cta) {
  const int64_t units = (C + kDownWarps * 32 - 1) / (kDownWarps * 32);     // 256-column units
  int64_t ks = (2 * static_cast<int64_t>(sms)) / ((M + 31) / 32 * n);      // at most two CTAs per SM: one wave, no tail
  if (ks > units) ks = units;
  if (ks < 1) ks = 1;
  // decode-sized batches are all latency: eight CTAs in one cluster (no zero-fill, no atomics) beat more CTAs + a memset
  if (ks > 8 && M * C <= (int64_t(1) << 21)) ks = 8;
  *c_per_cta = (units + ks - 1) / ks * (kDownWarps * 32);
  return (C + *c_per_cta - 1) / *c_per_cta;
}

int lora_down_ctas(int64_t M, int64_t C, int n, int sms) {
  int64_t c_per_cta = 0;
  return static_cast<int>((M + 7) / 8 * down_parts(M, C, n, sms, &c_per_cta) * n);
}

int lora_down_launch(const void* act, int64_t ldact, const DownBranch* br, int n, float scale, int64_t M, int64_t C, int* zero_ptr, int zero_words,
                     cudaStream_t stream) {
  if (M == 0) {
    if (zero_words > 0) NF4LL_CUDA(cudaMemsetAsync(zero_ptr, 0, sizeof(int) * zero_words, stream));
    return NF4LL_OK;
  }
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const __half* a = static_cast<const __half*>(act);
  const int64_t groups16 = (M + 15) / 16;
  if (groups16 * 4 >= 3 * static_cast<int64_t>(sms)) {
    // enough rows for (nearly) one CTA per SM at 16 rows each: a CTA takes the whole contraction and stores its rows directly. Sixteen warps
    // deep where each SM has one CTA; of more rows an SM holds two CTAs of eight warps or four of four, one of which computes or ends
    // while the others' loads are on their way. Under a mask / without, us, sixteen warps against this: 4096 x 8960 29.0 / 21.3 -> 23.7 / 17.0 (four
    // warps 31.1 / 23.5), 8192 x 3584 28.2 / 20.4 -> 19.1 / 14.0 (eight 21.6 / 15.7), 16384 x 3584 48.4 / 34.6 -> 34.4 / 25.2, 16384 x 18944 178 / 126 ->
    // 162 / 115; 2048 x 8960 16.0 / 11.8 with sixteen, 18.5 / 13.7 with eight.
    const dim3 grid(static_cast<unsigned>(groups16), 1);
    if (groups16 <= sms) return down_run<2, kDownDirect, 16>(grid, 0, a, ldact, br, n, scale, M, C, C, zero_ptr, zero_words, stream);
    if (groups16 <= 2 * static_cast<int64_t>(sms)) return down_run<2, kDownDirect, 8>(grid, 0, a, ldact, br, n, scale, M, C, C, zero_ptr, zero_words, stream);
    return down_run<2, kDownDirect, 4>(grid, 0, a, ldact, br, n, scale, M, C, C, zero_ptr, zero_words, stream);
  }
  const int64_t row_groups = (M + 31) / 32;
  int64_t c_per_cta = 0;
  const int64_t ks = down_parts(M, C, n, sms, &c_per_cta);
  const dim3 grid(static_cast<unsigned>(row_groups), static_cast<unsigned>(ks));
  if (ks == 1) return down_run<4, kDownDirect, kDownWarps>(grid, 0, a, ldact, br, n, scale, M, C, c_per_cta, zero_ptr, zero_words, stream);
  if (ks <= 8) {
    // Fewer rows per CTA while the grid stays within two CTAs per SM: more CTAs, each with more of its loads in flight. But not
    // where the kernel for middling batches streams a long contraction's weights meanwhile: it needs whole SMs, and the fewer
    // this one holds the better. Both kernels, 32 rows per CTA / fewer, us: 5120 x 27648 at 32, 64, 128 rows 43.8 / 47.2, 47.3 / 52.8,
    // 56.9 / 57.0, 3584 x 18944 at 64 and 96 rows 28.8 / 31.1 and 30.2 / 35.4, 8192 x 28672 at 64 rows 66.0 / 69.4, 1536 x 17920 at 96 rows
    // 20.6 / 24.5 (but at 187 and 333 rows 33.5 / 31.3 and 38.7 / 36.4, the worst of 33 calls beyond 128 rows), backward over the same
    // contractions alike. With shorter ones this kernel's own time tells: 4096 x 14336 at 64 and 128 rows 35.4 / 29.9 and 38.5 / 33.2,
    // 2048 x 11008 at 128 rows 29.8 / 25.9 (5120 x 5120 at 128 rows 19.6 / 21.6).
    const int64_t groups8 = (M + 7) / 8;
    const unsigned k = static_cast<unsigned>(ks);
    const bool aside = M > 16 && C > 16384;
    if (!aside && groups8 * ks * n <= 2 * static_cast<int64_t>(sms))
      return down_run<1, kDownCluster, kDownWarps>(dim3(static_cast<unsigned>(groups8), k), k, a, ldact, br, n, scale, M, C, c_per_cta, zero_ptr, zero_words, stream);
    if (!aside && groups16 * ks * n <= 2 * static_cast<int64_t>(sms))
      return down_run<2, kDownCluster, kDownWarps>(dim3(static_cast<unsigned>(groups16), k), k, a, ldact, br, n, scale, M, C, c_per_cta, zero_ptr, zero_words, stream);
    return down_run<4, kDownCluster, kDownWarps>(grid, k, a, ldact, br, n, scale, M, C, c_per_cta, zero_ptr, zero_words, stream);
  }
  for (int i = 0; i < n; ++i) NF4LL_CUDA(cudaMemsetAsync(br[i].t32, 0, sizeof(float) * 16 * M, stream));
  count_launch();
  lora_down_kernel<4, kDownAtomic, kDownWarps><<<dim3(grid.x, grid.y, n), kDownWarps * 32, 0, stream>>>(a, ldact, br[0], br[n - 1], scale, M, C,
                                                                                                    c_per_cta, zero_ptr, zero_words);
  NF4LL_CUDA(cudaGetLastError());
  return NF4LL_OK;
}

int lora_down_launch(const void* act, int64_t ldact, const uint8_t* mask, int64_t ld_mask, float keep_scale,
                     const void* R, float scale, int64_t M, int64_t C, void* t32, int* zero_ptr, int zero_words,
                     cudaStream_t stream) {
  const DownBranch one{mask, ld_mask, keep_scale, static_cast<const __half*>(R), static_cast<float*>(t32)};
  return lora_down_launch(act, ldact, &one, 1, scale, M, C, zero_ptr, zero_words, stream);
}

// ---------------------------------------------------------------------------------------------
// Column reduction: out[c][j] (+)= scale * sum_m drop(act)[m][c] * side[m][j]   (j < 16)
// as out^T[16, C] = side^T[16, M] . drop(act)[M, C]. One CTA = 64 columns x a range of rows, 4
// warps. The rows arrive in 64-row stages through a ring of shared-memory buffers filled by
// cp.async (act, mask and side as they lie in memory, two stages always in flight per CTA and four CTAs per SM: the kernel is
// a pass over act at memory speed). A warp fetches its own sixteen rows of every stage, applies the dropout to them in place,
// splits their side values into fp16 hi + lo fragments in registers (two MMAs recover ~22 mantissa bits) and contracts them
// against all 64 columns (ldmatrix.trans delivers the row-major act tile as the MMA's k-by-n operand), so that the warps of a CTA
// meet once, at the end: with three block barriers per stage and the side transposed through shared memory 2048 rows of
// 8960 + 1536 columns took 21.3 us (dropout on the 1536) and 24.0 (on the 8960) with operands out of HBM, 18.2 and 21.6 now; 21.0 and 23.5
// with operands in L2, 17.1 and 20.0 now. The three of them in an MLP block's step at 2048 rows: 578 us with the former kernel, 568 with this. Row ranges
// of different CTAs are combined with fp32 atomics, so the summation order across ranges is not fixed.
// out index = j * ld_j + c * ld_c: dA[16,K] uses (K, 1), dB[N,16] uses (1, 16).
// ---------------------------------------------------------------------------------------------
constexpr int kGradThreads = 128;
constexpr int kGradCols = 64;
constexpr int kGradStage = 64;
constexpr int kGradRing = 3;
constexpr int kActStride = 72;     // halves per shared row: 144 B keeps ldmatrix rows on distinct banks
constexpr int kGradActBytes = kGradStage * kActStride * 2;
constexpr int kGradMaskBytes = kGradStage * kGradCols;
constexpr int kSideStride = 20;    // floats per shared row of side: a fragment's reads fall on distinct banks
constexpr int kGradSideBytes = kGradStage * kSideStride * 4;
constexpr int kGradStageBytes = kGradActBytes + kGradMaskBytes + kGradSideBytes;
constexpr int kGradSmemBytes = kGradRing * kGradStageBytes;
static_assert(4 * 16 * (kGradCols + 1) * 4 <= kGradRing * kGradStageBytes, "the final reduction reuses the ring");

// One column reduction. A launch carries several of them (dA and dB of one projection or of three): column
// tiles [end[i-1], end[i]) of the grid belong to problem i.
struct GradProblem {
  const __half* act;
  int64_t ldact;
  const uint8_t* mask;
  int64_t ld_mask;
  float keep_scale;
  const float* side;
  float scale;
  int64_t C;
  int64_t rows_per_cta;
  float* out;
  int64_t ld_j, ld_c;
};

constexpr int kGradProblems = 6;
template <int P>
struct GradBatch {
  GradProblem problem[P];
  int end[P];
};

// P = 2 for one projection: a CTA's fields come out of either of two constants. Read at an index that is looked up, as of six, they cost each
// launch 0.1 us and long batches more: 17 rows of 1536 + 1536 columns 2.75 us, 2.82 so, 8192 of 3584 + 18944 126 and 130.
template <int P>
__global__ void __launch_bounds__(kGradThreads, 4)
lora_grad_kernel(const __grid_constant__ GradBatch<P> batch, int64_t M) {
  pdl_wait();
  pdl_launch_dependents();
  int which = 0;
  if (P == 2) which = static_cast<int>(blockIdx.x) >= batch.end[0] ? 1 : 0;
  else while (static_cast<int>(blockIdx.x) >= batch.end[which]) ++which;
  const GradProblem& pb = P == 2 ? (which ? batch.problem[1] : batch.problem[0]) : batch.problem[which];
  const __half* __restrict__ act = pb.act;
  const int64_t ldact = pb.ldact;
  const uint8_t* __restrict__ mask = pb.mask;
  const int64_t ld_mask = pb.ld_mask;
  const float keep_scale = pb.keep_scale;
  const float* __restrict__ side = pb.side;
  const float scale = pb.scale;
  const int64_t C = pb.C, rows_per_cta = pb.rows_per_cta;
  float* __restrict__ out = pb.out;
  const int64_t ld_j = pb.ld_j, ld_c = pb.ld_c;
  if (static_cast<int64_t>(blockIdx.y) * rows_per_cta >= M) return;      // this reduction has fewer row ranges than the other
  extern __shared__ __align__(16) uint8_t g_smem[];
  const uint32_t ring = smem_u32(g_smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int64_t c0 = static_cast<int64_t>(static_cast<int>(blockIdx.x) - (which == 0 ? 0 : P == 2 ? batch.end[0] : batch.end[which - 1])) * kGradCols;
  const int64_t r_begin = static_cast<int64_t>(blockIdx.y) * rows_per_cta;
  const int64_t r_end = (r_begin + rows_per_cta < M) ? r_begin + rows_per_cta : M;
  float acc[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;

  const int kb = warp * 16;        // this warp's sixteen rows of a stage
  // its part of a stage of loads: 16 rows x (128 B of act, 64 B of mask, 64 B of side), one commit group
  auto issue = [&](int64_t r0, int slot) {
    const uint32_t base = ring + slot * kGradStageBytes;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = lane + i * 32;
      const int r = kb + (idx >> 3), ch = idx & 7;
      const int64_t row = r0 + r, col = c0 + ch * 8;
      const bool v = row < r_end && col < C;
      cp_async16(base + r * (kActStride * 2) + ch * 16, v ? act + row * ldact + col : act, v);
    }
    if (mask) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int idx = lane + i * 32;
        const int r = kb + (idx >> 2), ch = idx & 3;
        const int64_t row = r0 + r, col = c0 + ch * 16;
        const bool v = row < r_end && col < C;
        cp_async16(base + kGradActBytes + r * kGradCols + ch * 16, v ? mask + row * ld_mask + col : mask, v);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int idx = lane + i * 32;
      const int r = kb + (idx >> 2), ch = idx & 3;
      const bool v = r0 + r < r_end;
      cp_async16(base + kGradActBytes + kGradMaskBytes + r * (kSideStride * 4) + ch * 16, v ? side + (r0 + r) * 16 + ch * 4 : side, v);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s0 = 0; s0 < kGradRing - 1; ++s0) issue(r_begin + s0 * kGradStage, s0);
  int it = 0;
  for (int64_t r0 = r_begin; r0 < r_end; r0 += kGradStage, ++it) {
    issue(r0 + (kGradRing - 1) * kGradStage, (it + kGradRing - 1) % kGradRing);   // past the range: empty, zero-filled
    cp_async_wait<kGradRing - 1>();
    __syncwarp();
    uint8_t* st = g_smem + (it % kGradRing) * kGradStageBytes;
    if (mask) {
      // dropout in place: 16 rows x 8 chunks of 8 columns over the warp
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int idx = lane + i * 32;
        const int r = kb + (idx >> 3), ch = idx & 7;
        uint4* ap = reinterpret_cast<uint4*>(st + r * (kActStride * 2) + ch * 16);
        const uint2 m = *reinterpret_cast<const uint2*>(st + kGradActBytes + r * kGradCols + ch * 8);
        *ap = drop8(*ap, m, keep_scale);
      }
      __syncwarp();
    }
    const float* sd = reinterpret_cast<const float*>(st + kGradActBytes + kGradMaskBytes) + (kb + 2 * t) * kSideStride + g;
    uint32_t ah0, ah1, ah2, ah3, al0, al1, al2, al3;
    split_half2(sd[0], sd[kSideStride], ah0, al0);
    split_half2(sd[8], sd[kSideStride + 8], ah1, al1);
    split_half2(sd[8 * kSideStride], sd[9 * kSideStride], ah2, al2);
    split_half2(sd[8 * kSideStride + 8], sd[9 * kSideStride + 8], ah3, al3);
    const uint32_t act_base = ring + (it % kGradRing) * kGradStageBytes;
#pragma unroll
    for (int np = 0; np < 4; ++np) {     // pairs of 8-column tiles
      // matrices: (k 0-7, n 0-7), (k 8-15, n 0-7), (k 0-7, n 8-15), (k 8-15, n 8-15) of this pair
      const int mrow = kb + ((lane >> 3) & 1) * 8 + (lane & 7);
      const int mcol = np * 16 + (lane >> 4) * 8;
      uint32_t b0, b1, b2, b3;
      ldmatrix_x4_trans(act_base + mrow * (kActStride * 2) + mcol * 2, b0, b1, b2, b3);
      mma16816(acc[2 * np], ah0, ah1, ah2, ah3, b0, b1);
      mma16816(acc[2 * np], al0, al1, al2, al3, b0, b1);
      mma16816(acc[2 * np + 1], ah0, ah1, ah2, ah3, b2, b3);
      mma16816(acc[2 * np + 1], al0, al1, al2, al3, b2, b3);
    }
    __syncwarp();                  // the slot is filled anew by the next trip
  }
  cp_async_wait<0>();
  __syncthreads();
  // combine the four warps' row slices (the ring is free now), then add into the output
  float (*s_red)[16][kGradCols + 1] = reinterpret_cast<float (*)[16][kGradCols + 1]>(g_smem);
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    s_red[warp][g][n * 8 + 2 * t] = acc[n][0];
    s_red[warp][g][n * 8 + 2 * t + 1] = acc[n][1];
    s_red[warp][g + 8][n * 8 + 2 * t] = acc[n][2];
    s_red[warp][g + 8][n * 8 + 2 * t + 1] = acc[n][3];
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 16 * kGradCols; idx += kGradThreads) {
    // dA (ld_c == 1): consecutive threads take consecutive columns; dB (ld_j == 1): consecutive ranks
    const int j = (ld_c == 1) ? idx / kGradCols : idx % 16;
    const int c = (ld_c == 1) ? idx % kGradCols : idx / 16;
    if (c0 + c < C) {
      const float v = s_red[0][j][c] + s_red[1][j][c] + s_red[2][j][c] + s_red[3][j][c];
      atomicAdd(out + j * ld_j + (c0 + c) * ld_c, v * scale);
    }
  }
}

struct GradPlan {
  int64_t col_tiles, msplit, rows_per;
};
static GradPlan grad_plan(int64_t M, int64_t C, int64_t sms, int64_t other_tiles) {
  GradPlan g;
  g.col_tiles = (C + kGradCols - 1) / kGradCols;
  const int64_t stages = (M + kGradStage - 1) / kGradStage;
  // four CTAs per SM (shared memory): one wave over both reductions of the launch, no tail
  int64_t msplit = 4 * sms / (g.col_tiles + other_tiles);
  if (msplit > stages) msplit = stages;
  if (msplit < 1) msplit = 1;
  g.rows_per = (stages + msplit - 1) / msplit * kGradStage;
  g.msplit = (M + g.rows_per - 1) / g.rows_per;
  return g;
}

// For each of n projections dA = u^T . drop(x) (u carries the LoRA scale, reference solution/fast_qwen.py:1370-1371) and / or
// dB = scale * dy^T . t (fast_qwen.py:1369), all in one launch: row ranges are as long as one wave of CTAs over all of them allows.
template <int P>
static int lora_grads_run(const nf4ll_grad* grads, int n, int64_t M, cudaStream_t stream) {
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  NF4LL_CUDA(cudaFuncSetAttribute(lora_grad_kernel<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmemBytes));
  int64_t tiles = 0;
  for (int i = 0; i < n; ++i) tiles += (grads[i].dA ? (grads[i].K + kGradCols - 1) / kGradCols : 0) + (grads[i].dB ? (grads[i].N + kGradCols - 1) / kGradCols : 0);
  GradBatch<P> b{};
  int used = 0;
  int64_t ranges = 1, at = 0;
  auto add = [&](GradProblem pr) {
    const GradPlan g = grad_plan(M, pr.C, sms, tiles - (pr.C + kGradCols - 1) / kGradCols);
    pr.rows_per_cta = g.rows_per;
    at += g.col_tiles;
    b.problem[used] = pr;
    b.end[used++] = static_cast<int>(at);
    if (g.msplit > ranges) ranges = g.msplit;
  };
  for (int i = 0; i < n; ++i) {
    const nf4ll_grad& g = grads[i];
    if (g.dA) add(GradProblem{static_cast<const __half*>(g.x), g.ldx, g.mask, g.ld_mask, g.keep_scale, static_cast<const float*>(g.u), 1.0f, g.K, 0, static_cast<float*>(g.dA), g.K, 1});
    if (g.dB) add(GradProblem{static_cast<const __half*>(g.dy), g.lddy, nullptr, 0, 1.0f, static_cast<const float*>(g.t), g.scale, g.N, 0, static_cast<float*>(g.dB), 1, 16});
  }
  PdlLaunch lc(dim3(static_cast<unsigned>(tiles), static_cast<unsigned>(ranges)), dim3(kGradThreads), kGradSmemBytes, stream);
  NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, lora_grad_kernel<P>, b, M));
  return NF4LL_OK;
}
static int lora_grads_launch(const nf4ll_grad* grads, int n, int64_t M, cudaStream_t stream) {
  return n == 1 ? lora_grads_run<2>(grads, n, M, stream) : lora_grads_run<kGradProblems>(grads, n, M, stream);
}

static int clear_grad(const nf4ll_grad& g, cudaStream_t stream) {
  // gradients that lie back to back are cleared by one fill
  const bool joined = g.dA && g.dB && static_cast<float*>(g.dB) == static_cast<float*>(g.dA) + 16 * g.K;
  if (g.dA) NF4LL_CUDA(cudaMemsetAsync(g.dA, 0, sizeof(float) * 16 * (joined ? g.K + g.N : g.K), stream));
  if (g.dB && !joined) NF4LL_CUDA(cudaMemsetAsync(g.dB, 0, sizeof(float) * 16 * g.N, stream));
  return NF4LL_OK;
}

static int check_grad(const nf4ll_grad& g, const char* who) {
  if (g.N <= 0 || g.K <= 0 || g.N % 8 || g.K % 8) {
    set_detail("%s: N=%lld K=%lld (multiples of 8)", who, static_cast<long long>(g.N), static_cast<long long>(g.K));
    return NF4LL_ERR_SHAPE;
  }
  if (g.dA && (!g.x || !g.u)) { set_detail("%s: dA needs x and u", who); return NF4LL_ERR_NULL; }
  if (g.dB && (!g.dy || !g.t)) { set_detail("%s: dB needs dy and t", who); return NF4LL_ERR_NULL; }
  auto off = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
  if ((g.dA && (off(g.x) || g.ldx % 8 || off(g.u) || (g.mask && (off(g.mask) || g.ld_mask % 16)))) || (g.dB && (off(g.dy) || g.lddy % 8 || off(g.t)))) {
    set_detail("%s: activations, t and u 16-byte aligned, leading dimensions multiples of 8; mask 16-byte aligned, ld_mask multiple of 16", who);
    return NF4LL_ERR_ALIGN;
  }
  return NF4LL_OK;
}

// ---------------------------------------------------------------------------------------------
// out[M,K] = fp16(sum over branches of drop(u . A)), A [16,K] fp16, u [M,16] fp32 (in two fp16 parts under a power of two per row: 22 bits
// of every rank down to 2^-17 of the row's largest, of smaller ones what is above 2^-39 of it), under the keep-mask of
// the branch's input: the LoRA terms of d(input) of projections that share an input, whose base terms one product adds to it. Two of
// them could not share a GEMM's epilogue otherwise (two masks on one tile). A CTA takes 64 columns, whose factors its warps
// keep in registers, and goes through blocks of sixteen rows. 2 B written and 1 B of mask read per branch and element.
// ---------------------------------------------------------------------------------------------
constexpr int kExpandWarps = 4, kExpandCols = 64;
struct ExpandBranch {
  const float* u;
  const __half* A;
  const uint8_t* mask;
  int64_t ld_mask;
  float keep_scale;
};

template <int N>
__global__ void __launch_bounds__(kExpandWarps * 32)
lora_expand_kernel(const ExpandBranch first, const ExpandBranch second, __half* __restrict__ out, int64_t ldo, int64_t M, int64_t K) {
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * kExpandCols;
  // Tile j of a group of 32 columns holds columns 8 i + 2 j, + 1 for i = 0..3, so that lane (g, t) ends with columns 8 t .. 8 t + 7 of
  // its rows in registers: 16-byte stores, 8-byte reads of the mask, and of lora_A 16 bytes of a rank's
  // row, which movmatrix turns into the right operand (with two-byte loads instead, 64 a lane, 951 / 2048 rows of 1536 took 5.8 / 7.5 us, now 3.9 / 6.3)
  constexpr int kGroups = kExpandCols / 32;
  uint32_t b0[N][kGroups][4], b1[N][kGroups][4];   // ranks 2 t, 2 t + 1 and + 8 of the tile's column g
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const __half* A = n ? second.A : first.A;
#pragma unroll
    for (int q = 0; q < kGroups; ++q) {
      const int64_t c = c0 + 32 * q + 8 * t;
      const uint4 zero = make_uint4(0, 0, 0, 0);
      const uint4 lo = c < K ? __ldg(reinterpret_cast<const uint4*>(A + static_cast<int64_t>(g) * K + c)) : zero;
      const uint4 hi = c < K ? __ldg(reinterpret_cast<const uint4*>(A + static_cast<int64_t>(g + 8) * K + c)) : zero;
      const uint32_t p0[4] = {lo.x, lo.y, lo.z, lo.w}, p1[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b0[n][q][j] = transpose8x8(p0[j]);
        b1[n][q][j] = transpose8x8(p1[j]);
      }
    }
  }
  const int64_t step = static_cast<int64_t>(gridDim.y) * kExpandWarps * 16;
  for (int64_t m0 = (static_cast<int64_t>(blockIdx.y) * kExpandWarps + warp) * 16; m0 < M; m0 += step) {
    const int64_t row[2] = {m0 + g, m0 + g + 8};
    float v[kGroups][2][8];                        // columns 8 t .. 8 t + 7 of each row
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const ExpandBranch& br = n ? second : first;
      uint32_t part[4][2];                         // (row g, ranks 2t..), (row g + 8, same), (row g, ranks 2t + 8..), (row g + 8, same)
      float back[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 zero = make_float2(0.f, 0.f);
        const float2* u = reinterpret_cast<const float2*>(br.u + row[i] * 16 + 2 * t);
        const float2 a = row[i] < M ? __ldcg(u) : zero, b = row[i] < M ? __ldcg(u + 4) : zero;
        const RowScale f = row_scale(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))));
        split_parts(a.x * f.to, a.y * f.to, part[i]);
        split_parts(b.x * f.to, b.y * f.to, part[i + 2]);
        back[i] = br.mask ? f.back * br.keep_scale : f.back;
      }
      uint2 keep[kGroups][2];
#pragma unroll
      for (int q = 0; q < kGroups; ++q)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int64_t c = c0 + 32 * q + 8 * t;
          keep[q][i] = br.mask && row[i] < M && c < K ? __ldg(reinterpret_cast<const uint2*>(br.mask + row[i] * br.ld_mask + c)) : make_uint2(0, 0);
        }
#pragma unroll
      for (int q = 0; q < kGroups; ++q)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < 2; ++i) mma16816(c, part[0][i], part[1][i], part[2][i], part[3][i], b0[n][q][j], b1[n][q][j]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int e = 2 * j + (i & 1);
            const uint32_t k = (e < 4 ? keep[q][i >> 1].x : keep[q][i >> 1].y) & 0xffu << 8 * (e & 3);
            const float d = !br.mask || k ? c[i] * back[i >> 1] : 0.f;
            v[q][i >> 1][e] = n ? v[q][i >> 1][e] + d : d;
          }
        }
    }
#pragma unroll
    for (int q = 0; q < kGroups; ++q)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int64_t c = c0 + 32 * q + 8 * t;
        if (row[i] < M && c < K) *reinterpret_cast<uint4*>(out + row[i] * ldo + c) = pack8(v[q][i]);
      }
  }
}

}  // namespace nf4ll

extern "C" int nf4ll_lora_down(const void* x, int64_t ldx, const uint8_t* mask, int64_t ld_mask, float keep_scale,
                               const void* A, float scale, int32_t r, int64_t M, int64_t K, void* t32, void* t16,
                               void* stream) {
  using namespace nf4ll;
  if (r != 16) { set_detail("nf4ll_lora_down: rank %d", r); return NF4LL_ERR_RANK; }
  if (!x || !A) { set_detail("nf4ll_lora_down: null pointer"); return NF4LL_ERR_NULL; }
  if (M < 0 || K <= 0 || K % 8) { set_detail("nf4ll_lora_down: M=%lld K=%lld", (long long)M, (long long)K); return NF4LL_ERR_SHAPE; }
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(A) & 15) || ldx % 8 ||
      (mask && ((reinterpret_cast<uintptr_t>(mask) & 15) || ld_mask % 16))) {
    set_detail("nf4ll_lora_down: x/A 16-byte aligned, ldx multiple of 8, mask 16-byte aligned with ld_mask multiple of 16");
    return NF4LL_ERR_ALIGN;
  }
  if (int rc = require_sm100()) return rc;
  if (!t32) { set_detail("nf4ll_lora_down: t32 is required (t16 is optional)"); return NF4LL_ERR_NULL; }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (int rc = lora_down_launch(x, ldx, mask, ld_mask, keep_scale, A, 1.0f, M, K, t32, nullptr, 0, st)) return rc;
  if (t16 && M > 0) {
    const int64_t n = M * 16;
    count_launch();
    scale_to_half_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(static_cast<const float*>(t32),
                                                                              static_cast<__half*>(t16), scale, n);
    NF4LL_CUDA(cudaGetLastError());
  }
  return NF4LL_OK;
}

extern "C" int nf4ll_lora_grads(const void* dy, int64_t lddy, const void* x, int64_t ldx, const uint8_t* mask,
                                int64_t ld_mask, float keep_scale, const void* t32, const void* u32, float scale,
                                int32_t r, int64_t M, int64_t N, int64_t K, void* dA, void* dB, int32_t accumulate,
                                void* stream_v) {
  using namespace nf4ll;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  if (r != 16) { set_detail("nf4ll_lora_grads: rank %d", r); return NF4LL_ERR_RANK; }
  if (M < 0) { set_detail("nf4ll_lora_grads: M=%lld", static_cast<long long>(M)); return NF4LL_ERR_SHAPE; }
  const nf4ll_grad one{dy, lddy, x, ldx, mask, ld_mask, keep_scale, t32, u32, scale, N, K, dA, dB};
  if (int rc = check_grad(one, "nf4ll_lora_grads")) return rc;
  if (int rc = require_sm100()) return rc;
  if (!accumulate)
    if (int rc = clear_grad(one, stream)) return rc;
  if (M > 0 && (dA || dB))
    if (int rc = lora_grads_launch(&one, 1, M, stream)) return rc;
  return NF4LL_OK;
}

extern "C" int nf4ll_lora_grads_batch(const nf4ll_grad* grads, int32_t n, int64_t M, int32_t accumulate, void* stream_v) {
  using namespace nf4ll;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
  const char* who = "nf4ll_lora_grads_batch";
  if (!grads) { set_detail("%s: null pointer", who); return NF4LL_ERR_NULL; }
  if (M < 0 || n < 1 || n > kGradProblems / 2) { set_detail("%s: M=%lld, %d projections (1..%d)", who, static_cast<long long>(M), n, kGradProblems / 2); return NF4LL_ERR_SHAPE; }
  bool any = false;
  for (int i = 0; i < n; ++i) {
    if (int rc = check_grad(grads[i], who)) return rc;
    if (grads[i].dA && grads[i].mask && grads[i].ld_mask < grads[i].K) { set_detail("%s: ld_mask must be >= K", who); return NF4LL_ERR_ALIGN; }
    any |= grads[i].dA || grads[i].dB;
  }
  if (!any) return NF4LL_OK;
  if (int rc = require_sm100()) return rc;
  for (int i = 0; i < n && !accumulate; ++i)
    if (int rc = clear_grad(grads[i], stream)) return rc;
  return M > 0 ? lora_grads_launch(grads, n, M, stream) : static_cast<int>(NF4LL_OK);
}

extern "C" int nf4ll_lora_expand(const nf4ll_expand* branches, int32_t n, int64_t M, int64_t K, void* out, int64_t ldo, void* stream) {
  using namespace nf4ll;
  const char* who = "nf4ll_lora_expand";
  if (!branches || !out) { set_detail("%s: null pointer", who); return NF4LL_ERR_NULL; }
  if (M < 0 || K <= 0 || K % 8 || n < 1 || n > 2) { set_detail("%s: M=%lld K=%lld, %d branches (1..2)", who, static_cast<long long>(M), static_cast<long long>(K), n); return NF4LL_ERR_SHAPE; }
  auto off = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
  ExpandBranch br[2]{};
  for (int i = 0; i < n; ++i) {
    const nf4ll_expand& b = branches[i];
    if (!b.u || !b.A) { set_detail("%s: a branch needs u and A", who); return NF4LL_ERR_NULL; }
    if (off(b.u) || off(b.A) || (b.mask && (off(b.mask) || b.ld_mask % 16 || b.ld_mask < K))) {
      set_detail("%s: u, A and mask 16-byte aligned, ld_mask a multiple of 16 and >= K", who);
      return NF4LL_ERR_ALIGN;
    }
    br[i] = ExpandBranch{static_cast<const float*>(b.u), static_cast<const __half*>(b.A), b.mask, b.ld_mask, b.keep_scale};
  }
  if (off(out) || ldo % 8 || ldo < K) { set_detail("%s: out 16-byte aligned, its leading dimension a multiple of 8 and >= K", who); return NF4LL_ERR_ALIGN; }
  if (M == 0) return NF4LL_OK;
  if (int rc = require_sm100()) return rc;
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // four CTAs per SM at most, each with a block of rows per warp at least
  const int64_t tiles = (K + kExpandCols - 1) / kExpandCols, blocks = (M + 16 * kExpandWarps - 1) / (16 * kExpandWarps);
  int64_t y = (4 * static_cast<int64_t>(sms) + tiles - 1) / tiles;
  y = y < blocks ? y : blocks;
  PdlLaunch lc(dim3(static_cast<unsigned>(tiles), static_cast<unsigned>(y)), dim3(kExpandWarps * 32), 0, static_cast<cudaStream_t>(stream));
  NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, n == 2 ? lora_expand_kernel<2> : lora_expand_kernel<1>, br[0], br[1], static_cast<__half*>(out), ldo, M, K));
  return NF4LL_OK;
}

extern "C" int nf4ll_lora_project(const void* x, int64_t ldx, const uint8_t* mask, int64_t ld_mask, float keep_scale, const void* A, float scale,
                                  int64_t M, int64_t K, void* t32, void* stream) {
  using namespace nf4ll;
  if (!x || !A || !t32) { set_detail("nf4ll_lora_project: null pointer"); return NF4LL_ERR_NULL; }
  if (M < 0 || K <= 0 || K % 8) { set_detail("nf4ll_lora_project: M=%lld K=%lld", (long long)M, (long long)K); return NF4LL_ERR_SHAPE; }
  if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(A) & 15) || ldx % 8 ||
      (mask && ((reinterpret_cast<uintptr_t>(mask) & 15) || ld_mask % 16))) {
    set_detail("nf4ll_lora_project: x/A 16-byte aligned, ldx multiple of 8, mask 16-byte aligned with ld_mask multiple of 16");
    return NF4LL_ERR_ALIGN;
  }
  if (int rc = require_sm100()) return rc;
  return lora_down_launch(x, ldx, mask, ld_mask, keep_scale, A, scale, M, K, t32, nullptr, 0, static_cast<cudaStream_t>(stream));
}

extern "C" int nf4ll_lora_shadow(const float* A, const float* B, int64_t K, int64_t N, void* A16, void* B16, void* Bt16, void* stream) {
  using namespace nf4ll;
  if (!A || !B || !A16 || !B16 || !Bt16) { set_detail("nf4ll_lora_shadow: null pointer"); return NF4LL_ERR_NULL; }
  if (K <= 0 || N <= 0) { set_detail("nf4ll_lora_shadow: K=%lld N=%lld", (long long)K, (long long)N); return NF4LL_ERR_SHAPE; }
  if ((reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(B16)) & 15) { set_detail("nf4ll_lora_shadow: B and B16 must be 16-byte aligned"); return NF4LL_ERR_ALIGN; }
  if (int rc = require_sm100()) return rc;
  const int64_t work = K * 16 > N ? K * 16 : N;
  const int64_t blocks = (work + 255) / 256 < 296 ? (work + 255) / 256 : 296;
  PdlLaunch lc(dim3(static_cast<unsigned>(blocks)), dim3(256), 0, static_cast<cudaStream_t>(stream));
  NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, lora_shadow_kernel, A, B, K, N, static_cast<__half*>(A16), static_cast<__half*>(B16), static_cast<__half*>(Bt16)));
  return NF4LL_OK;
}
