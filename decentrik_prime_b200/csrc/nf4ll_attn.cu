// Rotary embedding + causal grouped-query attention over packed varlen rows, forward and backward: what lies between the
// Q|K|V and O projections of a decoder layer (the reference has kernels of its own for it, solution/k_rope.py,
// k_attn.py). Head dimensions 64 and 128, fp16 in and out, fp32 softmax statistics and accumulation.
//
// What bounds it: launches and latency. A data loader's batch is a handful of sequences of tens to a few thousand rows; a
// 951-row batch at 12 heads is 0.8 GFLOP forward, so one kernel over all sequences and heads instead of a dozen launches
// per sequence is the whole gain (through PyTorch: 280 launches per layer and step). The contractions use mma.sync:
// tiles of 64 rows are too small to feed tcgen05, and at a few microseconds per launch there is nothing to win.
// Sequence boundaries travel in the kernel parameters, so no copy to the device is needed per batch.
// That holds for short sequences. One of 2048 rows, 28 heads, takes 624 us forward and backward (169 TFLOP/s, chained by the
// latencies of mma.sync and ldmatrix at eight warps per SM), one of 4096 rows 2158 (196); the caller
// (stack.py) takes other kernels for such batches.
//
//   rope     q, k rotated once into a buffer (a key row is read by every query tile after it)
//   forward  one CTA per 64 query rows and head, 4 warps of 16 rows, keys and values in 64-row blocks by cp.async; of long sequences
//            two times 4 warps, the blocks dealt out between them
//   dK, dV   a cluster of up to 8 CTAs per 64 key rows and key-value head, the group's query heads dealt out among them,
//            each looping over the later query rows; their sums meet through distributed shared memory in a fixed order. One
//            CTA for the whole group left most SMs idle: 951 rows, 12 heads of 128 in groups of 6, 115 us, 28 now
//   dQ       one CTA per 64 query rows and head, looping over the earlier key rows, shared out like the forward's
// The backward kernels rotate dQ and dK back in their epilogue (both halves of a rotated pair sit in one thread).
#include "nf4ll_pair.cuh"

namespace nf4ll {

constexpr int kAttnMaxSeqs = 128;            // sequences per launch (longer lists are cut)
constexpr int kAttnRows = 64;
constexpr int kAttnThreads = 128;

struct SeqTable {
  int n;
  int start[kAttnMaxSeqs + 1];               // first row of each sequence
  int tile[kAttnMaxSeqs + 1];                // tiles of 64 rows before each sequence
};

struct AttnParams {
  const __half* q;      // rotated [rows, ldr]: query heads, then key heads
  const __half* k;
  int64_t ldr;
  const __half* v;      // [rows, ldv]
  int64_t ldv;
  const __half* o;      // attention output [rows, ldo] (backward)
  __half* out;          // forward output
  int64_t ldo;
  const __half* dout;   // [rows, lddo]
  int64_t lddo;
  __half *dq, *dk, *dv; // [rows, ldd]
  int64_t ldd;
  float* lse;           // [heads, rows]: log2-sum-exp2 of the scaled scores
  float* delta;         // [heads, rows]: sum(dout * o)
  const float2* trig;   // [positions, hd / 2] (cos, sin)
  int heads, group;     // query heads, query heads per key-value head
  int64_t rows;
  float scale_log2, scale;
};

__device__ __forceinline__ void attn_cp16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void attn_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void attn_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A tile of ROWS x HD fp16 in shared memory: rows of HD * 2 bytes, 16-byte chunks XOR-swizzled by the row so that the
// ldmatrix rows of a matrix fall into different banks.
template <int HD>
__device__ __forceinline__ uint32_t tile_addr(uint32_t base, int row, int chunk) {
  return base + row * (HD * 2) + ((chunk ^ (row & 7)) << 4);
}
template <int HD, int ROWS, int THREADS = kAttnThreads>
__device__ __forceinline__ void load_tile(uint32_t base, const __half* src, int64_t ld, int row0, int end) {
  constexpr int CH = HD / 8;
#pragma unroll
  for (int i = 0; i < ROWS * CH / THREADS; ++i) {
    const int idx = threadIdx.x % THREADS + i * THREADS, r = idx / CH, c = idx % CH;
    const bool v = row0 + r < end;
    attn_cp16(tile_addr<HD>(base, r, c), v ? src + (row0 + r) * ld + c * 8 : src, v);
  }
}
// A fragment of rows r0 .. r0+15, columns 16 kk ..
template <int HD>
__device__ __forceinline__ void frag_a(uint32_t base, int r0, int kk, int lane, uint32_t (&a)[4]) {
  ldsm4(tile_addr<HD>(base, r0 + (lane & 15), kk * 2 + (lane >> 4)), a);
}
// B fragments of two 8-wide n-tiles (rows n0 .. n0+15 of a [n][k] tile), k columns 16 kk ..: b[0..1] first, b[2..3] second
template <int HD>
__device__ __forceinline__ void frag_b(uint32_t base, int n0, int kk, int lane, uint32_t (&b)[4]) {
  ldsm4(tile_addr<HD>(base, n0 + (lane & 7) + ((lane >> 4) << 3), kk * 2 + ((lane >> 3) & 1)), b);
}
// B fragments of two 8-wide n-tiles (columns n0 .. n0+15 of a [k][n] tile), k rows k0 .. k0+15
template <int HD>
__device__ __forceinline__ void frag_bt(uint32_t base, int k0, int n0, int lane, uint32_t (&b)[4]) {
  ldsm4t(tile_addr<HD>(base, k0 + (lane & 15), n0 / 8 + (lane >> 4)), b);
}

__device__ __forceinline__ void find_tile(const SeqTable& t, int tile, int& start, int& len, int& t0) {
  int lo = 0, hi = t.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.tile[mid] <= tile) lo = mid; else hi = mid - 1;
  }
  start = t.start[lo];
  len = t.start[lo + 1] - start;
  t0 = (tile - t.tile[lo]) * kAttnRows;
}

// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
rope_kernel(const __half* __restrict__ src, int64_t lds, __half* __restrict__ dst, int64_t ldd, const float2* __restrict__ trig, int heads,
            int hd, const __grid_constant__ SeqTable seqs) {
  pdl_wait();
  pdl_launch_dependents();
  const int half = hd / 2, per_row = heads * (half / 8);
  const int64_t work = static_cast<int64_t>(seqs.start[seqs.n] - seqs.start[0]) * per_row;      // may exceed 32 bits
  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; idx < work; idx += gridDim.x * 256) {
    const int r = static_cast<int>(work >> 32 ? idx / per_row : static_cast<uint32_t>(idx) / static_cast<uint32_t>(per_row));
    const int c = static_cast<int>(idx - static_cast<int64_t>(r) * per_row);
    const int head = c / (half / 8), j = (c - head * (half / 8)) * 8;
    const int row = seqs.start[0] + r;
    int lo = 0, hi = seqs.n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (seqs.start[mid] <= row) lo = mid; else hi = mid - 1;
    }
    const int pos = row - seqs.start[lo];
    const __half* s = src + row * lds + head * hd + j;
    float a[8], b[8], x[8], y[8];
    unpack8(*reinterpret_cast<const uint4*>(s), a);
    unpack8(*reinterpret_cast<const uint4*>(s + half), b);
    const float4* tp = reinterpret_cast<const float4*>(trig + static_cast<int64_t>(pos) * half + j);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 t = __ldg(tp + k);
      x[2 * k] = a[2 * k] * t.x - b[2 * k] * t.y;
      y[2 * k] = b[2 * k] * t.x + a[2 * k] * t.y;
      x[2 * k + 1] = a[2 * k + 1] * t.z - b[2 * k + 1] * t.w;
      y[2 * k + 1] = b[2 * k + 1] * t.z + a[2 * k + 1] * t.w;
    }
    __half* d = dst + row * ldd + head * hd + j;
    *reinterpret_cast<uint4*>(d) = pack8(x);
    *reinterpret_cast<uint4*>(d + half) = pack8(y);
  }
}

// ---------------------------------------------------------------------------------------------
template <int HD, int HALVES>
__global__ void __launch_bounds__(HALVES * kAttnThreads)
attn_fwd_kernel(const __grid_constant__ AttnParams p, const __grid_constant__ SeqTable seqs) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(128) uint8_t a_smem[];
  constexpr int TILE = kAttnRows * HD * 2, KS = HD / 16, NT = HD / 8;
  const int half = HALVES == 1 ? 0 : threadIdx.x / kAttnThreads, warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t sQ = smem_u32(a_smem), sK = sQ + TILE + half * 4 * TILE, sV = sK + 2 * TILE;
  int start, len, q0;
  find_tile(seqs, seqs.tile[seqs.n] - 1 - blockIdx.x, start, len, q0);      // later (longer) tiles first
  const int head = blockIdx.y, kvh = head / p.group;
  const __half* qp = p.q + start * p.ldr + head * HD;
  const __half* kp = p.k + start * p.ldr + kvh * HD;
  const __half* vp = p.v + start * p.ldv + kvh * HD;
  const int n_blocks = q0 / kAttnRows + 1;
  load_tile<HD, kAttnRows, HALVES * kAttnThreads>(sQ, qp, p.ldr, q0, len);
  auto load = [&](int b, int slot) {
    if (b < n_blocks) {
      load_tile<HD, kAttnRows>(sK + slot * TILE, kp, p.ldr, b * kAttnRows, len);
      load_tile<HD, kAttnRows>(sV + slot * TILE, vp, p.ldv, b * kAttnRows, len);
    }
    attn_commit();
  };
  auto sync = [&] {
    if (HALVES == 1) __syncthreads();
    else named_barrier(half + 1, kAttnThreads);       // the 128 threads of this half
  };
  load(half, 0);
  load(half + HALVES, 1);
  // below any finite score, and finite itself: a block whose scores are all -inf (keys that overflowed) adds nothing, wherever a chain starts
  float o[NT][4], m[2] = {-1e30f, -1e30f}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[n][i] = 0.f;
  const int row_a = q0 + warp * 16 + g;
  attn_wait<1>();
  __syncthreads();
  // the queries stay in registers where four warps have an SM's share of them (40 sequences of 30 rows 17.8 -> 16.4 us; with eight 81 -> 85
  // at 2048 rows, 12 heads)
  uint32_t qf[HALVES == 2 ? 1 : KS][4];
  if (HALVES == 1) {
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) frag_a<HD>(sQ, warp * 16, kk, lane, qf[kk]);
  }
  for (int b = half, slot = 0; b < n_blocks; b += HALVES, slot ^= 1) {
    const uint32_t kb = sK + slot * TILE, vb = sV + slot * TILE;
    float s[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[n][i] = 0.f;
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      if (HALVES == 2) frag_a<HD>(sQ, warp * 16, kk, lane, qf[0]);
      const uint32_t (&a)[4] = qf[HALVES == 2 ? 0 : kk];
#pragma unroll
      for (int n2 = 0; n2 < 4; ++n2) {
        uint32_t bf[4];
        frag_b<HD>(kb, n2 * 16, kk, lane, bf);
        mma16816(s[2 * n2], a[0], a[1], a[2], a[3], bf[0], bf[1]);
        mma16816(s[2 * n2 + 1], a[0], a[1], a[2], a[3], bf[2], bf[3]);
      }
    }
    if (b == n_blocks - 1) {                 // the diagonal block (rows past the sequence end are never keys of a live row)
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (b * kAttnRows + n * 8 + 2 * t + (i & 1) > row_a + (i >> 1) * 8) s[n][i] = -INFINITY;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float mx = -INFINITY;
#pragma unroll
      for (int n = 0; n < 8; ++n) mx = fmaxf(mx, fmaxf(s[n][2 * h], s[n][2 * h + 1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float mn = fmaxf(m[h], mx * p.scale_log2);
      const float corr = exp2_fast(m[h] - mn);
      m[h] = mn;
      float sum = 0.f;
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        s[n][2 * h] = exp2_fast(fmaf(s[n][2 * h], p.scale_log2, -mn));
        s[n][2 * h + 1] = exp2_fast(fmaf(s[n][2 * h + 1], p.scale_log2, -mn));
        sum += s[n][2 * h] + s[n][2 * h + 1];
      }
      l[h] = l[h] * corr + sum;
#pragma unroll
      for (int n = 0; n < NT; ++n) { o[n][2 * h] *= corr; o[n][2 * h + 1] *= corr; }
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const uint32_t a0 = pack_half2_rn(s[2 * kk][0], s[2 * kk][1]), a1 = pack_half2_rn(s[2 * kk][2], s[2 * kk][3]);
      const uint32_t a2 = pack_half2_rn(s[2 * kk + 1][0], s[2 * kk + 1][1]), a3 = pack_half2_rn(s[2 * kk + 1][2], s[2 * kk + 1][3]);
#pragma unroll
      for (int n2 = 0; n2 < NT / 2; ++n2) {
        uint32_t bf[4];
        frag_bt<HD>(vb, kk * 16, n2 * 16, lane, bf);
        mma16816(o[2 * n2], a0, a1, a2, a3, bf[0], bf[1]);
        mma16816(o[2 * n2 + 1], a0, a1, a2, a3, bf[2], bf[3]);
      }
    }
    sync();
    load(b + 2 * HALVES, slot);
    attn_wait<1>();
    sync();
  }
  if constexpr (HALVES == 2) {
    // the second half's sums through shared memory (its own key and value blocks have been read)
    attn_wait<0>();
    float* const other = reinterpret_cast<float*>(a_smem + TILE + 4 * TILE);       // [4 + o][thread], two planes of m and l first
    __syncthreads();
    const int tid = threadIdx.x % kAttnThreads;
    if (half) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        other[h * kAttnThreads + tid] = m[h];
        other[(2 + h) * kAttnThreads + tid] = l[h];
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) other[(4 + 4 * n + i) * kAttnThreads + tid] = o[n][i];
    }
    __syncthreads();
    if (half) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float m1 = other[h * kAttnThreads + tid], mn = fmaxf(m[h], m1), c0 = exp2_fast(m[h] - mn), c1 = exp2_fast(m1 - mn);
      m[h] = mn;
      l[h] = l[h] * c0 + other[(2 + h) * kAttnThreads + tid] * c1;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 2 * h; i < 2 * h + 2; ++i) o[n][i] = o[n][i] * c0 + other[(4 + 4 * n + i) * kAttnThreads + tid] * c1;
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
    l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
    const int r = row_a + 8 * h;
    if (r < len) {
      const float inv = 1.0f / l[h];
      __half* dst = p.out + (start + r) * p.ldo + head * HD + 2 * t;
#pragma unroll
      for (int n = 0; n < NT; ++n) *reinterpret_cast<uint32_t*>(dst + n * 8) = pack_half2_rn(o[n][2 * h] * inv, o[n][2 * h + 1] * inv);
      if (t == 0) p.lse[head * p.rows + start + r] = m[h] + log2f(l[h]);
    }
  }
}

// delta[head][row] = sum over the head's columns of dout * out; one warp per (row, head)
template <int HD>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __grid_constant__ AttnParams p, int first, int rows) {
  pdl_wait();
  pdl_launch_dependents();
  constexpr int L = HD / 8;                  // lanes per (row, head)
  const int64_t idx = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) / L;
  const int c = threadIdx.x % L;
  const bool live = idx < static_cast<int64_t>(rows) * p.heads;
  const uint32_t i = live ? static_cast<uint32_t>(idx) : 0;      // rows x heads fits: each holds 128 bytes of dout at least
  const int row = first + static_cast<int>(i / static_cast<uint32_t>(p.heads)), head = static_cast<int>(i % static_cast<uint32_t>(p.heads));
  float a[8], b[8], s = 0.f;
  unpack8(*reinterpret_cast<const uint4*>(p.dout + row * p.lddo + head * HD + c * 8), a);
  unpack8(*reinterpret_cast<const uint4*>(p.o + row * p.ldo + head * HD + c * 8), b);
#pragma unroll
  for (int k = 0; k < 8; ++k) s = fmaf(a[k], b[k], s);
#pragma unroll
  for (int x = L / 2; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
  if (live && c == 0) p.delta[head * p.rows + row] = s;
}

// Rotate a gradient back (transpose of the rotation) and store it: acc holds rows (g, g + 8) x HD columns of one warp.
template <int HD>
__device__ __forceinline__ void store_unrotated(const float (&acc)[HD / 8][4], const AttnParams& p, __half* base, int row_a, int len, int t, float mul) {
  constexpr int NT = HD / 8;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = row_a + 8 * h;
    if (r >= len) continue;
    const float4* tp = reinterpret_cast<const float4*>(p.trig + static_cast<int64_t>(r) * (HD / 2) + 2 * t);
    __half* dst = base + r * p.ldd + 2 * t;
#pragma unroll
    for (int n = 0; n < NT / 2; ++n) {
      const float4 cs = __ldg(tp + n * 4);   // (cos, sin) of columns 8 n + 2 t, + 1
      const float x0 = acc[n][2 * h] * mul, x1 = acc[n][2 * h + 1] * mul;
      const float y0 = acc[n + NT / 2][2 * h] * mul, y1 = acc[n + NT / 2][2 * h + 1] * mul;
      *reinterpret_cast<uint32_t*>(dst + n * 8) = pack_half2_rn(x0 * cs.x + y0 * cs.y, x1 * cs.z + y1 * cs.w);
      *reinterpret_cast<uint32_t*>(dst + HD / 2 + n * 8) = pack_half2_rn(y0 * cs.x - x0 * cs.y, y1 * cs.z - x1 * cs.w);
    }
  }
}

__device__ __forceinline__ float4 attn_peer128(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// 4 bytes global -> shared, zeros when `valid` is false
__device__ __forceinline__ void attn_cp4(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

template <int HD, int HALVES>
__global__ void __launch_bounds__(HALVES * kAttnThreads)
attn_dq_kernel(const __grid_constant__ AttnParams p, const __grid_constant__ SeqTable seqs) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(128) uint8_t a_smem[];
  constexpr int TILE = kAttnRows * HD * 2, KS = HD / 16, NT = HD / 8;
  const int half = HALVES == 1 ? 0 : threadIdx.x / kAttnThreads, warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t sQ = smem_u32(a_smem), sO = sQ + TILE, sK = sO + TILE + half * 4 * TILE, sV = sK + 2 * TILE;
  int start, len, q0;
  find_tile(seqs, seqs.tile[seqs.n] - 1 - blockIdx.x, start, len, q0);
  const int head = blockIdx.y, kvh = head / p.group;
  const __half* kp = p.k + start * p.ldr + kvh * HD;
  const __half* vp = p.v + start * p.ldv + kvh * HD;
  const int n_blocks = q0 / kAttnRows + 1;
  load_tile<HD, kAttnRows, HALVES * kAttnThreads>(sQ, p.q + start * p.ldr + head * HD, p.ldr, q0, len);
  load_tile<HD, kAttnRows, HALVES * kAttnThreads>(sO, p.dout + start * p.lddo + head * HD, p.lddo, q0, len);
  auto load = [&](int b, int slot) {
    if (b < n_blocks) {
      load_tile<HD, kAttnRows>(sK + slot * TILE, kp, p.ldr, b * kAttnRows, len);
      load_tile<HD, kAttnRows>(sV + slot * TILE, vp, p.ldv, b * kAttnRows, len);
    }
    attn_commit();
  };
  auto sync = [&] {
    if (HALVES == 1) __syncthreads();
    else named_barrier(half + 1, kAttnThreads);       // the 128 threads of this half
  };
  load(half, 0);
  load(half + HALVES, 1);
  const int row_a = q0 + warp * 16 + g;
  float lse[2], delta[2], dq[NT][4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const bool live = row_a + 8 * h < len;
    lse[h] = live ? p.lse[head * p.rows + start + row_a + 8 * h] : 0.f;
    delta[h] = live ? p.delta[head * p.rows + start + row_a + 8 * h] : 0.f;
  }
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) dq[n][i] = 0.f;
  attn_wait<1>();
  __syncthreads();
  for (int b = half, slot = 0; b < n_blocks; b += HALVES, slot ^= 1) {
    const uint32_t kb = sK + slot * TILE, vb = sV + slot * TILE;
#pragma unroll
    for (int hb = 0; hb < 2; ++hb) {         // 32 keys at a time
      float s[4][4], dp[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) { s[n][i] = 0.f; dp[n][i] = 0.f; }
#pragma unroll
      for (int kk = 0; kk < KS; ++kk) {
        uint32_t a[4], d[4];
        frag_a<HD>(sQ, warp * 16, kk, lane, a);
        frag_a<HD>(sO, warp * 16, kk, lane, d);
#pragma unroll
        for (int n2 = 0; n2 < 2; ++n2) {
          uint32_t bf[4];
          frag_b<HD>(kb, hb * 32 + n2 * 16, kk, lane, bf);
          mma16816(s[2 * n2], a[0], a[1], a[2], a[3], bf[0], bf[1]);
          mma16816(s[2 * n2 + 1], a[0], a[1], a[2], a[3], bf[2], bf[3]);
          frag_b<HD>(vb, hb * 32 + n2 * 16, kk, lane, bf);
          mma16816(dp[2 * n2], d[0], d[1], d[2], d[3], bf[0], bf[1]);
          mma16816(dp[2 * n2 + 1], d[0], d[1], d[2], d[3], bf[2], bf[3]);
        }
      }
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int key = b * kAttnRows + hb * 32 + n * 8 + 2 * t + (i & 1);
          const float pr = key > row_a + (i >> 1) * 8 ? 0.f : exp2_fast(fmaf(s[n][i], p.scale_log2, -lse[i >> 1]));
          s[n][i] = pr * (dp[n][i] - delta[i >> 1]);
        }
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        const uint32_t a0 = pack_half2_rn(s[2 * kk][0], s[2 * kk][1]), a1 = pack_half2_rn(s[2 * kk][2], s[2 * kk][3]);
        const uint32_t a2 = pack_half2_rn(s[2 * kk + 1][0], s[2 * kk + 1][1]), a3 = pack_half2_rn(s[2 * kk + 1][2], s[2 * kk + 1][3]);
#pragma unroll
        for (int n2 = 0; n2 < NT / 2; ++n2) {
          uint32_t bf[4];
          frag_bt<HD>(kb, hb * 32 + kk * 16, n2 * 16, lane, bf);
          mma16816(dq[2 * n2], a0, a1, a2, a3, bf[0], bf[1]);
          mma16816(dq[2 * n2 + 1], a0, a1, a2, a3, bf[2], bf[3]);
        }
      }
    }
    sync();
    load(b + 2 * HALVES, slot);
    attn_wait<1>();
    sync();
  }
  if constexpr (HALVES == 2) {
    attn_wait<0>();
    float* const other = reinterpret_cast<float*>(a_smem + 2 * TILE + 4 * TILE);   // the second half's sums, [value][thread]
    __syncthreads();
    const int tid = threadIdx.x % kAttnThreads;
    if (half) {
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) other[(4 * n + i) * kAttnThreads + tid] = dq[n][i];
    }
    __syncthreads();
    if (half) return;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) dq[n][i] += other[(4 * n + i) * kAttnThreads + tid];
  }
  store_unrotated<HD>(dq, p, p.dq + start * p.ldd + head * HD, row_a, len, t, p.scale);
}

template <int HD>
__global__ void __launch_bounds__(kAttnThreads)
attn_dkv_kernel(const __grid_constant__ AttnParams p, const __grid_constant__ SeqTable seqs) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(128) uint8_t a_smem[];
  constexpr int QR = 32;                     // query rows per step
  constexpr int TILE = kAttnRows * HD * 2, QT = QR * HD * 2, KS = HD / 16, NT = HD / 8;
  const uint32_t sK = smem_u32(a_smem), sV = sK + TILE, sQ = sV + TILE, sO = sQ + 2 * QT;
  float* sL = reinterpret_cast<float*>(a_smem + 2 * TILE + 4 * QT);      // [2][QR] lse, [2][QR] delta
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  int start, len, k0;
  // cluster of C CTAs: rank r takes the group's heads r, r + C, ...
  const int C = static_cast<int>(gridDim.x) / seqs.tile[seqs.n], rank = static_cast<int>(blockIdx.x) % C;
  find_tile(seqs, blockIdx.x / C, start, len, k0);                       // earlier key tiles have more query rows: first
  const int kvh = blockIdx.y;
  load_tile<HD, kAttnRows>(sK, p.k + start * p.ldr + kvh * HD, p.ldr, k0, len);
  load_tile<HD, kAttnRows>(sV, p.v + start * p.ldv + kvh * HD, p.ldv, k0, len);
  const int per_head = (len - k0 + QR - 1) / QR, steps = per_head * ((p.group - rank + C - 1) / C);
  auto issue = [&](int it) {
    const int head = kvh * p.group + rank + it / per_head * C, q0 = k0 + (it % per_head) * QR, slot = it & 1;
    load_tile<HD, QR>(sQ + slot * QT, p.q + start * p.ldr + head * HD, p.ldr, q0, len);
    load_tile<HD, QR>(sO + slot * QT, p.dout + start * p.lddo + head * HD, p.lddo, q0, len);
    if (threadIdx.x < QR) {
      const int r = q0 + threadIdx.x;
      const int64_t at = head * p.rows + start + (r < len ? r : 0);
      attn_cp4(smem_u32(sL + slot * QR + threadIdx.x), p.lse + at, r < len);
      attn_cp4(smem_u32(sL + 2 * QR + slot * QR + threadIdx.x), p.delta + at, r < len);
    }
  };
  issue(0);
  attn_commit();
  float dk[NT][4], dv[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) { dk[n][i] = 0.f; dv[n][i] = 0.f; }
  const int key_a = k0 + warp * 16 + g;
  for (int it = 0; it < steps; ++it) {
    if (it + 1 < steps) issue(it + 1);
    attn_commit();
    attn_wait<1>();
    __syncthreads();
    const int slot = it & 1, q0 = k0 + (it % per_head) * QR;
    const uint32_t qb = sQ + slot * QT, ob = sO + slot * QT;
    // transposed scores: 16 keys of this warp x 32 queries
    float s[4][4], dp[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) { s[n][i] = 0.f; dp[n][i] = 0.f; }
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      uint32_t a[4], d[4];
      frag_a<HD>(sK, warp * 16, kk, lane, a);
      frag_a<HD>(sV, warp * 16, kk, lane, d);
#pragma unroll
      for (int n2 = 0; n2 < 2; ++n2) {
        uint32_t bf[4];
        frag_b<HD>(qb, n2 * 16, kk, lane, bf);
        mma16816(s[2 * n2], a[0], a[1], a[2], a[3], bf[0], bf[1]);
        mma16816(s[2 * n2 + 1], a[0], a[1], a[2], a[3], bf[2], bf[3]);
        frag_b<HD>(ob, n2 * 16, kk, lane, bf);
        mma16816(dp[2 * n2], d[0], d[1], d[2], d[3], bf[0], bf[1]);
        mma16816(dp[2 * n2 + 1], d[0], d[1], d[2], d[3], bf[2], bf[3]);
      }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int qi = n * 8 + 2 * t + (i & 1), query = q0 + qi, key = key_a + (i >> 1) * 8;
        const float pr = (key > query || query >= len) ? 0.f : exp2_fast(fmaf(s[n][i], p.scale_log2, -sL[slot * QR + qi]));
        s[n][i] = pr;
        dp[n][i] = pr * (dp[n][i] - sL[2 * QR + slot * QR + qi]);
      }
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      const uint32_t a0 = pack_half2_rn(s[2 * kk][0], s[2 * kk][1]), a1 = pack_half2_rn(s[2 * kk][2], s[2 * kk][3]);
      const uint32_t a2 = pack_half2_rn(s[2 * kk + 1][0], s[2 * kk + 1][1]), a3 = pack_half2_rn(s[2 * kk + 1][2], s[2 * kk + 1][3]);
      const uint32_t e0 = pack_half2_rn(dp[2 * kk][0], dp[2 * kk][1]), e1 = pack_half2_rn(dp[2 * kk][2], dp[2 * kk][3]);
      const uint32_t e2 = pack_half2_rn(dp[2 * kk + 1][0], dp[2 * kk + 1][1]), e3 = pack_half2_rn(dp[2 * kk + 1][2], dp[2 * kk + 1][3]);
#pragma unroll
      for (int n2 = 0; n2 < NT / 2; ++n2) {
        uint32_t bf[4];
        frag_bt<HD>(ob, kk * 16, n2 * 16, lane, bf);
        mma16816(dv[2 * n2], a0, a1, a2, a3, bf[0], bf[1]);
        mma16816(dv[2 * n2 + 1], a0, a1, a2, a3, bf[2], bf[3]);
        frag_bt<HD>(qb, kk * 16, n2 * 16, lane, bf);
        mma16816(dk[2 * n2], e0, e1, e2, e3, bf[0], bf[1]);
        mma16816(dk[2 * n2 + 1], e0, e1, e2, e3, bf[2], bf[3]);
      }
    }
    __syncthreads();
  }
  if (C > 1) {
    // every CTA leaves its sums where the tiles were ([dk, dv][n][thread], 16 bytes each); rank r adds up the column groups
    // n = r, r + C, ... below the half and their partners of the rotation, over the ranks in order
    const uint32_t mine = smem_u32(a_smem) + threadIdx.x * 16;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      *reinterpret_cast<float4*>(a_smem + (n * kAttnThreads + threadIdx.x) * 16) = make_float4(dk[n][0], dk[n][1], dk[n][2], dk[n][3]);
      *reinterpret_cast<float4*>(a_smem + ((NT + n) * kAttnThreads + threadIdx.x) * 16) = make_float4(dv[n][0], dv[n][1], dv[n][2], dv[n][3]);
    }
    cluster_sync_all();
#pragma unroll 1
    for (int n = rank; n < NT / 2; n += C) {
      float sum[4][4];                       // dk of n and its partner, dv of both
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t at = mine + ((k >> 1) * NT + n + (k & 1) * (NT / 2)) * (kAttnThreads * 16);
        float4 v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = r < C ? attn_peer128(map_to_cta(at, r)) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 w = v[0];
#pragma unroll
        for (int r = 1; r < 8; ++r)
          if (r < C) { w.x += v[r].x; w.y += v[r].y; w.z += v[r].z; w.w += v[r].w; }
        sum[k][0] = w.x; sum[k][1] = w.y; sum[k][2] = w.z; sum[k][3] = w.w;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = key_a + 8 * h;
        if (r >= len) continue;
        const float4 cs = __ldg(reinterpret_cast<const float4*>(p.trig + static_cast<int64_t>(r) * (HD / 2) + n * 8 + 2 * t));
        const int64_t at = (start + r) * p.ldd + kvh * HD + n * 8 + 2 * t;
        const float x0 = sum[0][2 * h] * p.scale, x1 = sum[0][2 * h + 1] * p.scale, y0 = sum[1][2 * h] * p.scale, y1 = sum[1][2 * h + 1] * p.scale;
        *reinterpret_cast<uint32_t*>(p.dk + at) = pack_half2_rn(x0 * cs.x + y0 * cs.y, x1 * cs.z + y1 * cs.w);
        *reinterpret_cast<uint32_t*>(p.dk + at + HD / 2) = pack_half2_rn(y0 * cs.x - x0 * cs.y, y1 * cs.z - x1 * cs.w);
        *reinterpret_cast<uint32_t*>(p.dv + at) = pack_half2_rn(sum[2][2 * h], sum[2][2 * h + 1]);
        *reinterpret_cast<uint32_t*>(p.dv + at + HD / 2) = pack_half2_rn(sum[3][2 * h], sum[3][2 * h + 1]);
      }
    }
    __syncwarp();
    cluster_sync_all();                      // peers keep their sums until everybody has read them
    return;
  }
  store_unrotated<HD>(dk, p, p.dk + start * p.ldd + kvh * HD, key_a, len, t, p.scale);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = key_a + 8 * h;
    if (r >= len) continue;
    __half* dst = p.dv + (start + r) * p.ldd + kvh * HD + 2 * t;
#pragma unroll
    for (int n = 0; n < NT; ++n) *reinterpret_cast<uint32_t*>(dst + n * 8) = pack_half2_rn(dv[n][2 * h], dv[n][2 * h + 1]);
  }
}

// ---------------------------------------------------------------------------------------------
struct AttnShape {
  int heads, kv_heads, hd;
  int64_t rows;
};

static int attn_check(const AttnShape& s, const int32_t* lens, int n, const char* who) {
  if (!lens || n <= 0 || s.heads <= 0 || s.kv_heads <= 0 || s.heads % s.kv_heads || (s.hd != 64 && s.hd != 128)) {
    set_detail("%s: %d sequences, %d / %d heads of %d (head dimensions 64 and 128)", who, n, s.heads, s.kv_heads, s.hd);
    return NF4LL_ERR_SHAPE;
  }
  int64_t sum = 0;
  for (int i = 0; i < n; ++i) {
    if (lens[i] < 0) { set_detail("%s: sequence %d has %d rows", who, i, lens[i]); return NF4LL_ERR_SHAPE; }
    sum += lens[i];
  }
  if (sum != s.rows || s.rows > (int64_t(1) << 30)) {
    set_detail("%s: the sequences cover %lld of %lld rows", who, static_cast<long long>(sum), static_cast<long long>(s.rows));
    return NF4LL_ERR_SHAPE;
  }
  return NF4LL_OK;
}

// the next (up to kAttnMaxSeqs) sequences from `at` on; empty ones are skipped
static int attn_table(SeqTable* t, const int32_t* lens, int n, int at, int64_t* row) {
  t->n = 0;
  t->tile[0] = 0;
  t->start[0] = static_cast<int>(*row);
  while (at < n && t->n < kAttnMaxSeqs) {
    const int len = lens[at++];
    if (len == 0) continue;
    *row += len;
    t->start[t->n + 1] = static_cast<int>(*row);
    t->tile[t->n + 1] = t->tile[t->n] + (len + kAttnRows - 1) / kAttnRows;
    ++t->n;
  }
  return at;
}

// Eight warps per CTA in two halves that take the key blocks in turn, each with a ring of its own, and add up at the end: half as long a
// chain of blocks per tile, for twice the shared memory. From four blocks in the longest sequence on (with fewer the second half idles:
// sequences of 130 and 129 rows, 28 heads of 128, forward 12.5 us with one half, 14.1 with two), and where the chain is what takes the time:
// the forward while one and a half CTAs of one half per SM hold all tiles (two with heads of 64; three of 128 from 16 blocks on), dQ while the
// SMs' share of all key blocks is less than the longest chain (and a quarter with heads of 64), or from 16 blocks on six CTAs per SM hold them
// (three of 64). us with one half / two, forward: 12 heads of 128, 333 rows 16.3 / 11.8, 1024
// rows 40.2 / 32.1, 10 sequences of 200 rows 22.5 / 26.2; 14 heads of 64, 600 rows 18.2 / 12.4, 10 of 200 rows 15.5 / 20.4; 28 heads of 128, 2048 rows
// 155 / 159; backward with 12 heads of 128, 1024 rows 118 / 104, 14 of 64 and 10 sequences of 200 rows 41.7 / 45.7. Over 398 batches the choice
// takes 0.2 % longer than the faster of the two, 7 % at worst; always two 4 % and 40 %.
static int attn_halves(const SeqTable& t, int heads, int hd, bool backward, int* halves) {
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int64_t longest = 0, blocks = 0;
  for (int i = 0; i < t.n; ++i) {
    const int64_t n = t.tile[i + 1] - t.tile[i];
    longest = n > longest ? n : longest;
    blocks += n * (n + 1) / 2;
  }
  const int64_t ctas = static_cast<int64_t>(t.tile[t.n]) * heads;
  const bool small = hd == 64, many = longest >= 16;
  const bool chain = backward ? 4 * blocks * heads < (small ? 5 : 4) * longest * sms || (many && ctas < (small ? 3 : 6) * sms)
                              : 2 * ctas < (small ? 4 : many ? 6 : 3) * sms;
  *halves = longest > 3 && chain ? 2 : 1;
  return NF4LL_OK;
}

template <int HD>
static int attn_forward_hd(AttnParams p, const __half* qkv, int64_t ldq, __half* roped, const int32_t* lens, int n, int kv_heads, cudaStream_t stream) {
  constexpr int tile = kAttnRows * HD * 2;
  NF4LL_CUDA(cudaFuncSetAttribute(attn_fwd_kernel<HD, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 5 * tile));
  NF4LL_CUDA(cudaFuncSetAttribute(attn_fwd_kernel<HD, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 9 * tile));
  int64_t row = 0;
  for (int at = 0; at < n;) {
    SeqTable t;
    at = attn_table(&t, lens, n, at, &row);
    if (t.n == 0) continue;
    const int64_t work = static_cast<int64_t>(t.start[t.n] - t.start[0]) * (p.heads + kv_heads) * (HD / 16);
    PdlLaunch lr(dim3(static_cast<unsigned>((work + 255) / 256 < 1184 ? (work + 255) / 256 : 1184)), dim3(256), 0, stream);
    NF4LL_CUDA(cudaLaunchKernelEx(&lr.cfg, rope_kernel, qkv, ldq, roped, p.ldr, p.trig, p.heads + kv_heads, HD, t));
    int halves = 1;
    if (int rc = attn_halves(t, p.heads, HD, false, &halves)) return rc;
    PdlLaunch lf(dim3(static_cast<unsigned>(t.tile[t.n]), static_cast<unsigned>(p.heads)), dim3(halves * kAttnThreads), (1 + 4 * halves) * tile, stream);
    NF4LL_CUDA(cudaLaunchKernelEx(&lf.cfg, halves == 2 ? attn_fwd_kernel<HD, 2> : attn_fwd_kernel<HD, 1>, p, t));
  }
  return NF4LL_OK;
}

template <int HD>
static int attn_backward_hd(AttnParams p, const int32_t* lens, int n, int kv_heads, cudaStream_t stream) {
  constexpr int tile = kAttnRows * HD * 2, smem_kv = 4 * kAttnRows * HD * 2 + 4 * 32 * 4;
  NF4LL_CUDA(cudaFuncSetAttribute(attn_dq_kernel<HD, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * tile));
  NF4LL_CUDA(cudaFuncSetAttribute(attn_dq_kernel<HD, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 10 * tile));
  NF4LL_CUDA(cudaFuncSetAttribute(attn_dkv_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_kv));
  int64_t row = 0;
  for (int at = 0; at < n;) {
    SeqTable t;
    at = attn_table(&t, lens, n, at, &row);
    if (t.n == 0) continue;
    const int rows = t.start[t.n] - t.start[0];
    PdlLaunch ld(dim3(static_cast<unsigned>((static_cast<int64_t>(rows) * p.heads * (HD / 8) + 255) / 256)), dim3(256), 0, stream);
    NF4LL_CUDA(cudaLaunchKernelEx(&ld.cfg, attn_delta_kernel<HD>, p, t.start[0], rows));
    const unsigned parts = static_cast<unsigned>(p.group < 8 ? p.group : 8);
    PdlLaunch lk(dim3(static_cast<unsigned>(t.tile[t.n]) * parts, static_cast<unsigned>(kv_heads)), dim3(kAttnThreads), smem_kv, stream, parts, 1);
    NF4LL_CUDA(cudaLaunchKernelEx(&lk.cfg, attn_dkv_kernel<HD>, p, t));
    int halves = 1;
    if (int rc = attn_halves(t, p.heads, HD, true, &halves)) return rc;
    PdlLaunch lq(dim3(static_cast<unsigned>(t.tile[t.n]), static_cast<unsigned>(p.heads)), dim3(halves * kAttnThreads), (2 + 4 * halves) * tile, stream);
    NF4LL_CUDA(cudaLaunchKernelEx(&lq.cfg, halves == 2 ? attn_dq_kernel<HD, 2> : attn_dq_kernel<HD, 1>, p, t));
  }
  return NF4LL_OK;
}

}  // namespace nf4ll

extern "C" int nf4ll_attention_forward(const void* qkv, int64_t ldq, const int32_t* seq_lens, int32_t n_seqs, int64_t rows, int32_t heads,
                                       int32_t kv_heads, int32_t head_dim, const void* trig, void* roped, int64_t ldr, void* out, int64_t ldo,
                                       float* lse, void* stream) {
  using namespace nf4ll;
  const char* who = "nf4ll_attention_forward";
  if (rows == 0) return NF4LL_OK;
  if (!qkv || !trig || !roped || !out || !lse) { set_detail("%s: null pointer", who); return NF4LL_ERR_NULL; }
  if (int rc = attn_check({heads, kv_heads, head_dim, rows}, seq_lens, n_seqs, who)) return rc;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(trig) | reinterpret_cast<uintptr_t>(roped) | reinterpret_cast<uintptr_t>(out)) & 15 ||
      (ldq | ldr | ldo) % 8) {
    set_detail("%s: pointers 16-byte aligned, leading dimensions multiples of 8", who);
    return NF4LL_ERR_ALIGN;
  }
  if (int rc = require_sm100()) return rc;
  AttnParams p{};
  p.q = static_cast<const __half*>(roped);
  p.k = p.q + static_cast<int64_t>(heads) * head_dim;
  p.ldr = ldr;
  p.v = static_cast<const __half*>(qkv) + static_cast<int64_t>(heads + kv_heads) * head_dim;
  p.ldv = ldq;
  p.out = static_cast<__half*>(out); p.ldo = ldo;
  p.lse = lse;
  p.trig = static_cast<const float2*>(trig);
  p.heads = heads; p.group = heads / kv_heads; p.rows = rows;
  p.scale = 1.0f / sqrtf(static_cast<float>(head_dim));
  p.scale_log2 = p.scale * 1.4426950408889634f;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* src = static_cast<const __half*>(qkv);
  return head_dim == 128 ? attn_forward_hd<128>(p, src, ldq, static_cast<__half*>(roped), seq_lens, n_seqs, kv_heads, st)
                         : attn_forward_hd<64>(p, src, ldq, static_cast<__half*>(roped), seq_lens, n_seqs, kv_heads, st);
}

extern "C" int nf4ll_attention_backward(const void* qkv, int64_t ldq, const int32_t* seq_lens, int32_t n_seqs, int64_t rows, int32_t heads,
                                        int32_t kv_heads, int32_t head_dim, const void* trig, const void* roped, int64_t ldr, const void* out,
                                        int64_t ldo, const float* lse, const void* dout, int64_t lddo, float* delta, void* dqkv, int64_t ldd,
                                        void* stream) {
  using namespace nf4ll;
  const char* who = "nf4ll_attention_backward";
  if (rows == 0) return NF4LL_OK;
  if (!qkv || !trig || !roped || !out || !lse || !dout || !delta || !dqkv) { set_detail("%s: null pointer", who); return NF4LL_ERR_NULL; }
  if (int rc = attn_check({heads, kv_heads, head_dim, rows}, seq_lens, n_seqs, who)) return rc;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(trig) | reinterpret_cast<uintptr_t>(roped) | reinterpret_cast<uintptr_t>(out) |
       reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dqkv)) & 15 || (ldq | ldr | ldo | lddo | ldd) % 8) {
    set_detail("%s: pointers 16-byte aligned, leading dimensions multiples of 8", who);
    return NF4LL_ERR_ALIGN;
  }
  if (int rc = require_sm100()) return rc;
  AttnParams p{};
  p.q = static_cast<const __half*>(roped);
  p.k = p.q + static_cast<int64_t>(heads) * head_dim;
  p.ldr = ldr;
  p.v = static_cast<const __half*>(qkv) + static_cast<int64_t>(heads + kv_heads) * head_dim;
  p.ldv = ldq;
  p.o = static_cast<const __half*>(out); p.ldo = ldo;
  p.dout = static_cast<const __half*>(dout); p.lddo = lddo;
  p.dq = static_cast<__half*>(dqkv);
  p.dk = p.dq + static_cast<int64_t>(heads) * head_dim;
  p.dv = p.dk + static_cast<int64_t>(kv_heads) * head_dim;
  p.ldd = ldd;
  p.lse = const_cast<float*>(lse);
  p.delta = delta;
  p.trig = static_cast<const float2*>(trig);
  p.heads = heads; p.group = heads / kv_heads; p.rows = rows;
  p.scale = 1.0f / sqrtf(static_cast<float>(head_dim));
  p.scale_log2 = p.scale * 1.4426950408889634f;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return head_dim == 128 ? attn_backward_hd<128>(p, seq_lens, n_seqs, kv_heads, st) : attn_backward_hd<64>(p, seq_lens, n_seqs, kv_heads, st);
}
