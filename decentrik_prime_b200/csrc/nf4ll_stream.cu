// Small-batch forward (a handful of token rows): y[M,N] = x . W^T + bias + (s.T) . B^T, bound by the stream
// of NF4 bytes out of HBM, not by the tensor cores. Replaces, for decode-sized batches, the same
// reference call sites as the big-tile kernel (solution/fast_qwen.py:947, 1037, 1080-1112).
//
// A unit of work is 32 (or 16) weight rows; a team of W warps of one CTA owns it, each warp a part of the contraction, and
// their partial sums meet in shared memory in a fixed order (results do not depend on timing). Units are dealt out round
// the SMs. (A split of the contraction over CTAs, with partial sums and arrival counters in global memory, was measured
// first: the clearing of the counters, the fences and the second pass cost 6 us per call.) A warp fetches for itself:
// stages of four quantisation blocks by cp.async into a ring of its own (codes, absmax codes, second-level scales), three
// stages deep and across the ends of units. (Registers as the ring were measured first: a load's scoreboard is shared with
// the loads issued after it, so every block cost a trip to DRAM.) Every BYTE (two 4-bit codes) becomes two fp16 levels with
// ONE shared-memory load from a 256-entry table of half2 pairs. The table is replicated per lane (lane l reads word l of an
// entry: no bank conflicts whatever the codes are) at a stride of 256 B, which makes the byte permute that isolates a code
// byte the whole address computation; the other 128 B of an entry hold the stages' absmax words. The levels land directly in
// the A-operand layout of mma.sync.m16n8k16; the token rows are the B operand with the same column-to-slot assignment, loaded
// once per stage for all of the unit's 16-row tiles. The 64 weights of a block are accumulated on their own and folded into
// the running sum with that block's fp32 absmax, so the scale is applied once per block:
//     y[m,n] = sum_blocks absmax[n,b] * sum_{k in b} x[m,k] * fp16(NF4[code[n,k]])
// This differs from the big-tile kernel's bit-exact fp16 weights by the rounding of NF4[c] * absmax to
// fp16 (relative 2^-12), inside the 1e-3 tolerance of the path.
//
// 27648 x 5120 (73 MB) at 1 / 8 tokens: 26.7 / 29.4 us (2.7 / 2.5 TB/s), of which the fetch alone 19; 42 / 46 for the kernel that
// handed out units of 16 rows x a slice through a global counter. What is left over the fetch is the table lookups (4 us), the
// token loads (3 us at 8 tokens) and the MMAs (1 us) that do not hide behind it.
#include "nf4ll_stream.cuh"

namespace nf4ll {

__device__ __forceinline__ void mma16816_acc(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct StreamParams {
  const uint8_t* nib;
  const uint8_t* qabs;
  const float* scale2;
  const float* offset2;
  const float* code2;
  int64_t N, K;
  int64_t M;
  const __half* x;
  int64_t ldx;
  __half* y;
  int64_t ldy;
  const __half* bias;
  // several projections stacked along N (multiples of 32 rows), each with its own rank-16 branch
  int n_seg;
  int64_t seg_end[kMaxSegments];           // first row after the segment
  const float* seg_t[kMaxSegments];        // [M,16] fp32 = drop(x) . A^T, or null (no LoRA)
  const __half* seg_b[kMaxSegments];       // lora_B, offset so that it is indexed by the row of W
  float seg_scale[kMaxSegments];
  __half* y2;              // rows from `split` on go here (gate|up), null: one output
  int64_t ldy2, split;
  int early;               // the kernel before this one is a rank-16 projection of the same call
  int team;                // W: warps per unit, a divisor of kStreamWarps
};

constexpr int kStreamWarps = 12;
constexpr int kStreamRows = 32;              // most weight rows of a unit: one per lane, two 16-row operand tiles
constexpr int kStep = 4;                     // quantisation blocks per stage
constexpr int kStreamStages = 3;
constexpr int kEntryStride = 256;
constexpr int kTableBytes = 256 * kEntryStride;
constexpr int kAbsWords = 6;                 // per row and stage: two words of absmax codes, two pairs of scale and offset
constexpr int kPartBytes = 8 * kStreamRows * 4;              // one warp's sums of 8 tokens x 32 rows
constexpr int stream_smem(int rt) { return kTableBytes + 1024 + kStreamWarps * (kStreamRows * kStep * 4 + kPartBytes + kStreamStages * kStep * 16 * rt * 32); }
static_assert(stream_smem(2) <= 227 * 1024, "shared memory budget");
static_assert(kStreamWarps * kStreamStages * kAbsWords <= 256, "one unused half of a table entry per absmax word of 32 rows");

// offset into the table of the entry of byte I of `w` for this lane (lane_off = 4 * lane < 256): one byte permute
template <int I>
__device__ __forceinline__ uint32_t entry_offset(uint32_t w, uint32_t lane_off) {
  return prmt(w, lane_off, 0x5504u | (I << 4));
}

// the 8 weights of one 32-bit word of codes as four half2 registers (element order: high nibble first)
__device__ __forceinline__ void decode8(const uint8_t* table, uint32_t w, uint32_t lane_off, uint32_t (&h)[4]) {
  h[0] = *reinterpret_cast<const uint32_t*>(table + entry_offset<0>(w, lane_off));
  h[1] = *reinterpret_cast<const uint32_t*>(table + entry_offset<1>(w, lane_off));
  h[2] = *reinterpret_cast<const uint32_t*>(table + entry_offset<2>(w, lane_off));
  h[3] = *reinterpret_cast<const uint32_t*>(table + entry_offset<3>(w, lane_off));
}

__device__ __forceinline__ void mma16816_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void stream_cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void stream_cp4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// NT = number of 8-token tiles (M <= 8 NT), RT = number of 16-row tiles of a unit.
template <int NT, int RT>
__global__ void __launch_bounds__(kStreamWarps * 32, 1)
nf4_stream_kernel(const __grid_constant__ StreamParams p) {
  // Launched as a programmatic dependent of the kernel before it (the rank-16 projection T = x . A^T when there is a LoRA
  // branch): the table build and the first units' weight stream overlap that kernel; T is read and the first output
  // written after it.
  pdl_launch_dependents();
  extern __shared__ __align__(256) uint8_t st_smem[];
  constexpr int kRows = 16 * RT, kStepBytes = kStep * kRows * 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  float* s_code2 = reinterpret_cast<float*>(st_smem + kTableBytes);
  float* s_abs = reinterpret_cast<float*>(st_smem + kTableBytes + 1024) + warp * kStreamRows * kStep;      // this warp's [32 rows][4 blocks]
  float* s_part = reinterpret_cast<float*>(st_smem + kTableBytes + 1024 + kStreamWarps * kStreamRows * kStep * 4);      // [warp][8 tokens][32 rows]
  uint8_t* ring = reinterpret_cast<uint8_t*>(s_part) + kStreamWarps * kPartBytes + warp * kStreamStages * kStepBytes;
  uint8_t* words = st_smem + warp * kStreamStages * kAbsWords * kEntryStride + 128 + lane * 4;             // this lane's absmax words
  const int n_units = static_cast<int>(p.N / kRows);
  const int bpr = static_cast<int>(p.K / 64);       // quantisation blocks per weight row
  const bool aligned = (bpr & 3) == 0;
  const int team = warp / p.team, part = warp - team * p.team;
  const int first_unit = team * gridDim.x + blockIdx.x, unit_step = kStreamWarps / p.team * gridDim.x;
  const int steps = (bpr + kStep - 1) / kStep;      // this warp's part of every row, whole stages
  const int b_begin = steps * part / p.team * kStep;
  const int b_end = steps * (part + 1) / p.team * kStep < bpr ? steps * (part + 1) / p.team * kStep : bpr;
  // The fetching side's position: four blocks of unit `fu` from block `fb` on.
  int fu = b_begin < b_end ? first_unit : n_units, fb = b_begin;
  // lane l copies half (l & 1) of row l >> 1 (and of that row + 16) of every block, and the absmax words of row l mod kRows
  const uint8_t* fsrc = p.nib + (static_cast<int64_t>(fu) * kRows + (lane >> 1)) * (p.K / 2) + fb * 32 + (lane & 1) * 16;
  int64_t fq = (static_cast<int64_t>(fu) * kRows + lane % kRows) * bpr + fb;      // quantisation block of this lane's row
  const int64_t last_word = p.N * p.K / 64 - 4;     // of the absmax codes (their count is a multiple of 256)
  auto fetch = [&](int slot) {
    if (fu < n_units) {
      const int nb = b_end - fb < kStep ? b_end - fb : kStep;
      const uint32_t dst = smem_u32(ring + slot * kStepBytes) + lane * 16;
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        if (u < nb) {
          stream_cp16(dst + u * (kRows * 32), fsrc + u * 32);
          if (RT == 2) stream_cp16(dst + u * (kRows * 32) + 512, fsrc + 8 * p.K + u * 32);
        }
      }
      // absmax codes fq .. fq + nb - 1: one aligned word in one second-level group when rows are whole groups of four
      // blocks long, else two words and the groups of the first and of the last block
      const uint32_t wd = smem_u32(words) + slot * kAbsWords * kEntryStride;
      const int64_t w0 = fq & ~int64_t(3), g0 = fq >> 8;
      stream_cp4(wd, p.qabs + w0);
      stream_cp4(wd + 2 * kEntryStride, p.scale2 + g0);
      stream_cp4(wd + 3 * kEntryStride, p.offset2 + g0);
      if (!aligned) {
        const int64_t g1 = (fq + nb - 1) >> 8;
        stream_cp4(wd + kEntryStride, p.qabs + (w0 + 4 < last_word ? w0 + 4 : last_word));
        stream_cp4(wd + 4 * kEntryStride, p.scale2 + g1);
        stream_cp4(wd + 5 * kEntryStride, p.offset2 + g1);
      }
      fb += kStep;
      fsrc += kStep * 32;
      fq += kStep;
      if (fb >= b_end) {
        fu += unit_step;
        fb = b_begin;
        fsrc = p.nib + (static_cast<int64_t>(fu) * kRows + (lane >> 1)) * (p.K / 2) + fb * 32 + (lane & 1) * 16;
        fq = (static_cast<int64_t>(fu) * kRows + lane % kRows) * bpr + fb;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // Behind a rank-16 projection of the same call the weights (and x) may be read at once: that kernel itself went on only
  // after all earlier work on the stream had finished. Behind anything else only the table build overlaps it.
  bool waited = false;
  if (p.early) {
#pragma unroll
    for (int s = 0; s < kStreamStages; ++s) fetch(s);
  }
  {
    constexpr float lv[16] = {NF4LL_LEVELS};
    uint16_t* s_lv = reinterpret_cast<uint16_t*>(s_code2);      // until code2 takes its place
    if (threadIdx.x < 16) {
      float v = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) v = (static_cast<int>(threadIdx.x) == j) ? lv[j] : v;
      s_lv[threadIdx.x] = __half_as_ushort(__float2half_rn(v));
    }
    __syncthreads();
    // four lanes' copies of an entry per 16-byte store
    for (int idx = threadIdx.x; idx < 256 * 8; idx += kStreamWarps * 32) {
      const int v = idx >> 3;                       // byte value: even element in the high nibble
      const uint32_t e = s_lv[v >> 4] | (static_cast<uint32_t>(s_lv[v & 15]) << 16);
      *reinterpret_cast<uint4*>(st_smem + v * kEntryStride + (idx & 7) * 16) = make_uint4(e, e, e, e);
    }
    if (!p.early) {
      pdl_wait();
      waited = true;
#pragma unroll
      for (int s = 0; s < kStreamStages; ++s) fetch(s);
    }
    const float code2_mine = threadIdx.x < 256 ? p.code2[threadIdx.x] : 0.f;
    __syncthreads();
    if (threadIdx.x < 256) s_code2[threadIdx.x] = code2_mine;
    __syncthreads();
  }
  const uint32_t lane_off = lane * 4;
  int slot = 0;

  // The token rows of four blocks (with more than 16 tokens: of one), 32 bytes of each row and block, rows past M zeros. A
  // block's registers are refilled for the next stage as soon as it has been multiplied: x comes out of L2, and is the same
  // part of the contraction for every unit of a warp.
  constexpr int kX = NT <= 2 ? kStep : 1;
  uint4 x[kX][NT][2];
  auto load_x = [&](int b, uint4 (&dst)[NT][2]) {
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      dst[i][0] = dst[i][1] = make_uint4(0, 0, 0, 0);
      if (b < b_end && g + 8 * i < p.M) {
        const __half* src = p.x + (g + 8 * i) * p.ldx + t * 16 + static_cast<int64_t>(b) * 64;
        dst[i][0] = __ldg(reinterpret_cast<const uint4*>(src));
        dst[i][1] = __ldg(reinterpret_cast<const uint4*>(src + 8));
      }
    }
  };
  if (NT <= 2 && first_unit < n_units) {
#pragma unroll
    for (int u = 0; u < kX; ++u) load_x(b_begin + u, x[u]);
  }

  for (int unit = first_unit; unit < n_units; unit += unit_step) {
    const int64_t n0 = static_cast<int64_t>(unit) * kRows;
    float acc[RT][NT][4];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[r][i][j] = 0.f;
    int64_t q = (n0 + lane % kRows) * bpr + b_begin;        // quantisation block of this lane's row

    for (int b = b_begin; b < b_end; b += kStep, q += kStep) {
      const int nb = b_end - b < kStep ? b_end - b : kStep;
      const int b_next = b + kStep < b_end ? b + kStep : b_begin;
      asm volatile("cp.async.wait_group %0;" ::"n"(kStreamStages - 1) : "memory");
      __syncwarp();
      // absmax of this lane's row: codes -> fp32, shared by the warp
      {
        const uint8_t* wd = words + slot * kAbsWords * kEntryStride;
        uint32_t codes = *reinterpret_cast<const uint32_t*>(wd);
        const float s0 = *reinterpret_cast<const float*>(wd + 2 * kEntryStride), o0 = *reinterpret_cast<const float*>(wd + 3 * kEntryStride);
        float s1 = s0, o1 = o0;
        int turn = 4;                               // blocks of the first second-level group
        if (!aligned) {
          codes = __funnelshift_r(codes, *reinterpret_cast<const uint32_t*>(wd + kEntryStride), 8 * static_cast<int>(q & 3));
          s1 = *reinterpret_cast<const float*>(wd + 4 * kEntryStride);
          o1 = *reinterpret_cast<const float*>(wd + 5 * kEntryStride);
          const int left = 256 - static_cast<int>(q & 255);
          turn = left < 4 ? left : 4;
        }
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[j] = block_absmax(s_code2[(codes >> (8 * j)) & 255u], j < turn ? s0 : s1, j < turn ? o0 : o1);
        *reinterpret_cast<float4*>(s_abs + lane * 4) = make_float4(v[0], v[1], v[2], v[3]);
        __syncwarp();
      }
      float am[2 * RT][4];                          // rows g, g + 8, ...; blocks
#pragma unroll
      for (int r = 0; r < 2 * RT; ++r) {
        const float4 f = *reinterpret_cast<const float4*>(s_abs + (g + 8 * r) * 4);
        am[r][0] = f.x; am[r][1] = f.y; am[r][2] = f.z; am[r][3] = f.w;
      }
      const uint8_t* codes = ring + slot * kStepBytes + g * 32 + t * 8;
#pragma unroll
      for (int u = 0; u < kStep; ++u) {
        if (u < nb) {
          if (NT > 2) load_x(b + u, x[0]);
#pragma unroll
          for (int r = 0; r < RT; ++r) {
            const uint2 c0 = *reinterpret_cast<const uint2*>(codes + u * (kRows * 32) + r * 512);
            const uint2 c1 = *reinterpret_cast<const uint2*>(codes + u * (kRows * 32) + r * 512 + 256);
            uint32_t lo0[4], hi0[4], lo1[4], hi1[4];
            decode8(st_smem, c0.x, lane_off, lo0); decode8(st_smem, c0.y, lane_off, hi0);     // row g:   k 16t..16t+7, +8..+15
            decode8(st_smem, c1.x, lane_off, lo1); decode8(st_smem, c1.y, lane_off, hi1);     // row g+8
#pragma unroll
            for (int i = 0; i < NT; ++i) {
              const uint4 xa = x[u % kX][i][0], xb = x[u % kX][i][1];
              float blk[4];
              mma16816_first(blk, lo0[0], lo1[0], lo0[1], lo1[1], xa.x, xa.y);
              mma16816_acc(blk, lo0[2], lo1[2], lo0[3], lo1[3], xa.z, xa.w);
              mma16816_acc(blk, hi0[0], hi1[0], hi0[1], hi1[1], xb.x, xb.y);
              mma16816_acc(blk, hi0[2], hi1[2], hi0[3], hi1[3], xb.z, xb.w);
              acc[r][i][0] = fmaf(blk[0], am[2 * r][u], acc[r][i][0]);
              acc[r][i][1] = fmaf(blk[1], am[2 * r][u], acc[r][i][1]);
              acc[r][i][2] = fmaf(blk[2], am[2 * r + 1][u], acc[r][i][2]);
              acc[r][i][3] = fmaf(blk[3], am[2 * r + 1][u], acc[r][i][3]);
            }
          }
        }
        if (NT <= 2) load_x(b_next + u, x[u % kX]);
      }
      __syncwarp();                                 // everybody has read the stage and the absmax values
      fetch(slot);
      slot = slot + 1 == kStreamStages ? 0 : slot + 1;
    }

    // accumulator layout: acc[r][i][0..1] = (weight row 16 r + g, tokens 8i + 2t, +1); acc[r][i][2..3] = that row + 8
    if (!waited) {
      pdl_wait();                 // T comes from the kernel this one was launched behind
      waited = true;
    }
    int sg = 0;
    while (sg + 1 < p.n_seg && n0 >= p.seg_end[sg]) ++sg;
    const float* t32 = p.seg_t[sg];
    const int64_t row = n0 + lane % kRows;          // from here on a lane is a weight row
    __half* y = p.y + row;
    int64_t ldy = p.ldy;
    if (p.y2 && n0 >= p.split) { y = p.y2 + (row - p.split); ldy = p.ldy2; }
    const float bias = p.bias ? __half2float(p.bias[row]) : 0.f;
    float br[16];
    if (t32) {
      const uint4* bp = reinterpret_cast<const uint4*>(p.seg_b[sg] + row * 16);
      const float lora_scale = p.seg_scale[sg];
      float tmp[8];
      unpack8(__ldg(bp), tmp);
#pragma unroll
      for (int j = 0; j < 8; ++j) br[j] = tmp[j] * lora_scale;
      unpack8(__ldg(bp + 1), tmp);
#pragma unroll
      for (int j = 0; j < 8; ++j) br[8 + j] = tmp[j] * lora_scale;
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      if (8 * i < p.M) {
        // [token][row], rows XORed with the token so that neither side has bank conflicts
        float* mine = s_part + warp * (8 * kStreamRows);
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
          for (int j = 0; j < 4; ++j) mine[(2 * t + (j & 1)) * kStreamRows + ((16 * r + 8 * (j >> 1) + g) ^ (8 * t))] = acc[r][i][j];
        named_barrier(1 + team, p.team * 32);
        // the team's warps (of 16 rows: half warps) share the tokens out
        for (int k = RT == 2 ? part : 2 * part + (lane >> 4); k < 8; k += (3 - RT) * p.team) {
          const int64_t tok = 8 * i + k;
          if (tok >= p.M) break;
          float v = 0.f;
          for (int w = 0; w < p.team; ++w) v += s_part[(team * p.team + w) * (8 * kStreamRows) + k * kStreamRows + ((lane % kRows) ^ (8 * (k >> 1)))];
          v += bias;
          if (t32) {
            const float4* tr = reinterpret_cast<const float4*>(t32 + tok * 16);
            float l = 0.f;
#pragma unroll
            for (int j4 = 0; j4 < 4; ++j4) {
              const float4 tv = __ldcg(tr + j4);
              l = fmaf(tv.x, br[4 * j4], l); l = fmaf(tv.y, br[4 * j4 + 1], l);
              l = fmaf(tv.z, br[4 * j4 + 2], l); l = fmaf(tv.w, br[4 * j4 + 3], l);
            }
            v += l;
          }
          y[tok * ldy] = __float2half_rn(v);
        }
        __syncwarp();
        named_barrier(1 + team, p.team * 32);       // the sums have been read
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Rows and warps per unit: the pair with the least work in blocks over the rounds of units that the busiest warp takes, a unit
// costing its blocks and about three more (filling the pipeline, the exchange). Units of 16 rows cost 0.6 of one of 32
// (token rows and absmax words are fetched for half the weights); they pay where 32 leave SMs idle in the last round
// (5120 x 5120 at 1 token: 9.3 us in units of 16, 10.3 in units of 32; 5120 x 27648: 38.6 and 45.4).
static int64_t stream_plan(int64_t N, int64_t K, int sms, int force, int* row_tiles, int* team) {
  const int64_t steps = (K / 64 + kStep - 1) / kStep;
  int64_t best = 0;
  *row_tiles = 0;
  for (int rt = 2; rt >= 1; --rt) {
    const int64_t units = N / (16 * rt);
    for (int w : {1, 2, 3, 4, 6, 12}) {
      static_assert(kStreamWarps == 12, "its divisors");
      const int64_t at_once = static_cast<int64_t>(sms) * (kStreamWarps / w);
      const int64_t cost = (units + at_once - 1) / at_once * ((steps + w - 1) / w * kStep + 3) * (rt == 2 ? 10 : 6);
      if (force > 0 ? (rt == 1 + (force & 1) && w <= force) : (*row_tiles == 0 || cost < best || (cost == best && rt == *row_tiles))) {
        best = cost;
        *row_tiles = rt;
        *team = w;
      }
    }
  }
  return best;
}

double stream_time_us(int64_t N, int64_t K, int64_t M, int sms) {
  int rt = 0, team = 0;
  const int64_t cost = stream_plan(N, K, sms, 0, &rt, &team);      // in tenths of a block of 32 rows
  return 0.06 * cost * (M > 8 ? 1.3 : 1.0) + 0.0125 * M * cost / (rt == 2 ? 10 : 6);
}

template <int RT>
static auto stream_kernel(int64_t M) {
  return M <= 8 ? nf4_stream_kernel<1, RT> : (M <= 16 ? nf4_stream_kernel<2, RT> : (M <= 32 ? nf4_stream_kernel<4, RT> : nf4_stream_kernel<8, RT>));
}

int stream_forward_launch(const StreamCall& c, bool early, int force_team, cudaStream_t stream) {
  int dev = 0, sms = 148;
  NF4LL_CUDA(cudaGetDevice(&dev));
  NF4LL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const nf4ll_mat* W = c.W;
  StreamParams p{};
  p.nib = W->nib; p.qabs = W->qabs; p.scale2 = W->scale2; p.offset2 = W->offset2; p.code2 = W->code2;
  p.N = W->N; p.K = W->K; p.M = c.M;
  p.x = static_cast<const __half*>(c.x); p.ldx = c.ldx;
  p.y = static_cast<__half*>(c.y); p.ldy = c.ldy;
  p.y2 = static_cast<__half*>(c.y2); p.ldy2 = c.ldy2; p.split = c.split;
  p.bias = static_cast<const __half*>(c.bias);
  p.n_seg = c.n_seg;
  for (int i = 0; i < c.n_seg; ++i) {
    p.seg_end[i] = c.seg_end[i];
    p.seg_t[i] = c.seg_t[i]; p.seg_b[i] = c.seg_b[i]; p.seg_scale[i] = c.seg_scale[i];
  }
  p.early = early ? 1 : 0;
  int rt = 0;
  stream_plan(W->N, W->K, sms, force_team, &rt, &p.team);
  const auto kernel = rt == 2 ? stream_kernel<2>(c.M) : stream_kernel<1>(c.M);
  NF4LL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, stream_smem(rt)));
  const int64_t units = W->N / (16 * rt);
  PdlLaunch lc(dim3(static_cast<unsigned>(units < sms ? units : sms)), dim3(kStreamWarps * 32), stream_smem(rt), stream);
  NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, kernel, p));
  return NF4LL_OK;
}

}  // namespace nf4ll
