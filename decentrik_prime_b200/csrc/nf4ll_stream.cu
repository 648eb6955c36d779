// Small-batch forward (a handful of token rows): y[M,N] = x . W^T + bias + (s.T) . B^T, bound by the stream
// of NF4 bytes out of HBM, not by the tensor cores. Replaces, for decode-sized batches, the same
// reference call sites as the big-tile kernel (solution/fast_qwen.py:947, 1037, 1080-1112), gate|up with its gated product
// (solution/k_mlp.py:21-29) in the same launch.
//
// A tile is 16 weight rows of all K (of a CTA's part of K, where a row is too long for one: then a cluster shares the contraction).
// Two warps copy tiles into a ring of stages with bulk copies: rows of codes, the tile's absmax codes in one piece, its second-level
// scales. A team of warps shares a tile out along K: each keeps the token rows of its up to seven quantisation blocks in registers for the
// whole kernel and goes through tile after tile. Their sums meet in shared memory in a fixed order (and then the cluster's, through
// distributed shared memory: results do not depend on timing), where two more warps add them up, add the rank-16 term and the bias, and
// store.
//
// Every BYTE of codes (two 4-bit codes) becomes two fp16 levels with ONE shared-memory load from a 256-entry table of half2 pairs,
// replicated per lane (lane l reads word l of an entry: no bank conflicts whatever the codes are) at a stride of 256 B, which makes the byte
// permute that isolates a code byte the whole address computation; the other 128 B of an entry hold partial sums and scaled rank-16
// products. The levels land directly in the A-operand layout of mma.sync.m16n8k16; the token rows are the B operand with the same column-to-slot assignment. The
// 64 weights of a block are accumulated on their own and folded into the running sum with that block's fp32 absmax, so the scale is
// applied once per block:
//     y[m,n] = sum_blocks absmax[n,b] * sum_{k in b} x[m,k] * fp16(NF4[code[n,k]])
// This differs from the big-tile kernel's bit-exact fp16 weights by the rounding of NF4[c] * absmax to
// fp16 (relative 2^-12), inside the 1e-3 tolerance of the path.
//
// Measured, calls in a row without LoRA, the kernel before (every warp fetched 32 rows x 4 blocks for itself with cp.async and read
// the token rows anew for each) / this one, us at 1 and 8 rows: 3584 x 3584 6.6, 7.4 / 5.1, 5.4; 5120 x 5120 9.8, 11.1 / 7.7, 8.1; 27648 x 5120
// (73 MB) 26.7, 29.3 / 20.4, 21.0; 5120 x 27648 36.7, 42.2 / 23.5, 23.9; 3584 x 18944 18.6, 20.7 / 15, 15.2; gate|up 37888 x 3584 with its product
// 29.2, 32.7 / 21.1, 21.7. Of 27648 x 5120 the fetch alone takes 14 and the decode alone 19.7: what bounds it is shared memory (per 1024 weights
// 16 cycles of table reads, 4 of codes coming and 4 going, 5 of absmax values and sums: 1.1 of 1.45 us per tile) and the latencies that 12 warps
// of 128 registers leave (16 warps of 96: 22.2; 8 of 168: 21.2). Also tried: a third of the lookups by byte permutes instead (23.1), absmax
// values by warps of their own (35), absmax codes copied row by row (24.2: small copies cost 3 us), one tensor copy of a tile in swizzled
// 128-byte pieces (21.3; ahead only for rows of 1536 weights and less: 17920 x 1536 6.9, here 7.9).
//
// Every wait is bounded and reports through the status word (tested by withholding copies and the cluster's sums).
#include "nf4ll_pair.cuh"
#include "nf4ll_stream.cuh"

namespace nf4ll {

__device__ __forceinline__ void mma16816_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// contiguous bytes of global memory into shared memory; both addresses and the size are multiples of 16
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

__device__ __forceinline__ void stream_cp4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

constexpr int kStreamRows = 16;              // weight rows of a tile
constexpr int kStreamProducers = 2;          // warps that copy: their lanes' bulk copies are issued one after another, some 80 clocks each
constexpr int kStreamEpilogues = 2;          // warps that finish tiles
constexpr int kStreamMaxStages = 8;
constexpr int kStreamMaxCluster = 16;
constexpr int kStreamMaxSlots = 64;          // units of a cluster that one of its CTAs finishes
constexpr int kStreamMaxGroups = 64;         // second-level groups that a tile's blocks may touch
constexpr int kEntryStride = 256;
constexpr int kTableBytes = 256 * kEntryStride;
constexpr int kStreamBars = 2 * kStreamMaxStages + 2 * 4 + kStreamMaxSlots;
constexpr int kStreamWarps = 12;             // decoding warps
constexpr int kStreamAbs = kStreamWarps * kStreamRows * 8 * 4;       // absmax values of their tiles
constexpr int kStreamScales = 2 * kStreamMaxGroups * 4;              // second-level scales and offsets of a tile
constexpr int kStreamSlack = 512;            // what a warp with fewer blocks than others reads beyond its last row
constexpr int kStreamThreads = 32 * (kStreamWarps + kStreamProducers + kStreamEpilogues);
constexpr int kStreamFixed = kTableBytes + kStreamAbs + 1024 + 64 + 8 * kStreamBars + 16;      // table, absmax values, code2, levels, barriers, abort flag
constexpr int kStreamSmem = 227 * 1024;
// the most quantisation blocks whose token rows a decoding warp keeps in registers; buffers of partial sums
__host__ __device__ constexpr int stream_blocks(int nt) { return nt == 1 ? 7 : 5; }
__host__ __device__ constexpr int stream_bufs(int nt) { return nt == 1 ? 4 : 2; }
constexpr int kStreamSums = kStreamWarps * 4 * stream_bufs(1);       // entries of the table in whose unused halves partial sums lie
static_assert(kStreamSums == kStreamWarps * 8 * stream_bufs(2) && kStreamSums + 8 * kMaxSegments <= 256, "and scaled rank-16 products");

enum : int { kHoldCopies = 1, kHoldClusterSums = 3 };      // nf4ll_test_mid_withhold, as it applies here

struct StreamParams {
  const uint8_t* nib;
  const uint8_t* qabs;
  const float* scale2;
  const float* offset2;
  const float* code2;
  int64_t K;
  int bpr, M;                              // quantisation blocks of a weight row; tokens
  int64_t rows;                            // weight rows
  int groups;                              // second-level groups that a tile's blocks touch at most
  int units, cl, np, teams;                // units; CTAs of a cluster; warps of a team; teams
  // bytes: a row of codes in a stage, from one pair of rows to the next, in front of the absmax codes (behind the scales), a stage; stages of a team
  int row, pitch, off_q, stage, stages;
  int off_ring, off_xch;
  int qabs_bulk;                           // absmax codes may be copied 16 bytes at a time
  int early;                               // the kernel before this one is a rank-16 projection of the same call
  const __half* x;
  int64_t ldx;
  __half* y;
  int64_t ldy;
  const __half* bias;
  // several projections stacked along N (multiples of 16 rows), each with its own rank-16 branch
  int n_seg;
  int64_t seg_end[kMaxSegments];           // first row after the segment
  const float* seg_t[kMaxSegments];        // [M,16] fp32 = drop(x) . A^T, or null (no LoRA)
  const __half* seg_b[kMaxSegments];       // lora_B, offset so that it is indexed by the row of W
  float seg_scale[kMaxSegments];
  int64_t split;                           // gate|up: rows of a half, else 0
  __half* y2;                              // the second half's output
  int64_t ldy2;
  __half* h;                               // silu(first) * second, both halves of a unit in turn; null: left to a kernel of its own
  int64_t ldh;
  int withhold;                            // failure-detection hook: what is never signalled
  uint64_t wait_ns;                        // limit of the waits
  int32_t* status;
};

// offset into the table of the entry of byte I of `w` for this lane (lane_off = 4 * lane < 256): one byte permute
template <int I>
__device__ __forceinline__ uint32_t entry_offset(uint32_t w, uint32_t lane_off) {
  return prmt(w, lane_off, 0x5504u | (I << 4));
}

// the 8 weights of one 32-bit word of codes as four half2 registers (element order: high nibble first). Volatile: the compiler then leaves
// the reads ahead of the MMAs as they are written (27648 x 5120 at 8 rows 20.5 us, 20.8 without).
template <int I>
__device__ __forceinline__ uint32_t table_read(uint32_t table, uint32_t w, uint32_t lane_off) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(table + entry_offset<I>(w, lane_off)));
  return v;
}
__device__ __forceinline__ void decode8(uint32_t table, uint32_t w, uint32_t lane_off, uint32_t (&h)[4]) {
  h[0] = table_read<0>(table, w, lane_off); h[1] = table_read<1>(table, w, lane_off);
  h[2] = table_read<2>(table, w, lane_off); h[3] = table_read<3>(table, w, lane_off);
}

// A wait of a whole warp, bounded by polls and by time; its lanes agree on the outcome. CLUSTER: for barriers on which other CTAs arrive
// (polled, their arrivals wake a parked thread slowly).
struct StreamAbort : Abort {
  uint64_t limit_ns;
};
template <bool CLUSTER = false>
__device__ __forceinline__ bool stream_wait(uint32_t bar, uint32_t parity, const StreamAbort& ab, int code) {
#pragma unroll 1
  for (int i = 0; i < 8; ++i)
    if (__all_sync(0xffffffffu, CLUSTER ? mbar_test_wait_cluster(bar, parity) : mbar_test_wait(bar, parity))) return true;
#pragma unroll 1
  for (int i = 0; i < 64; ++i)
    if (__all_sync(0xffffffffu, CLUSTER ? mbar_test_wait_cluster(bar, parity) : mbar_try_wait(bar, parity))) return true;
  const uint64_t t0 = global_timer_ns();
#pragma unroll 1
  for (uint32_t i = 0; i < (CLUSTER ? kSpinLimit << 4 : kSpinLimit); ++i) {
    if (__all_sync(0xffffffffu, CLUSTER ? mbar_test_wait_cluster(bar, parity) : mbar_try_wait_hint(bar, parity, kParkNs))) return true;
    if (__any_sync(0xffffffffu, *ab.flag != 0)) return false;
    if (__any_sync(0xffffffffu, global_timer_ns() - t0 > ab.limit_ns)) break;
  }
  ab.raise(code);
  return false;
}

// NT: tiles of 8 tokens (M <= 8 NT). S: quantisation blocks per row that a decoding warp takes.
template <int NT, int S>
__global__ void __launch_bounds__(kStreamThreads, 1)
nf4_stream_kernel(const __grid_constant__ StreamParams p) {
  pdl_launch_dependents();
  extern __shared__ __align__(256) uint8_t st_smem[];
  constexpr int kWarps = kStreamWarps, kBufs = stream_bufs(NT), kGroups = (S + 3) / 4;
  constexpr int kEpiWarp = kWarps + kStreamProducers, kBarThreads = kStreamThreads - 32 * kStreamProducers;
  float* s_code2 = reinterpret_cast<float*>(st_smem + kTableBytes + kStreamAbs);
  uint16_t* s_lv = reinterpret_cast<uint16_t*>(s_code2 + 256);
  uint64_t* full = reinterpret_cast<uint64_t*>(s_lv + 32);      // [stages] the tile's codes, absmax codes and second-level scales are here
  uint64_t* empty = full + kStreamMaxStages;               // its team has used them
  uint64_t* part_full = empty + kStreamMaxStages;          // [kBufs] the team's partial sums are here
  uint64_t* part_empty = part_full + 4;
  uint64_t* xch_full = part_empty + 4;                     // [slots] the other CTAs' sums of a unit are here
  volatile int* abort_flag = reinterpret_cast<volatile int*>(xch_full + kStreamMaxSlots);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const StreamAbort ab{{abort_flag, p.status}, p.wait_ns};
  const int cl = p.cl, crank = cl > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int cluster = blockIdx.x / cl, n_clusters = gridDim.x / cl;
  // this CTA's part of every weight row, in quantisation blocks
  const int cb0 = static_cast<int>(static_cast<int64_t>(p.bpr) * crank / cl), nbc = static_cast<int>(static_cast<int64_t>(p.bpr) * (crank + 1) / cl) - cb0;
  // Units of a tile, gate|up of two (the gate rows and the up rows of the same outputs). Unit i of the cluster belongs to team
  // i mod teams, which has stages of its own; its tile j = i * halves + half goes through buffer j mod kBufs to an epilogue warp.
  // The teams divide the buffers, so every barrier has one team or warp a side, which meets its phases one after another.
  const int halves = p.h ? 2 : 1, my_units = (p.units - 1 - cluster) / n_clusters + 1;
  // first weight row of half hf of the cluster's unit i
  auto row_of = [&](int i, int hf) { return (cluster + static_cast<int64_t>(i) * n_clusters) * kStreamRows + (hf ? p.split : 0); };
  // the cluster's tiles in order, with their places in the teams' rings (which turn in step)
  struct Walk { int i, hf, team, st0, ph0; };
  auto walk_slot = [&](const Walk& w, int& phase) {
    const bool wrap = w.st0 + w.hf >= p.stages;
    phase = w.ph0 ^ (wrap ? 1 : 0);
    return w.team * p.stages + (wrap ? w.st0 + w.hf - p.stages : w.st0 + w.hf);
  };
  auto walk_on = [&](Walk& w) {
    if (++w.hf < halves) return;
    w.hf = 0; ++w.i;
    if (++w.team < p.teams) return;
    w.team = 0;
    w.st0 += halves;
    while (w.st0 >= p.stages) { w.st0 -= p.stages; w.ph0 ^= 1; }
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages * p.teams; ++i) {
      mbar_init(smem_u32(full + i), kStreamProducers + 32); mbar_init(smem_u32(empty + i), p.np);
    }
    for (int i = 0; i < kBufs; ++i) { mbar_init(smem_u32(part_full + i), p.np); mbar_init(smem_u32(part_empty + i), 1); }
    if (cl > 1) for (int i = 0; i < kStreamMaxSlots; ++i) mbar_init(smem_u32(xch_full + i), (cl - 1) * 32);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (threadIdx.x >= 32 && threadIdx.x < 48) {
    constexpr float lv[16] = {NF4LL_LEVELS};
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) v = (static_cast<int>(threadIdx.x) - 32 == j) ? lv[j] : v;
    s_lv[threadIdx.x - 32] = __half_as_ushort(__float2half_rn(v));
  }
  __syncthreads();
  if (cl > 1) cluster_arrive();

  // Behind a rank-16 projection of the same call the weights and x may be read at once: that kernel itself went on only
  // after all earlier work on the stream had finished. Behind anything else only the tables are laid out meanwhile.
  bool ok = true;
  if (warp >= kWarps && warp < kEpiWarp) {
    // ----------------------------------------------------------------------------- codes: each warp copies half of a tile's rows, a lane a row; the
    // first one the rows' absmax codes and second-level scales too
    if (!p.early) pdl_wait();
    const int half = warp - kWarps;
    bool copied = false;
    const int64_t last_group = (p.rows * p.bpr >> 8) - 1;
    for (Walk w{0, 0, 0, 0, 1}; w.i < my_units; walk_on(w)) {
      int ph;
      const int slot = walk_slot(w, ph);
      if (!stream_wait(smem_u32(empty + slot), ph, ab, 0x0801) || p.withhold == kHoldCopies) break;
      const int64_t n0 = row_of(w.i, w.hf);
      const uint32_t bar = smem_u32(full + slot), stage = smem_u32(st_smem + p.off_ring + slot * p.stage);
      const uint32_t row_bytes = nbc * 32, abs_bytes = half == 0 && p.qabs_bulk ? kStreamRows * p.bpr : 0;
      if (lane == 0) mbar_arrive_expect_tx(bar, kStreamRows / 2 * row_bytes + abs_bytes);
      __syncwarp();
      if (half == 0) {
        // groups of 256 blocks, four bytes each, hardly ever aligned
        const int64_t g0 = (n0 * p.bpr + cb0) >> 8;
        for (int i = lane; i < p.groups && g0 + i <= last_group; i += 32) {
          stream_cp4(stage + p.off_q - kStreamScales + 4 * i, p.scale2 + g0 + i);
          stream_cp4(stage + p.off_q - kStreamScales / 2 + 4 * i, p.offset2 + g0 + i);
        }
        if (!p.qabs_bulk)                           // absmax codes off a 16-byte boundary: four at a time
          for (int i = 4 * lane; i < kStreamRows * p.bpr; i += 128) stream_cp4(stage + p.off_q + i, p.qabs + n0 * p.bpr + i);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
      }
      if (cl == 1) {
        // two rows lie together there as here
        const int r = half * (kStreamRows / 2) + 2 * lane;
        if (lane < kStreamRows / 4) bulk_load(stage + (r >> 1) * p.pitch, p.nib + (n0 + r) * (p.K / 2), 2 * row_bytes, bar);
      } else {
        const int r = half * (kStreamRows / 2) + lane;
        if (lane < kStreamRows / 2) bulk_load(stage + (r >> 1) * p.pitch + (r & 1) * p.row, p.nib + (n0 + r) * (p.K / 2) + cb0 * 32, row_bytes, bar);
      }
      if (lane == kStreamRows / 2 && abs_bytes) bulk_load(stage + p.off_q, p.qabs + n0 * p.bpr, abs_bytes, bar);
      copied = true;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (*abort_flag && copied) {      // copies still in flight get a millisecond to land before the CTA goes away
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 1000000) {}
    }
    __syncwarp();
  } else {
    // four lanes' copies of an entry per 16-byte store
    const int tid = warp < kWarps ? threadIdx.x : threadIdx.x - 32 * kStreamProducers;
    for (int idx = tid; idx < 256 * 8; idx += kBarThreads) {
      const int v = idx >> 3;                       // byte value: even element in the high nibble
      const uint32_t e = s_lv[v >> 4] | (static_cast<uint32_t>(s_lv[v & 15]) << 16);
      *reinterpret_cast<uint4*>(st_smem + v * kEntryStride + (idx & 7) * 16) = make_uint4(e, e, e, e);
    }
    if (!p.early) pdl_wait();
    if (tid < 256) s_code2[tid] = p.code2[tid];
  }
  // partial sums: 4 NT times 128 bytes of which the table makes no use, between its entries, for a warp's tile
  auto sums = [&](int buf, int w, int c) { return reinterpret_cast<float*>(st_smem + ((buf * kWarps + w) * (4 * NT) + c) * kEntryStride + 128); };

  if (warp < kWarps) {
    // ----------------------------------------------------------------------------- decode
    const int g = lane >> 2, t = lane & 3;
    const int team = warp / p.np, part = warp - team * p.np;
    const int b0 = part * S, nb = max(0, min(S, nbc - b0));      // this warp's blocks, counted from the CTA's first
    // The token rows of the warp's blocks, for the whole kernel: lane (g, t) holds columns 16 t .. 16 t + 15 of token g. (Asked for
    // before the tables are laid out, they come between the first tiles' codes: 27648 x 5120 at 8 rows 22.4 us, 20.8 this way.)
    uint4 x[S][NT][2];
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        x[s][i][0] = x[s][i][1] = make_uint4(0, 0, 0, 0);
        if (s < nb && g + 8 * i < p.M && team < p.teams) {
          const __half* src = p.x + (g + 8 * i) * p.ldx + static_cast<int64_t>(cb0 + b0 + s) * 64 + t * 16;
          x[s][i][0] = __ldg(reinterpret_cast<const uint4*>(src));
          x[s][i][1] = __ldg(reinterpret_cast<const uint4*>(src + 8));
        }
      }
    named_barrier(1, kBarThreads);                  // the tables are there
    const uint32_t lane_off = lane * 4;
    // Rows of the operand tile are weight rows 0, 2, 4, 6, 1, 3, 5, 7 (+ 8): rows lie in pairs, the pairs 32 bytes off a multiple of 128 apart, so
    // that the four rows that half a warp reads at a time are in different banks.
    const int row = g < 4 ? 2 * g : 2 * g - 7;
    const uint8_t* my_codes = st_smem + p.off_ring + (row >> 1) * p.pitch + (row & 1) * p.row + b0 * 32 + t * 8;
    const uint32_t row8 = 4 * p.pitch, table = smem_u32(st_smem);
    // absmax: lane (group, row) decodes four blocks of a row of the tile
    float* abs = reinterpret_cast<float*>(st_smem + kTableBytes) + warp * (kStreamRows * 8);      // this warp's [groups][16 rows][4]
    const int arow = lane & 15, four = lane >> 4 << 2, count = min(4, nb - four);
    const uint32_t at = arow * p.bpr + cb0 + b0 + four;      // the first of them, counted from the tile's first row
    // the team's tiles: units team, team + teams, ...
    const int tiles = team < min(p.teams, my_units) ? ((my_units - 1 - team) / p.teams + 1) * halves : 0;
    int st = 0, ph = 0, j = team * halves, hf = 0;
    // the tile's first quantisation block, of which only the place in a group of 256 matters
    uint32_t q0 = static_cast<uint32_t>(row_of(team, 0)) * p.bpr;
    const uint32_t q_unit = static_cast<uint32_t>(p.teams * n_clusters * kStreamRows) * p.bpr, q_half = halves == 2 ? static_cast<uint32_t>(p.split) * p.bpr : 0;
    for (int n = 0; n < tiles; ++n) {
      const int slot = team * p.stages + st;
      const uint32_t q_low = q0 & 255;              // the tile's first block in its second-level group
      if (!stream_wait(smem_u32(full + slot), ph, ab, 0x0802)) { ok = false; break; }
      const uint8_t* codes = my_codes + slot * p.stage;
      if (four < S) {
        const uint8_t* stage = st_smem + p.off_ring + slot * p.stage + p.off_q;
        const uint32_t* word = reinterpret_cast<const uint32_t*>(stage + (at & ~3u));
        const uint32_t c4 = __funnelshift_r(word[0], word[1], 8 * (at & 3));
        const uint32_t pos = q_low + at - ((q_low + cb0) & ~255u);      // counted from the first group of which there are scales
        const float* sc = reinterpret_cast<const float*>(stage - kStreamScales) + (pos >> 8);
        const float s0 = sc[0], s1 = sc[1], o0 = sc[kStreamMaxGroups], o1 = sc[kStreamMaxGroups + 1];
        const int turn = 256 - static_cast<int>(pos & 255);             // blocks left in the group
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = k < count ? block_absmax(s_code2[(c4 >> (8 * k)) & 255u], k < turn ? s0 : s1, k < turn ? o0 : o1) : 0.f;
        *reinterpret_cast<float4*>(abs + lane * 4) = make_float4(v[0], v[1], v[2], v[3]);
      }
      __syncwarp();
      float4 am[kGroups][2];                        // rows `row` and + 8, four blocks each
#pragma unroll
      for (int a = 0; a < kGroups; ++a) {
        am[a][0] = *reinterpret_cast<const float4*>(abs + a * (kStreamRows * 4) + row * 4);
        am[a][1] = *reinterpret_cast<const float4*>(abs + a * (kStreamRows * 4) + row * 4 + 32);
      }
      float acc[NT][4];
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[i][k] = 0.f;
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const uint2 c0 = *reinterpret_cast<const uint2*>(codes + s * 32);
        const uint2 c1 = *reinterpret_cast<const uint2*>(codes + row8 + s * 32);
        uint32_t lo0[4], hi0[4], lo1[4], hi1[4];
        decode8(table, c0.x, lane_off, lo0); decode8(table, c0.y, lane_off, hi0);     // k 16t..16t+7, +8..+15
        decode8(table, c1.x, lane_off, lo1); decode8(table, c1.y, lane_off, hi1);     // row + 8
        const float4 a0 = am[s >> 2][0], a1 = am[s >> 2][1];
        const float f0 = (s & 3) == 0 ? a0.x : (s & 3) == 1 ? a0.y : (s & 3) == 2 ? a0.z : a0.w;
        const float f1 = (s & 3) == 0 ? a1.x : (s & 3) == 1 ? a1.y : (s & 3) == 2 ? a1.z : a1.w;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          const uint4 xa = x[s][i][0], xb = x[s][i][1];
          float blk[4];
          mma16816_first(blk, lo0[0], lo1[0], lo0[1], lo1[1], xa.x, xa.y);
          mma16816(blk, lo0[2], lo1[2], lo0[3], lo1[3], xa.z, xa.w);
          mma16816(blk, hi0[0], hi1[0], hi0[1], hi1[1], xb.x, xb.y);
          mma16816(blk, hi0[2], hi1[2], hi0[3], hi1[3], xb.z, xb.w);
          acc[i][0] = fmaf(blk[0], f0, acc[i][0]);
          acc[i][1] = fmaf(blk[1], f0, acc[i][1]);
          acc[i][2] = fmaf(blk[2], f1, acc[i][2]);
          acc[i][3] = fmaf(blk[3], f1, acc[i][3]);
        }
      }
      __syncwarp();                                 // everybody has used the codes and the absmax values
      if (lane == 0) mbar_arrive(smem_u32(empty + slot));
      const int buf = j % kBufs;
      if (!stream_wait(smem_u32(part_empty + buf), ((j / kBufs) & 1) ^ 1, ab, 0x0804)) { ok = false; break; }
      // acc[i][0..1]: weight row `row`, tokens 8 i + 2 t, + 1; acc[i][2..3]: that row + 8. Two tokens' rows to 128 bytes, turned by 8 t words so
      // that neither side has bank conflicts.
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        float* to = sums(buf, warp, 4 * i + t);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (8 * i + 2 * t + (k & 1) < p.M) to[((k & 1) * 16 + (k >> 1) * 8 + row + 8 * t) & 31] = acc[i][k];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(part_full + buf));
      if (++st == p.stages) { st = 0; ph ^= 1; }
      if (++hf == halves) { hf = 0; j += (p.teams - 1) * halves; q0 += q_unit - q_half; } else q0 += q_half;
      ++j;
    }
  } else if (warp >= kEpiWarp) {
    // ----------------------------------------------------------------------------- sums of the teams, of the cluster; LoRA, bias, output
    named_barrier(1, kBarThreads);
    if (p.early) pdl_wait();                        // T comes from the kernel this one was launched behind
    if (cl > 1) cluster_wait();
    const int k = lane >> 2, q = lane & 3;          // this lane's token (of a tile of eight) and four of the sixteen rows
    const int src_words = p.M * kStreamRows, xch_words = (cl - 1) * src_words;      // a CTA's sums of a tile; all of a tile
    // The rank-16 products, scaled, go into shared memory once, behind the partial sums: a tile then waits for neither global memory nor
    // the multiplication. Two tokens to 128 bytes, eight entries to a segment.
    auto scaled_t = [&](int sg, int tok) { return reinterpret_cast<float*>(st_smem + (kStreamSums + 8 * sg + (tok >> 1)) * kEntryStride + 128 + 64 * (tok & 1)); };
    {
      static_assert(16 * 4 <= 32 * kStreamEpilogues, "sixteen bytes of a token's product to a lane");
      const int piece = (warp - kEpiWarp) * 32 + lane;
      float4 f[kMaxSegments];
#pragma unroll
      for (int sg = 0; sg < kMaxSegments; ++sg)
        if (sg < p.n_seg && p.seg_t[sg] && piece < 4 * p.M) f[sg] = __ldcg(reinterpret_cast<const float4*>(p.seg_t[sg]) + piece);
#pragma unroll
      for (int sg = 0; sg < kMaxSegments; ++sg)
        if (sg < p.n_seg && p.seg_t[sg] && piece < 4 * p.M) {
          const float s = p.seg_scale[sg];
          reinterpret_cast<float4*>(scaled_t(sg, piece >> 2))[piece & 3] = make_float4(f[sg].x * s, f[sg].y * s, f[sg].z * s, f[sg].w * s);
        }
      named_barrier(2, 32 * kStreamEpilogues);
    }
    // units go round the warps, whose buffers differ; gate|up with two buffers is one warp's
    const int finishing = kBufs / halves < kStreamEpilogues ? 1 : kStreamEpilogues;
    // what a tile's result is made of besides sums and products, requested before they are waited for
    int seg = -1;                                   // its segment, where that has a rank-16 branch
    uint2 bias;
    uint4 br[4][2];
    auto request = [&](int i, int hf) {
      seg = -1;
      bias = make_uint2(0, 0);
      if (i >= my_units || (cl > 1 && crank != i % cl)) return;
      const int64_t n0 = row_of(i, hf);
      int sg = 0;
      while (sg + 1 < p.n_seg && n0 >= p.seg_end[sg]) ++sg;
      if (p.bias) bias = __ldg(reinterpret_cast<const uint2*>(p.bias + n0 + 4 * q));
      if (!p.seg_t[sg]) return;
      seg = sg;
      const uint4* bp = reinterpret_cast<const uint4*>(p.seg_b[sg] + (n0 + 4 * q) * 16);
#pragma unroll
      for (int r = 0; r < 4; ++r) { br[r][0] = __ldg(bp + 2 * r); br[r][1] = __ldg(bp + 2 * r + 1); }
    };
    for (int i = warp - kEpiWarp; ok && i < my_units && warp - kEpiWarp < finishing; i += finishing) {
      const int owner = cl > 1 ? i % cl : 0, slot = cl > 1 ? i / cl : 0, team = p.teams > 1 ? i % p.teams : 0;
      float gate[NT][4];                            // gate|up: the first half's results as rounded
      for (int hf = 0; hf < halves; ++hf) {
        const int j = i * halves + hf, buf = j % kBufs;
        const int64_t n0 = row_of(i, hf);
        const bool mine = crank == owner;
        request(i, hf);
        ok = stream_wait(smem_u32(part_full + buf), (j / kBufs) & 1, ab, 0x0806);
        if (!ok) break;
        float4 v[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          v[n] = make_float4(0.f, 0.f, 0.f, 0.f);
          const float* from = sums(buf, team * p.np, 4 * n + (k >> 1)) + (((k & 1) * 16 + 4 * q + 8 * (k >> 1)) & 31);
          if (8 * n + k < p.M)
#pragma unroll 4
            for (int w = 0; w < p.np; ++w) {
              const float4 b = *reinterpret_cast<const float4*>(from + w * (4 * NT * kEntryStride / 4));
              v[n].x += b.x; v[n].y += b.y; v[n].z += b.z; v[n].w += b.w;
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(part_empty + buf));
        if (!mine) {
          const int src = crank < owner ? crank : crank - 1;
          const uint32_t base = map_to_cta(smem_u32(st_smem + p.off_xch) + ((slot * halves + hf) * xch_words + src * src_words) * 4, owner);
#pragma unroll
          for (int n = 0; n < NT; ++n)
            if (8 * n + k < p.M)
              asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(base + (n * 128 + k * 16 + 4 * q) * 4), "f"(v[n].x), "f"(v[n].y), "f"(v[n].z),
                           "f"(v[n].w) : "memory");
          if (!(p.withhold == kHoldClusterSums && crank == cl - 1)) mbar_arrive_remote(map_to_cta(smem_u32(xch_full + slot * halves + hf), owner));
          continue;
        }
        if (cl > 1) {
          ok = stream_wait<true>(smem_u32(xch_full + slot * halves + hf), 0, ab, 0x0807);
          if (!ok) break;
          // the parts of the contraction in ascending order: a fixed order
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            if (8 * n + k < p.M) {
              const float* from = reinterpret_cast<const float*>(st_smem + p.off_xch) + (slot * halves + hf) * xch_words + n * 128 + k * 16 + 4 * q;
              float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
              for (int r = 0; r < cl; ++r) {
                const float4 b = r == crank ? v[n] : *reinterpret_cast<const float4*>(from + (r < crank ? r : r - 1) * src_words);
                a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
              }
              v[n] = a;
            }
          }
        }
        // two ranks side by side: even and odd ones add up apart
        uint64_t l2[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) l2[n][0] = l2[n][1] = l2[n][2] = l2[n][3] = 0;
        if (seg >= 0) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint64_t t2[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              const float4* from = reinterpret_cast<const float4*>(scaled_t(seg, 8 * n + k < p.M ? 8 * n + k : 0)) + 2 * c;
              const float4 a = from[0], b = from[1];
              t2[n][0] = f32x2(a.x, a.y); t2[n][1] = f32x2(a.z, a.w); t2[n][2] = f32x2(b.x, b.y); t2[n][3] = f32x2(b.z, b.w);
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const uint32_t w[4] = {br[r][c].x, br[r][c].y, br[r][c].z, br[r][c].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const uint64_t b2 = half2_to_f32x2(w[e]);
#pragma unroll
                for (int n = 0; n < NT; ++n) l2[n][r] = fma2(t2[n][e], b2, l2[n][r]);
              }
            }
          }
        }
        const float2 blo = __half22float2(*reinterpret_cast<const __half2*>(&bias.x)), bhi = __half22float2(*reinterpret_cast<const __half2*>(&bias.y));
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const int tok = 8 * n + k;
          if (tok < p.M) {
            float l[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) { const float2 f = f32x2_split(l2[n][r]); l[r] = f.x + f.y; }
            const uint2 out = make_uint2(pack_half2_rn((v[n].x + blo.x) + l[0], (v[n].y + blo.y) + l[1]), pack_half2_rn((v[n].z + bhi.x) + l[2], (v[n].w + bhi.y) + l[3]));
            __half* dst = p.split && n0 >= p.split ? p.y2 + tok * p.ldy2 + (n0 - p.split) : p.y + tok * p.ldy + n0;
            *reinterpret_cast<uint2*>(dst + 4 * q) = out;
            if (p.h) {
              // the product of the rounded values, as the stand-alone kernel would read them
              const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&out.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&out.y));
              const float f[4] = {f0.x, f0.y, f1.x, f1.y};
              if (hf == 0) {
#pragma unroll
                for (int r = 0; r < 4; ++r) gate[n][r] = f[r];
              } else {
                float o[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) o[r] = gate[n][r] * fast_sigmoid(gate[n][r]) * f[r];
                *reinterpret_cast<uint2*>(p.h + tok * p.ldh + (n0 - p.split) + 4 * q) = make_uint2(pack_half2_rn(o[0], o[1]), pack_half2_rn(o[2], o[3]));
              }
            }
          }
        }
      }
    }
  }
  __syncwarp();
  if (cl > 1) {
    if (warp < kEpiWarp) cluster_wait();
    cluster_sync_all();                             // nobody leaves while a peer may still write to its shared memory
  }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
struct StreamPlan {
  int cl, np, s, teams, stages, row, pitch, off_q, stage, off_ring, off_xch, smem, groups;
  int64_t units;
  int clusters;
  double us;
};

template <int NT>
static const void* stream_kernel(int s) {
  constexpr int kMost = stream_blocks(NT);
  switch (s) {
    case 1: return reinterpret_cast<const void*>(nf4_stream_kernel<NT, 1>);
    case 2: return reinterpret_cast<const void*>(nf4_stream_kernel<NT, 2>);
    case 3: return reinterpret_cast<const void*>(nf4_stream_kernel<NT, 3>);
    case 4: return reinterpret_cast<const void*>(nf4_stream_kernel<NT, 4>);
    case 5: return reinterpret_cast<const void*>(nf4_stream_kernel<NT, 5>);
    case 6: return reinterpret_cast<const void*>(nf4_stream_kernel<NT, kMost < 6 ? kMost : 6>);
    default: return reinterpret_cast<const void*>(nf4_stream_kernel<NT, kMost>);
  }
}

// How many clusters of `cl` CTAs the current device holds at once, a CTA taking an SM to itself
static int stream_clusters(int cl) {
  constexpr int kDevices = 64;
  static int known[kDevices][kStreamMaxCluster + 1];      // 0: not asked yet; written with the same value by any thread
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
  int n = __atomic_load_n(&known[dev][cl], __ATOMIC_RELAXED);
  if (n > 0) return n;
  if (cl == 1) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 0;
  } else {
    const void* kernel = stream_kernel<1>(1);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem) != cudaSuccess) return 0;
    if (cl > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return 0;
    PdlLaunch probe(dim3(cl), dim3(kStreamThreads), kStreamSmem, nullptr, cl, 1, false, false);
    probe.cfg.numAttrs = 1;                    // the cluster dimension only
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &probe.cfg) != cudaSuccess) n = 0;
  }
  if (n > 0) __atomic_store_n(&known[dev][cl], n, __ATOMIC_RELAXED);
  else (void)cudaGetLastError();
  return n;
}

// Time of a plan in us, behind other calls, without a rank-16 branch: of a launch, of the clusters' exchange, of a tile, of the blocks that a
// scheduler's warps decode one after another, of a tile's traffic through shared memory (a ring of two stages does not always hide the
// fetch). Fitted to 300 plans of 24 weights from 1536 x 1536 to 37888 x 3584 at 8 and at 16 rows; picking by it takes 0.7 % longer than the
// fastest plans at 8 rows, 8 % at worst.
static double stream_us(int nt, int cl, int64_t tiles, int teams, int np, int s, int64_t blocks, int stages) {
  const double turns = static_cast<double>((tiles + teams - 1) / teams), chain = turns * ((np * teams + 3) / 4) * s, r = static_cast<double>(tiles);
  if (nt == 1) return 2.57 + (cl > 1 ? 1.63 + 0.173 * r : 0) + 0.45 * r + turns * (0.08 + 0.01 * s) + 0.0156 * chain + (stages < 3 ? 0.0082 : 0.0053) * r * static_cast<double>(blocks);
  if (cl > 1) return 3.8 + r * (0.5 + 0.06 * cl + 0.025 * s + 0.018 * static_cast<double>(blocks));
  return (3.5 + 0.303 * r + 0.0476 * turns * s + 0.0166 * r * static_cast<double>(blocks)) * (s == 5 ? 1.15 : 1.0);
}

// With a rank-16 projection in front whose CTAs hold `busy` SMs for a while: a grid that wants more SMs than are left starts the last of its
// CTAs that much later. What that costs a plan, against another round of tiles on the SMs that are free (and 0.1 us a tile for the
// products where the tokens are few). Fitted to 824 calls at 1 to 16 rows, of which both were timed: picking by it takes 0.2 % (from
// nine rows on 0.3 %) longer than the faster of the two, without it 0.4 % (1.4 %). us with / without: Q|K|V at 9 rows 1536 x 8960 11.4 / 14.2, 1024 x 8192
// 9.6 / 11.5; 1152 x 9088 at 1 row 8.4 / 9.3, 1024 x 27648 at 8 rows 11.9 / 13.7.
static double stream_beside_us(int nt, bool late, int64_t tiles, int64_t K) {
  return (nt == 1 ? 0.1 * static_cast<double>(tiles) : 0) + (late ? fmin((nt == 1 ? 0.25 : 0.5) + 0.00015 * static_cast<double>(K), 1.9) : 0);
}

// M: tokens, sixteen at most. `force`: low byte warps of a team, next byte CTAs of a cluster, next byte teams (0: free)
static bool stream_search(int64_t M, int64_t N, int64_t K, bool pair, int busy, int force, StreamPlan* best) {
  const int nt = M > 8 ? 2 : 1;
  const int64_t bpr = K / 64, units = N / kStreamRows / (pair ? 2 : 1);
  const int warps = kStreamWarps, f_np = force & 255, f_cl = force >> 8 & 255, f_teams = force >> 16, halves = pair ? 2 : 1;
  bool found = false;
  if (units > (1 << 24)) return false;
  for (int cl = 1; cl <= (nt == 1 ? kStreamMaxCluster : 8) && cl <= bpr; ++cl) {
    if (f_cl && cl != f_cl) continue;
    // Beyond eight only for rows that eight CTAs cannot hold: such clusters leave SMs of a GPC idle. The kernel for middling batches takes
    // what is left: rows longer still, and weights so tall that a cluster's sums leave room for one stage. us at 1 and 8 rows, here / there
    // (and before, when all of it went to the tile kernels): 4096 x 45056 31.4, 32.0 / 48.6, 48.9 (76); 8192 x 49152 75.0, 75.7 / 94 (162);
    // 16384 x 53248 145, 191 (with one stage 268) / 193 (330).
    if (cl > 8 && found && best->cl <= 8) break;
    if (found && best->cl == 1) break;            // a cluster costs 2 us and more: only where one CTA cannot hold the tokens
    const int64_t blocks = (bpr + cl - 1) / cl;
    const int least = static_cast<int>((blocks + stream_blocks(nt) - 1) / stream_blocks(nt));
    if (blocks > warps * stream_blocks(nt)) continue;
    const int all = stream_clusters(cl);
    if (all <= 0) continue;
    // The projection's SMs, eight of a GPC at a time, leave room for two clusters less at least (one of more than eight CTAs): 44 of 45
    // clusters of three wait for them and 43 do not, 32 of 33 of four and 31, 15 of 15 of nine and 14, whether it has 8 or 16 of them.
    const int others = (stream_clusters(1) - busy) / cl, fewer = cl == 1 ? all : cl > 8 ? all - 1 : all - 2;
    const int beside = busy <= 0 ? all : fewer < others ? fewer : others;
    for (int turn = 0; turn < (beside > 0 && beside < all ? 2 : 1); ++turn) {
      const int most = turn ? beside : all;
      StreamPlan p{};
      p.cl = cl; p.units = units;
      const int64_t rounds = (units + most - 1) / most;
      p.clusters = static_cast<int>((units + rounds - 1) / rounds);
      p.row = static_cast<int>(blocks * 32);
      p.pitch = (2 * p.row + 95) / 128 * 128 + 32;
      p.groups = static_cast<int>((15 * bpr + blocks + 254) / 256 + 1);
      const int64_t slots = (rounds + cl - 1) / cl * halves;
      if (p.groups > kStreamMaxGroups || (cl > 1 && slots > kStreamMaxSlots)) continue;
      p.off_xch = (kStreamFixed + 127) / 128 * 128;
      p.off_ring = static_cast<int>(p.off_xch + (cl > 1 ? (slots * (cl - 1) * M * kStreamRows * 4 + 127) / 128 * 128 : 0));
      p.off_q = kStreamRows / 2 * p.pitch + kStreamScales;
      p.stage = static_cast<int>((p.off_q + kStreamRows * bpr + 16 + 127) / 128 * 128);
      const int64_t room = kStreamSmem - p.off_ring - kStreamSlack;
      const int fit = static_cast<int>(room / p.stage < kStreamMaxStages ? room / p.stage : kStreamMaxStages);
      if (cl > 8 && fit < 2) continue;
      for (int np = least; np <= warps && np <= blocks; ++np) {
        if (f_np && np != (f_np < least ? least : f_np < warps && f_np < blocks ? f_np : warps < blocks ? warps : static_cast<int>(blocks))) continue;
        p.s = static_cast<int>((blocks + np - 1) / np);
        p.np = np;
        int most_teams = 0;
        for (int t = 1; t * halves <= stream_bufs(nt) && t * np <= warps && t <= fit && (t == 1 || t <= rounds); t *= 2) most_teams = t;
        for (int teams = 1; teams <= most_teams; teams *= 2) {
          if (f_teams && teams != (f_teams < most_teams ? f_teams : most_teams)) continue;
          p.teams = teams;
          p.stages = fit / teams;
          p.smem = p.off_ring + p.stages * teams * p.stage + kStreamSlack;
          p.us = stream_us(nt, cl, rounds * halves, teams, np, p.s, blocks, p.stages);
          if (busy > 0) p.us += stream_beside_us(nt, p.clusters > beside, rounds * halves, K);
          if (!found || p.us < best->us) { *best = p; found = true; }
        }
      }
    }
  }
  return found;
}

static bool stream_plan(int64_t M, int64_t N, int64_t K, bool pair, int busy, int force, StreamPlan* plan) {
  static thread_local KeptPlans<StreamPlan, 6> kept;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const int64_t key[6] = {M, N, K, busy, force, static_cast<int64_t>(dev) << 1 | (pair ? 1 : 0)};
  return kept.get(key, plan, [&](StreamPlan* p) { return stream_search(M, N, K, pair, busy, force, p); });
}

// The plan of a call of M <= 16 tokens. Beyond eight, gate|up forms its product in the launch only where one CTA holds a row: one warp
// finishes both halves of a unit, which is too slow for a cluster's (55296 x 5120 at 16 rows 107 us).
static bool stream_call_plan(int64_t M, int64_t N, int64_t K, bool gate_up, int busy, int force, bool* fused, StreamPlan* plan) {
  *fused = gate_up;
  if (stream_plan(M, N, K, gate_up, busy, force, plan) && !(gate_up && M > 8 && plan->cl > 1)) return true;
  if (!gate_up || M <= 8) return false;
  *fused = false;
  return stream_plan(M, N, K, false, busy, force, plan);
}

bool stream_takes(int64_t M, int64_t N, int64_t K, bool gate_up) {
  if (K <= 64 * kStreamWarps * stream_blocks(1) && N <= (int64_t(1) << 28)) return true;      // one CTA holds a tile's rows
  StreamPlan p{};
  return stream_plan(M < 8 ? M : 8, N, K, gate_up, 0, 0, &p);
}

// Beside the plan's own time: the gated product's launch, or what it costs the warp that forms it, of a tile; and with rank-16 products
// made by this call, what is left of that kernel and what a tile's epilogue takes.
double stream_time_us(int64_t M, int64_t N, int64_t K, bool gate_up, int busy) {
  bool fused = false;
  StreamPlan p{};
  if (!stream_call_plan(M, N, K, gate_up, busy, 0, &fused, &p)) return 1e30;
  const double tiles = static_cast<double>((p.units + p.clusters - 1) / p.clusters * (fused ? 2 : 1));
  return p.us + (fused ? 0.35 * tiles : gate_up ? 1.3 : 0) + (busy > 0 ? 1.3 + (gate_up ? 0.25 : 0.1) * tiles : 0);
}

int stream_forward_launch(const StreamCall& c, bool early, int force, int32_t* status, cudaStream_t stream) {
  const nf4ll_mat* W = c.W;
  // sixteen tokens at a time, eight where rows are too long for that; more than sixteen are asked for by the tuning hook only
  for (int64_t m0 = 0, rows = 0; m0 < c.M; m0 += rows) {
    const int64_t left = c.M - m0;
    const int busy = early && m0 == 0 ? c.busy : 0;
    bool fused = false;
    StreamPlan pl{};
    rows = left < 16 ? left : 16;
    if (!stream_call_plan(rows, W->N, W->K, c.h != nullptr, busy, force, &fused, &pl)) {
      rows = left < 8 ? left : 8;
      if (!stream_call_plan(rows, W->N, W->K, c.h != nullptr, busy, force, &fused, &pl)) {
        set_detail("weight-streaming kernel: W[%lld,%lld] is too large", static_cast<long long>(W->N), static_cast<long long>(W->K));
        return NF4LL_ERR_SHAPE;
      }
    }
    const int nt = rows > 8 ? 2 : 1;
    StreamParams p{};
    p.nib = W->nib; p.qabs = W->qabs; p.scale2 = W->scale2; p.offset2 = W->offset2; p.code2 = W->code2;
    p.K = W->K; p.bpr = static_cast<int>(W->K / 64); p.M = static_cast<int>(rows);
    p.units = static_cast<int>(pl.units); p.cl = pl.cl; p.np = pl.np; p.teams = pl.teams;
    p.row = pl.row; p.pitch = pl.pitch; p.off_q = pl.off_q; p.stage = pl.stage; p.stages = pl.stages;
    p.rows = W->N; p.groups = pl.groups;
    p.off_xch = pl.off_xch; p.off_ring = pl.off_ring;
    p.qabs_bulk = (reinterpret_cast<uintptr_t>(W->qabs) & 15) == 0;
    p.early = early && m0 == 0 ? 1 : 0;
    p.x = static_cast<const __half*>(c.x) + m0 * c.ldx; p.ldx = c.ldx;
    p.y = static_cast<__half*>(c.y) + m0 * c.ldy; p.ldy = c.ldy;
    p.bias = static_cast<const __half*>(c.bias);
    p.n_seg = c.n_seg;
    for (int i = 0; i < c.n_seg; ++i) {
      p.seg_end[i] = c.seg_end[i];
      p.seg_t[i] = c.seg_t[i] ? c.seg_t[i] + m0 * 16 : nullptr;
      p.seg_b[i] = c.seg_b[i]; p.seg_scale[i] = c.seg_scale[i];
    }
    if (c.h) {
      p.split = c.split;
      p.y2 = static_cast<__half*>(c.y2) + m0 * c.ldy2; p.ldy2 = c.ldy2;
      if (fused) { p.h = static_cast<__half*>(c.h) + m0 * c.ldh; p.ldh = c.ldh; }
    }
    p.status = status;
    p.withhold = c.withhold;
    p.wait_ns = c.withhold ? static_cast<uint64_t>(c.wait_us) * 1000 : kWaitLimitNs;
    const void* kernel = nt == 1 ? stream_kernel<1>(pl.s) : stream_kernel<2>(pl.s);
    NF4LL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem));
    if (pl.cl > 8) NF4LL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    PdlLaunch lc(dim3(static_cast<unsigned>(pl.clusters * pl.cl)), dim3(kStreamThreads), pl.smem, stream, pl.cl > 1 ? pl.cl : 0, pl.cl > 1 ? 1 : 0);
    void* args[] = {&p};
    NF4LL_CUDA(cudaLaunchKernelExC(&lc.cfg, kernel, args));
    if (c.h && !fused)
      if (int rc = nf4ll_swiglu_forward(p.y, c.ldy, p.y2, c.ldy2, static_cast<__half*>(c.h) + m0 * c.ldh, c.ldh, rows, c.split, stream)) return rc;
  }
  return NF4LL_OK;
}

}  // namespace nf4ll
