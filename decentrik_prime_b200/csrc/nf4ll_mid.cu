// Middling batches (17 to some hundreds of token rows, 2560 against small weights; from 9 on where it is ahead of the
// streaming kernel), forward and backward-dX: the WEIGHTS are the 128-row operand of
// tcgen05.mma, the tokens its N operand (any multiple of 16 up to 240 columns, 224 with LoRA: what shared memory holds two tiles of), the contraction is cut over the CTAs of a
// thread-block cluster. Serves the reference call sites solution/fast_qwen.py:947, 1037, 1080-1112 and, backward, 1310-1364.
//
//   forward    y^T[128 weight rows, tokens] = W[rows, K] . x^T
//   backward   dx^T[128 columns, tokens]    = (W[N, columns])^T . dy^T          (fp32 in tensor memory)
//
// Why: the kernels whose 128-row operand is the batch decode a weight once per 256 rows (or pad a short batch to 128), cut
// small outputs up by a cooperative launch that meets in global memory, and cost 16 us for 17 rows of 1536 x 1536, where this
// one costs 7.5. Here a weight is decoded once per up to 256 tokens, and what a launch costs is its pipeline.
//
// What bounds it. Items of 128 x 128 weights go round four teams of decoding warps; the weights are the bit-exact fp16 ones.
//   forward    a lane of tensor memory is a weight row: a thread turns 64 bytes of codes into 128 weights with a table of fp32
//              level pairs in shared memory (an 8-byte load, a packed multiply and one conversion per pair; 73 clocks per 2048
//              weights and SM against 108 for byte permutes over a block's sixteen products) and writes them with tcgen05.st
//              as the A operand, so that shared memory carries the codes, the table and the tokens only.
//   backward   the contraction runs down the columns of codes, so the operand goes through shared memory (MN-major).
// With few tokens the decode is the pace (0.46 us per item forward, 0.6 backward), with many the tensor core and the feeding
// of token tiles (0.14 us + 3.1 ns per token). A single warp issues about one instruction per ten clocks beside sixteen that
// decode, so the loops of the issuing warp and of the producers are kept short: divisions by run-time values in them cost a
// third of the kernel's time. The MMAs are issued under elect.sync by a warp that walks the loop as a whole: 32 clocks per MMA
// of 64 columns, which is the tensor core's rate, against 66 from a lane picked by a branch on the thread index.
// Codes come in boxes of 128 rows x 128 bytes (64-byte rows were fed at half the rate), backward with one row block 64.
//
// The CTAs of a cluster take slices of the contraction and then exchange their partial sums through distributed shared memory:
// each finishes a part of the unit's tokens, adding the slices up in ascending order (results do not depend on timing). No
// counters to clear, no co-residency of the whole grid, and a programmatic launch like any other. A cluster goes through its
// units one after another; four warps finish a unit while the next one is decoded (two accumulators where tensor memory has
// room), and all twenty finish the last one. Outputs are turned round in shared memory and stored 16 bytes at a time: with
// 2-byte stores from the accumulators' layout the four warps fell behind the decode (17920 x 1536 at 512 rows 40 us, now 34).
//
// Measured, calls in a row, before (tile and swapped-operand kernels) and now, us: forward 1536 x 1536 at 17 / 333 / 951 rows
// 16.3 / 21.5 / 22.9, now 7.5 / 10.3 / 12.3; 8960 x 1536 at 187 rows 24.4, now 12.0; 5120 x 27648 at 64 rows 55, now 44;
// 18944 x 3584 at 333 rows 57, now 46; 27648 x 5120 at 333 rows 148, now 96. Backward 1536 x 8960 at 187 rows 24.4, now 14.7;
// 18944 x 3584 at 187 rows 69, now 40; 5120 x 27648 at 333 rows 164, now 99.
//
// Every wait is bounded and reports through the status word (tested by withholding codes, rank-16 operands and partial sums).
// Warp roles: 0 codes, 1 MMA issue, 2 token tiles, 3 idle, 4-7 rank-16 operands and epilogue, 8-23 decode.
#include <cuda.h>

#include "nf4ll_mid.cuh"
#include "nf4ll_pair.cuh"

namespace nf4ll {

constexpr int kMidTeams = 4;                               // teams of four decode warps, an item each, in turn
constexpr int kMidEpiWarp = 4, kMidDecodeWarp = 8;
constexpr int kMidThreads = 32 * (kMidDecodeWarp + 4 * kMidTeams);
constexpr int kMidBars = 8;                                // barrier pairs of the decoded-weight slots
constexpr int kMidCodeBytes = 128 * 128;                   // codes of a stage: 128 rows x four quantisation blocks, two items (backward with one row block: one)
constexpr int kMidMaxCodes = 8;
constexpr int kMidLutBytes = 256 * 128;
constexpr int kMidTurnRow = 32 * 4 + 16, kMidTurnBytes = 8 * kMidTurnRow;      // eight tokens of a warp's 32 columns, fp32, padded
constexpr int kMidSmem = 227 * 1024;
// Forward, up to so many rows: the rank-16 product keeps its 32 bits, as in the streaming kernel: two fp16 parts of it are
// multiplied (22 bits), and values that fp16 cannot hold are added in fp32. Longer batches round it to fp16 like the tile kernels and the dense GEMM.
// Where the branch is most of the output, rel-L2 against fp64 of 5120 x 27648 / 27648 x 5120 at 64 rows 2.6e-4 / 2.9e-4
// rounded, 2.07e-4 / 2.08e-4 in two parts, which is the output's own rounding. Time with LoRA, rounded / in two parts: 5120 x 27648 at 64 rows
// 47.0 / 47.2 us, 27648 x 5120 at 64 rows 43.0 / 43.7, gate|up of it at 24 rows 44.4 / 44.6, 1536 x 1536 at 24 rows 9.3 / 9.5.
constexpr int64_t kMidSplitRows = 64;

enum : int { kHoldCodes = 1, kHoldRank16 = 2, kHoldSums = 3 };      // nf4ll_test_mid_withhold

struct MidParams {
  const uint8_t* qabs;
  const float* scale2;
  const float* offset2;
  const float* code2;
  int N, K, M, NO, steps;          // steps: 64-wide steps of the contraction
  int nt, cl, tiles_t, units, nbuf, na, nx, nc, nc_log;
  int ts;                          // token columns that a CTA of the cluster finishes
  int off_a, off_x, off_lora, off_xch, off_lut, off_turn, off_misc;      // shared memory
  int early, qabs_mode, x_alias, any_lora;
  int withhold;                    // failure-detection hook: what is never signalled
  uint64_t wait_ns;                // limit of the waits
  int split;                       // forward: the tokens' side of the rank-16 operands in two fp16 parts
  __half* out;
  int64_t ldo;
  const __half* bias;
  int accumulate;
  int n_seg;
  int seg_end[kMaxSegments];
  const float* seg_left[kMaxSegments];
  const __half* seg_right[kMaxSegments];
  float seg_scale[kMaxSegments];
  const uint8_t* mask;
  int64_t ld_mask;
  float keep_scale;
  int gu_inter;
  __half* out_u;
  int64_t ldu;
  __half* out_h;
  int64_t ldh;
  int32_t* status;
};

__device__ __forceinline__ bool mid_elect() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// D[tmem] (+)= A[tmem] . B[smem]
__device__ __forceinline__ void mid_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mid_tmem_st16(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void mid_tmem_ld8(uint32_t taddr, float (&f)[8]) {
  uint32_t v[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "r"(taddr)
      : "memory");
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v[j]);
}
__device__ __forceinline__ void mid_tmem_add(uint32_t taddr, float d) {      // one column
  uint32_t v;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(taddr) : "memory");
  tmem_ld_wait();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(__float_as_uint(__uint_as_float(v) + d)) : "memory");
  tmem_st_wait();
}
__device__ __forceinline__ void mid_st_cluster(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// two weights of a byte of codes through the table of level pairs: fp32 products, each rounded once (the values of decode_word)
template <int I>
__device__ __forceinline__ uint32_t mid_pair(uint32_t w, uint32_t lut, uint64_t absmax2) {
  const uint32_t byte = prmt(w, 0u, 0x4440u | I);
  uint32_t addr, d;
  asm("mad.lo.u32 %0, %1, 128, %2;" : "=r"(addr) : "r"(byte), "r"(lut));
  asm("{\n\t.reg .b64 v;\n\t.reg .f32 a, b;\n\t"
      "ld.shared.b64 v, [%1];\n\t"
      "mul.rn.f32x2 v, v, %2;\n\t"
      "mov.b64 {a, b}, v;\n\t"
      "cvt.rn.f16x2.f32 %0, b, a;\n\t}"
      : "=r"(d) : "r"(addr), "l"(absmax2));
  return d;
}
__device__ __forceinline__ uint4 mid_decode8(uint32_t w, uint32_t lut, uint64_t absmax2) {
  return make_uint4(mid_pair<0>(w, lut, absmax2), mid_pair<1>(w, lut, absmax2), mid_pair<2>(w, lut, absmax2), mid_pair<3>(w, lut, absmax2));
}
__device__ __forceinline__ uint64_t mid_twice(float v) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}

// A wait of a whole warp. Its lanes vote, so that they agree on the outcome: the tensor-memory instructions, elect.sync and the
// barriers behind it want all of them, and a lane that saw the phase complete while another saw the abort flag would go on alone.
// (Time without / with the vote, us: 18944 x 3584 at 333 rows forward 45.4 / 45.8, backward 72.0 / 73.0, 8960 x 1536 at 187 rows 12.2 / 11.7.)
// Bounded by polls and by time; CLUSTER: for barriers on which other CTAs arrive (polled, their arrivals wake a parked thread slowly).
struct MidAbort : Abort {
  uint64_t limit_ns;
};
template <bool CLUSTER = false>
__device__ __forceinline__ bool mid_wait(uint32_t bar, uint32_t parity, const MidAbort& ab, int code) {
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
// Copies or MMAs that may be under way when the kernel gives up get a millisecond to finish
__device__ __forceinline__ void mid_drain(uint32_t bar, uint32_t parity) {
  const uint64_t t0 = global_timer_ns();
  for (int i = 0; i < (1 << 16) && !mbar_test_wait(bar, parity) && global_timer_ns() - t0 < 1000000; ++i) {}
}

template <int MODE, int RB>
__global__ void __launch_bounds__(kMidThreads, 1)
nf4_mid_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_nib, const __grid_constant__ MidParams p) {
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sCode = smem_u32(smem);                           // [nc][128 rows][128 B], 128-byte swizzle
  const uint32_t sA = sCode + p.off_a;                             // backward: [na][2][128 rows][128 B] decoded weights, 128-byte swizzle
  const uint32_t sX = sCode + p.off_x;                             // [nx][nt rows][128 B] token tiles, 128-byte swizzle
  const uint32_t sL = sCode + p.off_lora;                          // rank-16 operands: [RB][4096] weights' side | [RB][nt * 32] tokens' side
  const uint32_t sXch = sCode + p.off_xch;                         // partial sums of the other CTAs of the cluster
  const uint32_t sLut = sCode + p.off_lut;
  uint8_t* misc = smem + p.off_misc;
  float* sCode2 = reinterpret_cast<float*>(misc);
  float* sLv = sCode2 + 256;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sLv + 16);
  uint64_t* a_full = bars;                       // [kMidBars] the item's weights are written (four warps) and its token tiles here (items of row block 0)
  uint64_t* a_empty = a_full + kMidBars;         // [kMidBars] the MMAs that read them have completed
  uint64_t* c_full = a_empty + kMidBars;         // [kMidMaxCodes]
  uint64_t* c_empty = c_full + kMidMaxCodes;
  uint64_t* acc_full = c_empty + kMidMaxCodes;   // [2]
  uint64_t* acc_empty = acc_full + 2;            // [2]
  uint64_t* l_full = acc_empty + 2;
  uint64_t* l_empty = l_full + 1;
  uint64_t* xch_full = l_empty + 1;              // the other CTAs' partial sums of this CTA's columns are here
  uint64_t* xch_free = xch_full + 1;             // the other CTAs are ready for this CTA's partial sums
  uint64_t* drain = xch_free + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  static_assert((1024 + 64 + 8 * (2 * kMidBars + 2 * kMidMaxCodes + 9) + 8) % 16 == 0, "the words of `wide` are read sixteen bytes at a time");
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint32_t* wide = tmem_slot + 2;                // [2 units in turn][RB][4]: tokens beyond fp16's range, sixteen to a word, bits 0, 2, 4, ... (16-byte aligned)

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const MidAbort ab{{abort_flag, p.status}, p.wait_ns};
  const int cl = p.cl;
  const int crank = cl > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int cluster = blockIdx.x / cl, n_clusters = gridDim.x / cl;
  const int bpr = p.K >> 6;
  // this CTA's slice of the contraction, in groups of kHalves * 2 steps. An item is 128 x 128 weights; a group has
  // kHalves * RB, in the order (half, row block). The last item of the whole contraction may be of one step or of none.
  constexpr int kHalves = MODE == kBwd ? 1 : 2;
  constexpr int kPer = MODE == kBwd && RB == 1 ? 1 : 2;          // items of a stage of codes
  constexpr int kStage = kMidCodeBytes / 2 * kPer;
  const int groups_all = (p.steps + 2 * kHalves - 1) / (2 * kHalves);
  const int grp0 = groups_all * crank / cl, grp1 = groups_all * (crank + 1) / cl;
  // first weight row (forward) or output column (backward) of a unit's row block
  auto row0_of = [&](int unit, int rb) {
    const int tile = unit / p.tiles_t;
    if (RB == 2 && p.gu_inter) return tile * 128 + (rb ? p.gu_inter : 0);
    return (tile * RB + rb) * 128;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < kMidBars; ++i) { mbar_init(smem_u32(a_full + i), i % RB == 0 ? 5 : 4); mbar_init(smem_u32(a_empty + i), 1); }
    for (int i = 0; i < kMidMaxCodes; ++i) { mbar_init(smem_u32(c_full + i), 1); mbar_init(smem_u32(c_empty + i), 4); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(acc_full + i), 1); mbar_init(smem_u32(acc_empty + i), 4); }
    mbar_init(smem_u32(l_full), 4);
    mbar_init(smem_u32(l_empty), 1);
    mbar_init(smem_u32(xch_full), cl > 1 ? (cl - 1) * 4 : 1);
    mbar_init(smem_u32(xch_free), cl > 1 ? cl - 1 : 1);
    mbar_init(smem_u32(drain), 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (threadIdx.x < 16) {
    constexpr float lv[16] = {NF4LL_LEVELS};
    float v = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) v = (static_cast<int>(threadIdx.x) == j) ? lv[j] : v;
    sLv[threadIdx.x] = v;
  }
  __syncthreads();                             // barriers and levels are there
  if (cl > 1) cluster_arrive_together();
  // the two producers go on at once; the others lay out the tables first. Nothing before pdl_wait() reads global memory.
  if (warp != 0 && warp != 2) {
    if (warp == 1) {
      tmem_alloc(smem_u32(tmem_slot), 512);
      tmem_relinquish();
    }
    for (int idx = MODE == kBwd ? 256 * 8 : warp == 1 ? lane : threadIdx.x - 64; idx < 256 * 8; idx += kMidThreads - 64) {      // two of an entry's sixteen copies per store
      const int v = idx >> 3;
      const uint32_t e0 = __float_as_uint(sLv[v >> 4]), e1 = __float_as_uint(sLv[v & 15]);
      sts128(sLut + idx * 16, make_uint4(e0, e1, e0, e1));
    }
    if (!p.early) pdl_wait();
    if (threadIdx.x >= kMidThreads - 256) sCode2[threadIdx.x - (kMidThreads - 256)] = p.code2[threadIdx.x - (kMidThreads - 256)];
    tc_fence_before();
    named_barrier(3, kMidThreads - 64);
    tc_fence_after();
  } else if (!p.early) {
    pdl_wait();
  }
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t d_cols = RB * p.nt;           // columns of one accumulator
  // tensor memory: nbuf accumulators | backward with a mask: the rank-16 product | forward: decoded weights
  const uint32_t l_col = p.nbuf * d_cols;
  const uint32_t a_col = 512 - p.na * 64;

  if (warp == 0) {
    // ----------------------------------------------------------------------------- codes
    if (lane == 0) {
      tma_prefetch_desc(&tmap_nib);
      int i = 0;
      bool ok = true;
      for (int u = cluster; ok && u < p.units; u += n_clusters)
        for (int g = grp0; ok && g < grp1; ++g)
#pragma unroll
          for (int rb = 0; rb < (MODE == kFwd ? RB : 1); ++rb, ++i) {
            if (p.withhold == kHoldCodes && i == 1) { ok = false; break; }
            const int c = i & (p.nc - 1);
            if (!wait_or_abort(smem_u32(c_empty + c), ((i >> p.nc_log) & 1) ^ 1, ab, 0x0701)) { ok = false; break; }
            mbar_arrive_expect_tx(smem_u32(c_full + c), kStage);
            const int r0 = row0_of(u, rb);
            if (MODE == kFwd) tma_load_2d(sCode + c * kStage, &tmap_nib, g * 128, r0, smem_u32(c_full + c));
            else tma_load_2d(sCode + c * kStage, &tmap_nib, r0 / 2, g * 128, smem_u32(c_full + c));
          }
      if (*abort_flag)        // copies still in flight get a bounded chance to land before the CTA goes away
        for (int k = (i > p.nc ? i - p.nc : 0); k < i; ++k) mid_drain(smem_u32(c_full + (k & (p.nc - 1))), (k >> p.nc_log) & 1);
    }
  } else if (warp == 2) {
    // ----------------------------------------------------------------------------- token tiles
    if (lane == 0) {
      tma_prefetch_desc(&tmap_x);
      // a slot holds the two token tiles of an item and of the next row block's; it is free when the last of the items that
      // used it has been multiplied. Item i = hg * RB; barriers go round with the items.
      int hi = 0;                                  // running count of slots filled
      bool ok = true;
      for (int u = cluster; ok && u < p.units; u += n_clusters) {
        const int t0 = (u % p.tiles_t) * p.nt;
        for (int hg = grp0 * kHalves; hg < grp1 * kHalves; ++hg, ++hi) {
          const int i = hi * RB;
          if (hi >= p.nx) {
            const int e = (hi - p.nx) * RB + RB - 1;
            if (!wait_or_abort(smem_u32(a_empty + e % kMidBars), (e / kMidBars) & 1, ab, 0x0702)) { ok = false; break; }
          }
          const int nb = max(0, min(2, p.steps - hg * 2));
          const uint32_t bar = smem_u32(a_full + i % kMidBars), dst = sX + (hi & (p.nx - 1)) * p.nt * 256;
          mbar_arrive_expect_tx(bar, nb * p.nt * 128);
          for (int k = 0; k < nb; ++k) tma_load_2d(dst + k * p.nt * 128, &tmap_x, (hg * 2 + k) * 64, t0, bar);
        }
      }
      if (*abort_flag)        // copies still in flight get a bounded chance to land
        for (int k = (hi > p.nx ? hi - p.nx : 0); k < hi; ++k) mid_drain(smem_u32(a_full + k * RB % kMidBars), (k * RB / kMidBars) & 1);
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------------------------- MMA issue: the whole warp walks the loop, one elected
    // lane issues (operands stay in uniform registers: 38 clocks per MMA of 64 columns against 66 from a lane picked by a branch)
    const uint32_t idesc = (1u << 4) | (MODE == kBwd ? 1u << 15 : 0u) | (static_cast<uint32_t>(p.nt >> 3) << 17) | (8u << 24);
    const uint64_t xdesc0 = make_smem_desc(sX, 16, 1024, kSwizzle128B);
    const uint64_t adesc0 = make_smem_desc(sA, 16384, 1024, kSwizzle128B);
    const uint32_t nt = p.nt, a_tm = tmem_base + a_col;
    bool ok = true;
    int i = 0, ul = 0, slot = 0;
    for (int u = cluster; ok && u < p.units; u += n_clusters, ++ul) {
      const int buf = p.nbuf == 2 ? ul & 1 : 0;
      if (!mid_wait(smem_u32(acc_empty + buf), ((p.nbuf == 2 ? ul >> 1 : ul) & 1) ^ 1, ab, 0x0703)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d0 = tmem_base + buf * d_cols;
      uint32_t more = 0;                           // the unit's first MMA on an accumulator overwrites it
      for (int hg = grp0 * kHalves; ok && hg < grp1 * kHalves; ++hg) {
        const int nb = p.steps - hg * 2;
        const uint64_t xdesc = xdesc0 + (((i / RB) & (p.nx - 1)) * nt * 16);
#pragma unroll
        for (int rb = 0; rb < RB; ++rb, ++i) {
          if (!mid_wait(smem_u32(a_full + i % kMidBars), (i / kMidBars) & 1, ab, 0x0705)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = d0 + rb * nt, a = a_tm + slot * 64;
          const uint64_t adesc = adesc0 + slot * 2048;
          if (++slot == p.na) slot = 0;
          if (mid_elect()) {
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              if (s < nb) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                  const uint32_t acc = s == 0 && kk == 0 ? more : 1u;
                  if (MODE == kFwd) mid_mma_ts(d, a + s * 32 + kk * 8, xdesc + s * nt * 8 + kk * 2, idesc, acc);
                  else tc_mma_f16(d, adesc + (s * 4 + kk) * 128, xdesc + s * nt * 8 + kk * 2, idesc, acc);
                }
              }
            }
            tc_commit(smem_u32(a_empty + i % kMidBars));
          }
          __syncwarp();
        }
        more = 1;
      }
      if (ok && p.any_lora && crank == 0) {
        // the rank-16 branches: left to the end, so that their operands may still be on their way until then
        if (!mid_wait(smem_u32(l_full), ul & 1, ab, 0x0706)) { ok = false; break; }
        tc_fence_after();
        if (mid_elect()) {
#pragma unroll
          for (int rb = 0; rb < RB; ++rb) {
            const uint64_t wdesc = make_smem_desc(sL + rb * 4096, 128, 256, kSwizzleNone);
            const uint64_t tdesc = make_smem_desc(sL + RB * 4096 + rb * p.nt * 32, 128, 256, kSwizzleNone);
            if (MODE == kBwd && p.mask) tc_mma_f16(tmem_base + l_col + rb * p.nt, wdesc, tdesc, idesc, 0u);
            else tc_mma_f16(d0 + rb * p.nt, wdesc, tdesc, idesc, 1u);
            if (MODE == kFwd && p.split)
              tc_mma_f16(d0 + rb * p.nt, wdesc, make_smem_desc(sCode + p.off_turn + rb * 256, 128, kMidTurnBytes / 2, kSwizzleNone), idesc, 1u);
          }
          tc_commit(smem_u32(l_empty));
        }
        __syncwarp();
      }
      if (mid_elect()) tc_commit(smem_u32(acc_full + buf));
      __syncwarp();
    }
  }
  bool ok = true;
  if (warp >= kMidDecodeWarp) {
    // ----------------------------------------------------------------------------- decode
    // A team takes a whole stage of codes, two items (backward with one row block: one); a thread has one row of it, a pair of
    // quantisation blocks per item. The pairs' absmax codes and scales are fetched a stage ahead.
    const int team = (warp - kMidDecodeWarp) >> 2, q = warp & 3, r = q * 32 + lane;
    const uint32_t lut = sLut + (lane & 15) * 8;
    const uint32_t tA = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + a_col;
    const int last_block = p.N * bpr - 1;
    constexpr int kStagesPerGroup = MODE == kFwd ? RB : 1;
    const int n_pos = (grp1 - grp0) * kStagesPerGroup;
    struct Pairs { uint32_t q0, q1; float s0, o0, s1, o1; };
    // first block of pair h of stage `pos` of unit `u`
    auto block_of = [&](int u, int pos, int h) {
      const int g = grp0 + pos / kStagesPerGroup;
      if (MODE == kFwd) return min(row0_of(u, pos % kStagesPerGroup) + r, p.N - 1) * bpr + g * 4 + 2 * h;
      return min(g * 128 + r, p.N - 1) * bpr + (row0_of(u, 0) >> 6) + 2 * h;
    };
    auto load_pairs = [&](int u, int pos, Pairs& a) {
      const int b0 = block_of(u, pos, 0);
      if (p.qabs_mode == 4 && kPer == 2) {
        a.q0 = __ldg(reinterpret_cast<const uint32_t*>(p.qabs + min(b0, last_block - 3)));
        a.s0 = __ldg(p.scale2 + (b0 >> 8)); a.o0 = __ldg(p.offset2 + (b0 >> 8));
      } else if (p.qabs_mode >= 2) {
        const int c0 = min(b0, last_block - 1), c1 = min(b0 + 2, last_block - 1);
        a.q0 = __ldg(reinterpret_cast<const uint16_t*>(p.qabs + c0));
        if (kPer == 1) { a.s0 = __ldg(p.scale2 + (c0 >> 8)); a.o0 = __ldg(p.offset2 + (c0 >> 8)); return; }
        a.q1 = __ldg(reinterpret_cast<const uint16_t*>(p.qabs + c1));
        a.s0 = __ldg(p.scale2 + (c0 >> 8)); a.o0 = __ldg(p.offset2 + (c0 >> 8));
        a.s1 = __ldg(p.scale2 + (c1 >> 8)); a.o1 = __ldg(p.offset2 + (c1 >> 8));
      }
    };
    auto absmax = [&](int b) {                   // blocks that do not come in aligned pairs: fetched when needed
      b = min(b, last_block);
      return block_absmax(sCode2[__ldg(p.qabs + b)], __ldg(p.scale2 + (b >> 8)), __ldg(p.offset2 + (b >> 8)));
    };
    int u = cluster, pos = team;
    while (pos >= n_pos && u < p.units) { pos -= n_pos; u += n_clusters; }
    Pairs cur{};
    if (u < p.units) load_pairs(u, pos, cur);
    int slot0 = kStagesPerGroup == 2 ? (team >> 1) * 4 + (team & 1) : team * kPer;       // slot of the stage's first item
    while (slot0 >= p.na) slot0 -= p.na;
    for (int si = team; ok && u < p.units; si += kMidTeams) {
      const int g = grp0 + pos / kStagesPerGroup;
      int un = u, pn = pos + kMidTeams;
      while (pn >= n_pos && un < p.units) { pn -= n_pos; un += n_clusters; }
      Pairs nxt{};
      if (un < p.units) load_pairs(un, pn, nxt);
      const int cs = si & (p.nc - 1);
      if (!mid_wait(smem_u32(c_full + cs), (si >> p.nc_log) & 1, ab, 0x0707)) { ok = false; break; }
      const uint32_t code = sCode + cs * kStage;
#pragma unroll
      for (int h = 0; h < kPer; ++h) {
        // the item: its place in the order in which they are multiplied, its steps, its slot
        const int i = kStagesPerGroup == 2 ? (si >> 1) * 4 + h * 2 + (si & 1) : si * kPer + h;
        const int nb = min(2, p.steps - (MODE == kBwd ? g * 2 : g * 4 + h * 2));
        int slot = slot0 + h * kStagesPerGroup;
        while (slot >= p.na) slot -= p.na;
        uint4 c[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (kPer == 1) c[k] = lds128(code + r * 64 + ((k ^ ((r >> 1) & 3)) << 4));                        // 128 rows of 64 bytes
          else c[k] = lds128(code + r * 128 + (((h * 4 + k) ^ (r & 7)) << 4));                              // 128 rows of 128 bytes
        }
        float am0, am1;
        if (p.qabs_mode >= 2) {
          const bool quad = p.qabs_mode == 4 && kPer == 2;
          const uint32_t w = quad ? cur.q0 >> (16 * h) : h ? cur.q1 : cur.q0;
          const float s2 = quad || h == 0 ? cur.s0 : cur.s1, o2 = quad || h == 0 ? cur.o0 : cur.o1;
          am0 = block_absmax(sCode2[w & 0xffu], s2, o2);
          am1 = block_absmax(sCode2[(w >> 8) & 0xffu], s2, o2);
        } else {
          const int b = block_of(u, pos, h);
          am0 = absmax(b); am1 = absmax(b + 1);
        }
        if (i >= p.na) {                           // the slot's former weights: item i - na
          const int e = i - p.na;
          if (!mid_wait(smem_u32(a_empty + e % kMidBars), (e / kMidBars) & 1, ab, 0x0708)) { ok = false; break; }
        }
        if (MODE == kFwd) {
          tc_fence_after();
          const uint64_t m0 = mid_twice(am0), m1 = mid_twice(am1);
          const uint32_t dst = tA + slot * 64;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (k < nb * 2) {
              const uint64_t m = k < 2 ? m0 : m1;
              const uint4 o0 = mid_decode8(c[k].x, lut, m), o1 = mid_decode8(c[k].y, lut, m), o2 = mid_decode8(c[k].z, lut, m),
                          o3 = mid_decode8(c[k].w, lut, m);
              const uint32_t v[16] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w, o2.x, o2.y, o2.z, o2.w, o3.x, o3.y, o3.z, o3.w};
              mid_tmem_st16(dst + k * 16, v);
            }
          }
          tmem_st_wait();
          tc_fence_before();
        } else {
          if (r < nb * 64) {
            // columns 0-63 and 64-127 of the item in tiles of 128 rows x 128 bytes; byte planes instead of the table, whose
            // reads would compete with the stores and the tensor core's reads for shared memory (measured: 17.5 us with the
            // planes, 18.9 with the table, 8960 x 1536 at 187 rows)
            const uint32_t dst = sA + slot * 32768 + r * 128;
            dequant_block_to_smem(dst, r & 7, c[0], c[1], am0);
            dequant_block_to_smem(dst + 16384, r & 7, c[2], c[3], am1);
          }
          fence_proxy_async_smem();
        }
        __syncwarp();
        // the codes go back only when they have been used: an arrival right behind the loads let the next copy overtake them
        if (lane == 0) {
          mbar_arrive(smem_u32(a_full + i % kMidBars));
          if (h == kPer - 1) mbar_arrive(smem_u32(c_empty + cs));
        }
      }
      slot0 += kMidTeams * kPer;                   // four stages on
      while (slot0 >= p.na) slot0 -= p.na;
      cur = nxt; u = un; pos = pn;
    }
  }
  if (warp >= kMidEpiWarp) {
    // ----------------------------------------------------------------------------- rank-16 operands, epilogue
    // Four warps of their own finish a unit while the next one is decoded; the decoding warps help with the last one. A crew
    // is four warps, one per lane quarter of tensor memory.
    if (p.early) pdl_wait();                     // the rank-16 products come from the kernel before this one
    if (cl > 1) cluster_wait_together();
    const int crew = (warp - kMidEpiWarp) >> 2;
    const int q = warp & 3, r = q * 32 + lane, tid = threadIdx.x - kMidEpiWarp * 32;
    const int last = (p.units - 1 - cluster) / n_clusters;                 // the cluster's last unit, counted from 0
    auto peers = [&](uint64_t* bar) {            // one arrival at every other CTA of the cluster
      if (lane < cl && lane != crank) mbar_arrive_remote(map_to_cta(smem_u32(bar), lane));
    };
    // each warp's scratch; the helping warps' is in the token tiles, which nobody reads any more by then
    const uint32_t turned = crew == 0 ? sCode + p.off_turn + (warp - kMidEpiWarp) * kMidTurnBytes
                                      : sCode + p.off_lora - (warp - kMidDecodeWarp + 1) * kMidTurnBytes;
    if (cl > 1 && !p.x_alias && warp == kMidEpiWarp) peers(xch_free);
    for (int ul = crew ? last : 0; ul <= last; ++ul) {
      const int u = cluster + ul * n_clusters, crews = ul == last ? 1 + kMidTeams : 1;
      const int t0 = (u % p.tiles_t) * p.nt, vt = min(p.nt, p.M - t0);
      if (p.any_lora && crank == 0 && crew == 0 && ok) {
        ok = mid_wait(smem_u32(l_empty), (ul & 1) ^ 1, ab, 0x0709);
        if (ok) {
#pragma unroll
          for (int rb = 0; rb < RB; ++rb) {
            const int r0 = row0_of(u, rb);
            int sg = 0;
            if (MODE == kFwd) while (sg + 1 < p.n_seg && r0 >= p.seg_end[sg]) ++sg;
            const float* left = p.seg_left[sg];
            const __half* right = p.seg_right[sg];
            const float sc = p.seg_scale[sg];
            // weights' side: chunk (row, half of the rank) -> (row / 8) * 256 + half * 128 + (row % 8) * 16
            for (int c = tid; c < 256; c += 128) {
              uint4 v = make_uint4(0, 0, 0, 0);
              uint32_t at;
              if (MODE == kFwd) {
                const int row = c >> 1, h = c & 1;
                if (left && r0 + row < p.seg_end[sg]) v = __ldg(reinterpret_cast<const uint4*>(right + static_cast<int64_t>(r0 + row) * 16 + h * 8));
                at = (row >> 3) * 256 + h * 128 + (row & 7) * 16;
              } else {
                const int j = c >> 4, c8 = c & 15;
                if (left && r0 + c8 * 8 < p.NO) v = __ldg(reinterpret_cast<const uint4*>(right + static_cast<int64_t>(j) * p.K + r0 + c8 * 8));
                at = c8 * 256 + (j >> 3) * 128 + (j & 7) * 16;
              }
              sts128(sL + rb * 4096 + at, v);
            }
            // tokens' side, scaled and rounded to fp16; or in two parts, fp16 each, a token with values beyond fp16's range
            // left out here, its bit set, and added in fp32 by the epilogue
            auto side = [&](int row, int h, float (&v)[8]) {
              const float4* src = reinterpret_cast<const float4*>(left + static_cast<int64_t>(t0 + row) * 16 + h * 8);
              const bool there = left && row < vt;
              const float4 a = there ? __ldcg(src) : make_float4(0.f, 0.f, 0.f, 0.f), b = there ? __ldcg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
              v[0] = a.x * sc; v[1] = a.y * sc; v[2] = a.z * sc; v[3] = a.w * sc;      // the kernel before this one wrote them
              v[4] = b.x * sc; v[5] = b.y * sc; v[6] = b.z * sc; v[7] = b.w * sc;
            };
            const uint32_t sT = sL + RB * 4096 + rb * p.nt * 32;
            if (MODE == kFwd && p.split) {
              const int row = tid >> 1, h = tid & 1;               // 64 tokens at most; two lanes hold the halves of a token's rank
              float v[8], r[8];
              side(row, h, v);
              uint4 hi = pack8(v);
              auto off = [](uint32_t w) { return ((w & 0x7c007c00u) + 0x04000400u) & 0x80008000u; };      // an infinity or NaN of the two
              const uint32_t out = __ballot_sync(0xffffffffu, (off(hi.x) | off(hi.y) | off(hi.z) | off(hi.w)) != 0);
              const uint32_t pair = (out | (out >> 1)) & 0x55555555u;
              if (lane == 0) wide[((ul & 1) * RB + rb) * 4 + q] = pair;
              unpack8(hi, r);
#pragma unroll
              for (int j = 0; j < 8; ++j) r[j] = v[j] - r[j];
              uint4 lo = pack8(r);
              if ((pair >> (lane & 30)) & 1) hi = lo = make_uint4(0, 0, 0, 0);
              // the low parts lie in the warps' scratch (this warp's sixteen tokens in its own), idle until the unit's epilogue
              sts128(sCode + p.off_turn + (row >> 3) * (kMidTurnBytes / 2) + rb * 256 + h * 128 + (row & 7) * 16, lo);
              if (row < p.nt) sts128(sT + (row >> 3) * 256 + h * 128 + (row & 7) * 16, hi);
            } else {
              for (int c = tid; c < 2 * p.nt; c += 128) {
                const int row = c >> 1, h = c & 1;
                float v[8];
                side(row, h, v);
                sts128(sT + (row >> 3) * 256 + h * 128 + (row & 7) * 16, pack8(v));
              }
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && p.withhold != kHoldRank16) mbar_arrive(smem_u32(l_full));
        }
      }
      const int buf = p.nbuf == 2 ? ul & 1 : 0;
      const bool split = MODE == kFwd && p.split && p.any_lora && crank == 0 && crew == 0;
      if (split && ok) ok = mid_wait(smem_u32(l_full), ul & 1, ab, 0x070d);      // the other warps' bits are there
      if (crew == 0 && ok) ok = mid_wait(smem_u32(acc_full + buf), (p.nbuf == 2 ? ul >> 1 : ul) & 1, ab, 0x070a);
      if (split && ok) {
        // rank-16 terms of tokens beyond fp16's range: added to their columns of the accumulator in fp32
        uint32_t any = 0;
#pragma unroll
        for (int rb = 0; rb < RB; ++rb) {
          const uint4 w = lds128(smem_u32(wide + ((ul & 1) * RB + rb) * 4));
          any |= w.x | w.y | w.z | w.w;
        }
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; any && i < RB * 4; ++i) {
          const int rb = i >> 2, tg = (i & 3) * 16;
          uint32_t bits = wide[(ul & 1) * RB * 4 + i];
          const int n = row0_of(u, rb) + r;
          int sg = 0;
          while (sg + 1 < p.n_seg && n - r >= p.seg_end[sg]) ++sg;
          for (; bits; bits &= bits - 1) {
            const int t = tg + ((__ffs(bits) - 1) >> 1);
            const uint32_t at = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * d_cols + rb * p.nt + t;
            const float* left = p.seg_left[sg] + static_cast<int64_t>(t0 + t) * 16;
            float l = 0.f;
            if (n < p.seg_end[sg])
              for (int k = 0; k < 16; ++k) l = fmaf(__ldcg(left + k), __half2float(p.seg_right[sg][static_cast<int64_t>(n) * 16 + k]) * p.seg_scale[sg], l);
            __syncwarp();
            mid_tmem_add(at, l);
          }
        }
        tc_fence_before();
      }
      if (crews > 1) {
        // the decoding warps have met none of the earlier phases of the barriers below: they go on behind the first crew
        named_barrier(2, 128 * (1 + kMidTeams));
        if (*abort_flag) ok = false;
      }
      tc_fence_after();
      const uint32_t tD = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * d_cols;
      const uint32_t tL = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + l_col;
      const bool masked = MODE == kBwd && p.mask && p.any_lora;
      float bias[RB];
      int row[RB];
      bool row_ok[RB];
#pragma unroll
      for (int rb = 0; rb < RB; ++rb) {
        const int r0 = row0_of(u, rb);
        row[rb] = r0 + r;
        row_ok[rb] = (RB == 2 && p.gu_inter) ? row[0] < p.gu_inter : row[rb] < p.NO;
        bias[rb] = MODE == kFwd && p.bias && row_ok[rb] ? __half2float(p.bias[row[rb]]) : 0.f;
      }
      // eight tokens of the warp's 32 columns from `col` on: turned round in shared memory, rounded once, 16 bytes per store
      auto put = [&](const float (&f)[8], __half* base, int64_t ld, int col, int end, int t) {
#pragma unroll
        for (int j = 0; j < 8; ++j) asm volatile("st.shared.f32 [%0], %1;" ::"r"(turned + j * kMidTurnRow + lane * 4), "f"(f[j]) : "memory");
        __syncwarp();
        const int token = lane >> 2, part = lane & 3;
        const uint4 a = lds128(turned + token * kMidTurnRow + part * 32), b = lds128(turned + token * kMidTurnRow + part * 32 + 16);
        if (t + token < vt && col + part * 8 < end) {
          float v[8] = {__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(a.w),
                        __uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z), __uint_as_float(b.w)};
          uint4* dst = reinterpret_cast<uint4*>(base + static_cast<int64_t>(t0 + t + token) * ld + col + part * 8);
          if (MODE == kBwd && p.accumulate) {
            float old[8];
            unpack8(*dst, old);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] += old[j];
          }
          *dst = pack8(v);
        }
        __syncwarp();
      };
      // the rank-16 product under the keep-mask (rank 0 of the cluster has it), added to eight token columns
      auto add_masked = [&](int rb, int t, float (&f)[8]) {
        float l[8];
        __syncwarp();
        mid_tmem_ld8(tL + rb * p.nt + t, l);
        if (row_ok[rb]) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (t + j < vt && __ldg(p.mask + static_cast<int64_t>(t0 + t + j) * p.ld_mask + row[rb])) f[j] = fmaf(l[j], p.keep_scale, f[j]);
        }
      };
      int tb = 0, te = vt;                       // token columns this CTA finishes
      if (cl > 1) {
        // partial sums to the CTAs that finish them, [source][row block][column / 4][row][4] fp32
        tb = min(crank * p.ts, vt); te = min(tb + p.ts, vt);
        int turn = 0;                            // chunks of eight columns go round the crews
        if (p.x_alias && warp == kMidEpiWarp && ok) peers(xch_free);       // this CTA's operand rings are idle
        if (ok) ok = mid_wait<true>(smem_u32(xch_free), ul & 1, ab, 0x070b);
        if (ok) {
          for (int k = 1; k < cl; ++k) {
            int dst = crank + k;                 // peers in turn, so that not all write to the same one
            if (dst >= cl) dst -= cl;
            const int slot = crank < dst ? crank : crank - 1;
            const uint32_t base = map_to_cta(sXch, dst) + (static_cast<uint32_t>(slot * RB * (p.ts >> 2)) * 128 + r) * 16;
            const int b = min(dst * p.ts, vt), e = min(b + p.ts, vt);
#pragma unroll
            for (int rb = 0; rb < RB; ++rb)
              for (int t = b; t < e; t += 8) {
                const bool mine = turn == crew;
                if (++turn == crews) turn = 0;
                if (!mine) continue;
                float f[8];
                __syncwarp();
                mid_tmem_ld8(tD + rb * p.nt + t, f);
                if (masked && crank == 0) add_masked(rb, t, f);
                const uint32_t at = base + static_cast<uint32_t>(rb * (p.ts >> 2) + ((t - b) >> 2)) * 2048;
                mid_st_cluster(at, f[0], f[1], f[2], f[3]);
                mid_st_cluster(at + 2048, f[4], f[5], f[6], f[7]);
              }
          }
          asm volatile("fence.acq_rel.cluster;" ::: "memory");
        }
        if (crews > 1) named_barrier(2, 128 * (1 + kMidTeams));
        if (ok) {
          __syncwarp();
          if (crew == 0 && !(p.withhold == kHoldSums && crank == cl - 1)) peers(xch_full);
          ok = mid_wait<true>(smem_u32(xch_full), ul & 1, ab, 0x070c);
        }
      }
      if (ok) {
        for (int t = tb + crew * 8; t < te; t += crews * 8) {
          float f[RB][8];
#pragma unroll
          for (int rb = 0; rb < RB; ++rb) {
            __syncwarp();
            float own[8];
            mid_tmem_ld8(tD + rb * p.nt + t, own);
            if (masked && crank == 0) add_masked(rb, t, own);
            if (cl == 1) {
#pragma unroll
              for (int j = 0; j < 8; ++j) f[rb][j] = own[j];
            } else {
              // the slices in ascending order: a fixed order
#pragma unroll
              for (int j = 0; j < 8; ++j) f[rb][j] = 0.f;
              for (int s = 0; s < cl; ++s) {
                float v[8];
                if (s == crank) {
#pragma unroll
                  for (int j = 0; j < 8; ++j) v[j] = own[j];
                } else {
                  const int slot = s < crank ? s : s - 1;
                  const uint32_t at = sXch + (static_cast<uint32_t>((slot * RB + rb) * (p.ts >> 2) + ((t - tb) >> 2)) * 128 + r) * 16;
                  const uint4 a = lds128(at), b = lds128(at + 2048);
                  v[0] = __uint_as_float(a.x); v[1] = __uint_as_float(a.y); v[2] = __uint_as_float(a.z); v[3] = __uint_as_float(a.w);
                  v[4] = __uint_as_float(b.x); v[5] = __uint_as_float(b.y); v[6] = __uint_as_float(b.z); v[7] = __uint_as_float(b.w);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) f[rb][j] += v[j];
              }
            }
          }
          if (RB == 2 && p.gu_inter) {
            float h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {          // the product of the rounded values, as the stand-alone kernel would read them
              f[0][j] = __half2float(__float2half_rn(f[0][j]));
              f[RB - 1][j] = __half2float(__float2half_rn(f[RB - 1][j]));
              h[j] = f[0][j] * fast_sigmoid(f[0][j]) * f[RB - 1][j];
            }
            put(f[0], p.out, p.ldo, row[0] - lane, p.gu_inter, t);
            put(f[RB - 1], p.out_u, p.ldu, row[0] - lane, p.gu_inter, t);
            put(h, p.out_h, p.ldh, row[0] - lane, p.gu_inter, t);
          } else {
#pragma unroll
            for (int rb = 0; rb < RB; ++rb) {
              if (MODE == kFwd) {
#pragma unroll
                for (int j = 0; j < 8; ++j) f[rb][j] += bias[rb];
              }
              put(f[rb], p.out, p.ldo, row[rb] - lane, p.NO, t);
            }
          }
        }
      }
      // the accumulator may be overwritten
      tc_fence_before();
      __syncwarp();
      if (lane == 0 && crew == 0) mbar_arrive(smem_u32(acc_empty + buf));
      if (cl > 1 && ul < last) {
        named_barrier(1, 128);                   // all four warps have read the partial sums
        if (warp == kMidEpiWarp && ok) peers(xch_free);
      }
    }
  }

  // ------------------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncwarp();
  if (cl > 1 && warp < kMidEpiWarp) cluster_wait_together();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (*abort_flag) {                         // none of this warp's MMAs may still be running when tensor memory is freed
      if (mid_elect()) tc_commit(smem_u32(drain));
      __syncwarp();
      mid_drain(smem_u32(drain), 0);
      __syncwarp();
    }
    tmem_dealloc(tmem_base, 512);
  }
  if (cl > 1) cluster_sync_all();                // nobody leaves while a peer may still write to its shared memory
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
static int mid_encode(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t inner, uint64_t outer, uint64_t stride_bytes,
                      uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swizzle, const char* what) {
  EncodeTiledFn encode = nullptr;
  if (int rc = get_encode_fn(&encode)) return rc;
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {stride_bytes};
  const cuuint32_t box[2] = {box_inner, box_outer};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_detail("cuTensorMapEncodeTiled (%s) failed with CUresult %d", what, static_cast<int>(r));
    return NF4LL_ERR_CUDA;
  }
  return NF4LL_OK;
}

// How many clusters of `cl` CTAs the current device holds at once (148, 74, 45, 33, 26, 22, 15, 15 for 1 to 8 on the B200s at hand)
int mid_clusters(int cl) {
  constexpr int kDevices = 64;
  static int known[kDevices][9];               // 0: not asked yet; written with the same value by any thread
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
  int n = __atomic_load_n(&known[dev][cl], __ATOMIC_RELAXED);
  if (n > 0) return n;
  auto kernel = nf4_mid_kernel<kFwd, 1>;       // one CTA per SM in every variant
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMidSmem) != cudaSuccess) return 0;
  if (cl == 1) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 0;
  } else {
    PdlLaunch probe(dim3(cl), dim3(kMidThreads), kMidSmem, nullptr, cl, 1, false, false);
    probe.cfg.numAttrs = 1;                    // the cluster dimension only
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &probe.cfg) != cudaSuccess) n = 0;
  }
  if (n > 0) __atomic_store_n(&known[dev][cl], n, __ATOMIC_RELAXED);
  else (void)cudaGetLastError();
  return n;
}

struct MidLayout {
  int off_a, off_x, off_lora, off_xch, off_lut, off_turn, off_misc, total;
};
static MidLayout mid_layout(int mode, const MidPlan& p, bool lora) {
  MidLayout l{};
  int at = p.nc * (mode == kBwd && p.rb == 1 ? kMidCodeBytes / 2 : kMidCodeBytes);
  l.off_a = at;
  if (mode == kBwd) at += p.na * 32768;
  l.off_x = at;
  at += p.nx * p.nt * 256;
  const int ring = at;
  l.off_lora = at;
  if (lora) at += p.rb * (4096 + p.nt * 32);
  const int ts = (p.nt / 8 + p.cl - 1) / p.cl * 8;
  const int xch = p.cl > 1 ? (p.cl - 1) * p.rb * ts * 512 : 0;
  l.off_xch = p.x_alias ? 0 : at;
  if (!p.x_alias) at += xch;
  l.off_lut = at;
  if (mode == kFwd) at += kMidLutBytes;
  l.off_turn = at;
  at += 4 * kMidTurnBytes;
  l.off_misc = at;
  at += 1024 + 64 + 8 * (2 * kMidBars + 2 * kMidMaxCodes + 16) + 16 + 2 * 2 * 4 * 4;
  l.total = at + 1024;                          // the base is rounded up to 1024
  if (p.x_alias && xch + 4 * kMidTeams * kMidTurnBytes > ring) l.total = kMidSmem + 1;
  return l;
}

// Fills in the buffers of a plan whose rb, nt, cl, units and clusters are set; false: it does not fit.
static bool mid_buffers(int mode, bool mask, bool lora, MidPlan* p) {
  const int d = p->rb * p->nt;
  const bool many = p->units > p->clusters;
  const int extra = mode == kBwd && mask ? d : 0;
  for (int nbuf = many ? 2 : 1; nbuf >= 1; --nbuf) {
    const int room = 512 - nbuf * d - extra;
    if (room < 0) continue;
    p->nbuf = nbuf;
    p->x_alias = false;
    const int na_max = mode == kBwd ? 4 : room / 64 < 7 ? room / 64 : 7;
    if (na_max < (nbuf == 2 ? 4 : 2)) continue;
    static const int kDepth[][2] = {{8, 4}, {4, 4}, {8, 2}, {4, 2}};      // stages of codes, slots of token tiles
    for (int na = na_max; na >= (mode == kFwd ? na_max : 2); --na)
      for (const auto& d2 : kDepth)
        for (int alias = 0; alias <= (p->cl > 1 && !many ? 1 : 0); ++alias) {
          p->x_alias = alias != 0;
          p->nc = d2[0]; p->na = na; p->nx = d2[1];
          if (mid_layout(mode, *p, lora).total <= kMidSmem) return true;
        }
  }
  return false;
}

// Time of a plan in us, behind other calls: a fixed cost, a cost per item of the busiest CTA (the decode's, or that of feeding
// and multiplying nt tokens), the exchange and the epilogue. Fitted to 5116 plans of nine weights from 1536 x 1536 to
// 27648 x 5120 at 17 to 951 rows; picking by it takes 0.7 % longer than the fastest plans, 12 % at worst.
static double mid_us(int mode, int rb, int nt, int cl, int64_t rounds, int64_t items, int nbuf) {
  static const double kFit[2][2][8] = {{{5.0, 0, 0.459, 0.137, 0.0031, 0.46, 0.0048, 0.0279}, {2.1, 1.31, 0.463, 0.087, 0.003, 2.1, 0.0098, 0.0216}},
                                       {{4.32, 0, 0.604, 0.459, 0.0013, 1.73, 0, 0.0266}, {5.88, 0.39, 0.0968, 0.627, 0.0007, 0, 0, 0.0204}}};
  const double* f = kFit[mode == kBwd ? 1 : 0][rb - 1];
  const double fed = f[3] + f[4] * nt, item = fed > f[2] ? fed : f[2];
  const double epilogue = f[5] + f[6] * nt * rb / cl;
  return f[0] + (cl > 1 ? f[1] + f[7] * nt * rb * static_cast<double>(rounds) : 0) + static_cast<double>(rounds * items) * item +
         epilogue * static_cast<double>(nbuf == 1 ? rounds : 1);
}

static bool mid_search(int mode, int64_t M, int64_t NO, int64_t KC, bool mask, int64_t gu_inter, bool lora, int f_rb, int f_nt, int f_cl, MidPlan* plan) {
  const int64_t steps = KC / 64, halves = mode == kBwd ? 1 : 2, groups = (steps + 2 * halves - 1) / (2 * halves);
  const int64_t blocks = gu_inter ? (gu_inter + 127) / 128 * 2 : (NO + 127) / 128;
  bool found = false;
  for (int rb = gu_inter ? 2 : 1; rb <= 2; ++rb) {
    if (f_rb && rb != f_rb) continue;
    const int64_t tiles_o = (blocks + rb - 1) / rb;
    for (int64_t tiles_t = 1; tiles_t <= 16; ++tiles_t) {
      int nt = static_cast<int>(((M + tiles_t - 1) / tiles_t + 15) / 16 * 16);
      if (f_nt) nt = f_nt;
      else if (nt > 256 || (tiles_t > 1 && nt < 48)) continue;
      const int64_t tt = (M + nt - 1) / nt, units = tiles_o * tt;
      if ((f_nt && tiles_t > 1) || units > (1 << 24)) continue;
      for (int cl = 1; cl <= 8 && cl <= groups; ++cl) {
        if (f_cl && cl != f_cl) continue;
        const int most = mid_clusters(cl);
        if (most <= 0) continue;
        MidPlan p{};
        p.rb = rb; p.nt = nt; p.cl = cl;
        p.split = mode == kFwd && M <= kMidSplitRows && nt <= kMidSplitRows;
        p.tiles_o = static_cast<int>(tiles_o); p.tiles_t = static_cast<int>(tt); p.units = static_cast<int>(units);
        const int64_t rounds = (units + most - 1) / most;
        p.clusters = static_cast<int>((units + rounds - 1) / rounds);
        const int64_t items = (groups + cl - 1) / cl * halves * rb;
        p.items = rounds * items;
        p.us = mid_us(mode, rb, nt, cl, rounds, items, 2);
        if (found && p.us >= plan->us) continue;
        if (!mid_buffers(mode, mask, lora, &p)) continue;
        p.us = mid_us(mode, rb, nt, cl, rounds, items, p.nbuf);
        if (!found || p.us < plan->us) { *plan = p; found = true; }
      }
    }
  }
  return found;
}

static thread_local int64_t g_mid_searches = 0;
bool mid_plan(int mode, int64_t M, int64_t NO, int64_t KC, bool mask, int64_t gu_inter, bool lora, int rb, int nt, int cl, MidPlan* plan) {
  static thread_local KeptPlans<MidPlan, 6> kept;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  const int64_t key[6] = {M, NO, KC, gu_inter, mode | (mask ? 2 : 0) | (lora ? 4 : 0) | (static_cast<int64_t>(dev) << 8), rb | (nt << 4) | (cl << 16)};
  return kept.get(key, plan, [&](MidPlan* p) {
    ++g_mid_searches;
    return mid_search(mode, M, NO, KC, mask, gu_inter, lora, rb, nt, cl, p);
  });
}
int64_t mid_searches() { return g_mid_searches; }
static thread_local int64_t g_mid_calls = 0;
int64_t mid_calls() { return g_mid_calls; }

template <int MODE, int RB>
static int mid_launch_cfg(const CUtensorMap& mx, const CUtensorMap& mn, const MidParams& p, const MidPlan& pl, int smem, cudaStream_t stream) {
  auto kernel = nf4_mid_kernel<MODE, RB>;
  NF4LL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMidSmem));
  PdlLaunch lc(dim3(static_cast<unsigned>(pl.clusters * pl.cl)), dim3(kMidThreads), smem, stream, pl.cl > 1 ? pl.cl : 0, pl.cl > 1 ? 1 : 0);
  NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, kernel, mx, mn, p));
  return NF4LL_OK;
}

int mid_launch(const MidCall& c, const MidPlan& pl, bool early, int32_t* status, cudaStream_t stream) {
  ++g_mid_calls;
  const nf4ll_mat* W = c.W;
  const bool fwd = c.mode == kFwd;
  MidParams p{};
  p.qabs = W->qabs; p.scale2 = W->scale2; p.offset2 = W->offset2; p.code2 = W->code2;
  p.N = static_cast<int>(W->N); p.K = static_cast<int>(W->K); p.M = static_cast<int>(c.M);
  p.NO = static_cast<int>(fwd ? W->N : W->K);
  p.steps = static_cast<int>((fwd ? W->K : W->N) / 64);
  p.nt = pl.nt; p.cl = pl.cl; p.tiles_t = pl.tiles_t; p.units = pl.units; p.nbuf = pl.nbuf; p.na = pl.na; p.nx = pl.nx; p.nc = pl.nc;
  p.nc_log = pl.nc == 8 ? 3 : pl.nc == 4 ? 2 : 1;
  p.ts = (pl.nt / 8 + pl.cl - 1) / pl.cl * 8;
  p.split = pl.split ? 1 : 0;
  p.n_seg = c.n_seg;
  for (int i = 0; i < c.n_seg; ++i) {
    p.seg_end[i] = static_cast<int>(c.seg_end[i]);
    p.seg_left[i] = c.seg_left[i]; p.seg_right[i] = c.seg_right[i]; p.seg_scale[i] = c.seg_scale[i];
    if (c.seg_left[i]) p.any_lora = 1;
  }
  const MidLayout l = mid_layout(c.mode, pl, p.any_lora != 0);
  p.off_a = l.off_a; p.off_x = l.off_x; p.off_lora = l.off_lora; p.off_xch = l.off_xch; p.off_lut = l.off_lut; p.off_turn = l.off_turn; p.off_misc = l.off_misc;
  p.early = early ? 1 : 0;
  const uintptr_t blocks_aligned = static_cast<uintptr_t>(W->K / 64) | reinterpret_cast<uintptr_t>(W->qabs);
  p.qabs_mode = blocks_aligned % 4 == 0 ? 4 : blocks_aligned % 2 == 0 ? 2 : 1;
  p.x_alias = pl.x_alias ? 1 : 0;
  p.out = static_cast<__half*>(c.out); p.ldo = c.ldo;
  p.bias = static_cast<const __half*>(c.bias);
  p.accumulate = c.accumulate;
  p.mask = c.mask; p.ld_mask = c.ld_mask; p.keep_scale = c.keep_scale;
  p.gu_inter = static_cast<int>(c.gu_inter);
  p.out_u = static_cast<__half*>(c.out_u); p.ldu = c.ldu;
  p.out_h = static_cast<__half*>(c.out_h); p.ldh = c.ldh;
  p.status = status;
  p.withhold = c.withhold;
  p.wait_ns = c.withhold ? static_cast<uint64_t>(c.wait_us) * 1000 : kWaitLimitNs;
  const bool wide = fwd || pl.rb == 2;           // backward with one row block: its 128 columns are 64 bytes of codes
  CUtensorMap mx, mn;
  if (int rc = mid_encode(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, c.act, static_cast<uint64_t>(p.steps) * 64, static_cast<uint64_t>(c.M),
                          static_cast<uint64_t>(c.ldact) * 2, 64, static_cast<uint32_t>(pl.nt), CU_TENSOR_MAP_SWIZZLE_128B, "token tile")) return rc;
  if (int rc = mid_encode(&mn, CU_TENSOR_MAP_DATA_TYPE_UINT8, W->nib, static_cast<uint64_t>(W->K / 2), static_cast<uint64_t>(W->N),
                          static_cast<uint64_t>(W->K / 2), wide ? 128 : 64, 128, wide ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, "codes")) return rc;
  if (fwd) return pl.rb == 1 ? mid_launch_cfg<kFwd, 1>(mx, mn, p, pl, l.total, stream) : mid_launch_cfg<kFwd, 2>(mx, mn, p, pl, l.total, stream);
  return pl.rb == 1 ? mid_launch_cfg<kBwd, 1>(mx, mn, p, pl, l.total, stream) : mid_launch_cfg<kBwd, 2>(mx, mn, p, pl, l.total, stream);
}

}  // namespace nf4ll
