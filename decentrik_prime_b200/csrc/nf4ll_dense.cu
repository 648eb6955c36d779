// Large-batch GEMM behind nf4ll_forward / nf4ll_forward_multi / nf4ll_forward_gate_up / nf4ll_backward_dx:
// the weight is dequantised ONCE into an fp16 scratch (nf4ll_dequant.cu, bit-exact fp16 weights) and this kernel
// multiplies by it, with the LoRA branch, bias, dropout mask and gated product fused as in the in-kernel-decode
// kernels.
//
// Why: the kernels that decode inside the GEMM decode every weight once per 256-row (pair: 512-row) block of the
// batch, so from several hundred rows on the decode and its shared-memory traffic, not the tensor pipe, set their
// pace. One pass over the weights in HBM / L2 costs 2.5 B per weight instead.
//
// What bounds it: the tensor pipe, with shared-memory and L2-to-SM bandwidth close behind it and, in long runs, the
// power cap. Per CTA pair a 512 x 256 tile: two accumulators of tcgen05.mma.cta_group::2 (M = 256, N = 256, K = 16) that
// fill tensor memory, operands by TMA (128-byte swizzle) through a ring of four 64-wide stages. Consecutive MMAs
// alternate between the accumulators on the SAME weight operand: measured 1075 clocks per 64-wide stage (1024 at full
// rate) against 1590 when one accumulator took its four steps before the other, and 646 per stage of half the work for a
// 256 x 256 tile, which also needs 64 B per clock and SM from L2 where the GPU delivered 38.
// There is no second set of accumulators to hide the epilogue behind; instead the two run out of step at a tile's ends:
// the last k-blocks go to accumulator 0 first, which is drained while accumulator 1 gets them, and the next tile starts
// on accumulator 0 while accumulator 1 is drained. Persistent, one pair per two SMs.
//
// Work distribution: tiles in an order that keeps eight row blocks together (their activations and the weight columns
// in flight stay in L2); whole waves are dealt out one tile per pair. Where the tiles left over would occupy at most half
// of the pairs, a second launch cuts each of them into 2-4 equal parts of the contraction, one pair per part, all pairs
// of a tile in one cluster: the parts exchange partial sums through distributed shared memory (the operand rings are idle
// by then) so that each finishes its share of the columns. Summation order is fixed. Passing the partial sums through
// global memory was measured first: 18 B per clock and SM of writes and 2-3k clocks per dependent read made the exchange
// cost 36k clocks for 2048 x 1536 x 8960, more than half of the GEMM itself.
//
// Warps: 0 TMA producer, 1 MMA issuer (rank 0 of each pair), 2-9 epilogue in two groups of four. The epilogue is kept in
// small loops: straight-line code runs at instruction-fetch speed here (every line is fetched once per tile).
#include "nf4ll_dense.cuh"

namespace nf4ll {

constexpr int kDnStages = 4;
constexpr int kDnABytes = 2 * 128 * 128;               // this CTA's 128 activation rows x 64 fp16 of each accumulator
constexpr int kDnBBytes = 128 * 128;                   // this CTA's half of the 256 weight rows / columns
constexpr int kDnStageBytes = kDnABytes + kDnBBytes;
constexpr int kDnEpiWarps = 8;
constexpr int kDnThreads = 32 * (2 + kDnEpiWarps);
constexpr int kDnStaging = kDnEpiWarps * 4096;         // per epilogue warp one box of 32 rows x 64 columns fp16
constexpr int kDnSmemBytes = 1024 + kDnStages * kDnStageBytes + kDnStaging + 256;
constexpr int kDnLoraStep = 4096;                      // bytes of one rank-16 operand (128 x 16 fp16)

// 2-D tile load whose completion is counted on the barrier of either CTA of the pair (here: rank 0's)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* tmap, int x, int y, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(cluster_bar)
      : "memory");
}
// arrive on the barrier at the same shared-memory offset in the CTAs of `mask` once this thread's MMAs are done
__device__ __forceinline__ void tc_commit2_mask(uint32_t bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask)
               : "memory");
}
__device__ __forceinline__ void st_cluster128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Wait without polling: shared memory runs close to its bandwidth here (operand reads, TMA writes), and every poll is
// an access to it. One test, then the suspended wait, which the hardware resumes when the phase completes.
__device__ __forceinline__ bool dense_wait(uint32_t bar, uint32_t parity, const Abort& ab, int code) {
  if (mbar_test_wait_cluster(bar, parity)) return true;
  const uint64_t t0 = global_timer_ns();
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    if (*ab.flag) return false;
    if ((i & 63u) == 63u && global_timer_ns() - t0 > kWaitLimitNs) break;
  }
  ab.raise(code);
  return false;
}

// tile index -> (row block, column block): groups of eight row blocks, columns within a group, rows fastest
__device__ __forceinline__ void dense_tile_pos(const DenseParams& p, int tile, int& tm, int& to) {
  const int per_group = 8 * p.tiles_o;
  const int g = tile / per_group, r = tile - g * per_group;
  const int gm = (p.tiles_m - g * 8 < 8) ? p.tiles_m - g * 8 : 8;
  to = r / gm;
  tm = g * 8 + (r - to * gm);
}

// The rank-16 steps of a tile: one over all 256 columns when both 128-column halves belong to the same branch, else one
// per half, of 128 columns: a branch whose product is infinite or NaN must not reach the other half's columns (times
// zeros it would). A half without a branch multiplies one block of zeros, which TMA supplies by reading outside a factor, by
// itself.
struct DenseLora {
  int n;              // steps: 0, 1 (whole tile) or 2 (halves)
  int seg[2];         // -1: no branch
};
template <int MODE>
__device__ __forceinline__ DenseLora dense_lora(const DenseParams& p, int64_t o0) {
  DenseLora l;
  l.n = 0; l.seg[0] = l.seg[1] = 0;
  if (p.n_lora == 0) return l;
  if (MODE == kBwd || (p.n_seg == 0 && p.gu_inter == 0)) { l.n = 1; return l; }
  int s0 = 0, s1 = 1;
  if (p.gu_inter == 0) {
    s1 = 0;
    for (int i = 1; i < p.n_seg; ++i) {
      if (o0 >= p.seg_begin[i]) s0 = i;
      if (o0 + 128 >= p.seg_begin[i] && p.seg_begin[i] < p.NO) s1 = i;
    }
  }
  l.seg[0] = p.lora_index[s0] >= 0 ? s0 : -1;
  l.seg[1] = p.lora_index[s1] >= 0 ? s1 : -1;
  if (s0 == s1) l.n = l.seg[0] >= 0 ? 1 : 0;
  else l.n = (l.seg[0] >= 0 || l.seg[1] >= 0) ? 2 : 0;
  return l;
}

// PARTS = 1: whole tiles first_tile .. end_tile - 1, dealt out to the pairs. PARTS > 1: cluster c works on tile
// first_tile + c, its pairs on PARTS equal parts of the contraction.
template <int MODE, int PARTS>
__global__ void __launch_bounds__(kDnThreads, 1)
dense_gemm_kernel(const __grid_constant__ DenseMaps maps, const __grid_constant__ DenseParams p) {
  constexpr int S = kDnStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sStaging = smem + S * kDnStageBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStaging + kDnStaging);
  uint64_t* full = bars;               // [S] rank 0 only: both CTAs' boxes of the stage have landed
  uint64_t* empty = bars + S;          // [S] the MMAs that read the stage are done (multicast commit)
  uint64_t* acc_full = bars + 2 * S;   // [2] accumulator complete (multicast commit)
  uint64_t* acc_empty = acc_full + 2;  // [2] rank 0 only: both CTAs' epilogue warps have read it
  uint64_t* pre_full = acc_full + 4;   // [2] LoRA product of the next tile in the accumulator (multicast commit)
  uint64_t* pre_done = acc_full + 6;   // [2] rank 0 only: it has been multiplied by the dropout mask
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank(), rank = crank & 1, lead = crank & ~1u;      // lead: cluster rank of this pair's rank 0
  const int part = PARTS > 1 ? static_cast<int>(crank >> 1) : 0;
  const int step = PARTS > 1 ? p.end_tile : static_cast<int>(gridDim.x >> 1);
  const int tile0 = p.first_tile + (PARTS > 1 ? static_cast<int>(blockIdx.x) / (2 * PARTS) : static_cast<int>(blockIdx.x >> 1));
  const int kb0 = p.nkb * part / PARTS, kb1 = p.nkb * (part + 1) / PARTS;
  const uint16_t both = static_cast<uint16_t>(3u << lead);
  const Abort ab{abort_flag, p.status};
  const bool lora_part = p.n_lora > 0 && part == 0;
  const bool premask = MODE == kBwd && lora_part && p.mask != nullptr;

  if (warp == 0 && lane == 0) { tma_prefetch_desc(&maps.act); tma_prefetch_desc(&maps.w); }
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) { mbar_init(smem_u32(full + s), 1); mbar_init(smem_u32(empty + s), 1); }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(acc_full + b), 1);
      mbar_init(smem_u32(acc_empty + b), 2 * kDnEpiWarps);
      mbar_init(smem_u32(pre_full + b), 1);
      mbar_init(smem_u32(pre_done + b), 2 * kDnEpiWarps);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc2(smem_u32(tmem_slot), 512);
    tmem_relinquish2();
  }
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  cluster_sync_all();          // the barriers exist before anybody signals across CTAs
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Only the weight and the rank-16 operands come from the kernel right before this one (the dequantisation pass), and only
  // the producer reads them; that kernel itself started after everything earlier on the stream had finished. The second
  // launch of a GEMM has the first one before it and waits for it in the same place.

  if (warp == 0) {
    // ----------------------------------------------------------------------------- TMA producer (own rows, own half)
    if (lane == 0) {
      int n = 0;               // stages filled so far
      bool ok = true;
      auto acquire = [&](uint32_t bytes_per_cta) -> uint32_t {      // the barrier the stage's loads are counted on
        const int s = n % S;
        if (!dense_wait(smem_u32(empty + s), ((n / S) & 1) ^ 1, ab, 0x0101)) { ok = false; return 0; }
        if (rank == 0) mbar_arrive_expect_tx(smem_u32(full + s), 2 * bytes_per_cta);
        return map_to_cta(smem_u32(full + s), lead);
      };
      // the rank-16 operands of a tile: per step a left block for each accumulator and a right block
      auto load_lora = [&](int tile) {
        int tm, to;
        dense_tile_pos(p, tile, tm, to);
        const int64_t o0 = static_cast<int64_t>(to) * (p.gu_inter ? 128 : 256);
        const DenseLora l = dense_lora<MODE>(p, o0);
        if (l.n == 0) return;
        const bool none0 = MODE == kFwd && l.n == 2 && l.seg[0] < 0, none1 = MODE == kFwd && l.n == 2 && l.seg[1] < 0;
        const uint32_t bar = acquire((l.n * 3 - (none0 || none1 ? 2 : 0)) * kDnLoraStep);
        if (!ok) return;
        const uint32_t base = smem_u32(smem) + (n % S) * kDnStageBytes;
        const int m0 = tm * 512 + static_cast<int>(rank) * 128;
        for (int k = 0; k < l.n; ++k) {
          const bool none = k ? none1 : none0;
          const int sg = none ? l.seg[1 - k] : l.seg[k];
          const uint32_t kb = base + k * 3 * kDnLoraStep;
#pragma unroll 1
          for (int h = 0; h < 4 && !none; ++h) {
            const int row = static_cast<int>(p.lora_index[sg] * p.M) + m0 + (h >> 1) * 256;
            tma_load_2d_pair(kb + h * 2048, &maps.left, (h & 1) * 8, row, bar);
          }
          const uint32_t rb = kb + 2 * kDnLoraStep;
          if (MODE == kFwd) {
            // this CTA's half of the step's columns: 128 of 256, or 64 of 128 (the box brings 64 more, which are not used)
            int y = static_cast<int>(l.n == 1 ? o0 + rank * 128 - p.seg_begin[sg]
                                              : (p.gu_inter ? o0 : o0 + k * 128 - p.seg_begin[sg]) + rank * 64);
            if (none) y = static_cast<int>(p.seg_rows[sg]);     // outside: zeros
            tma_load_2d_pair(rb, &maps.right[sg], 0, y, bar);
            tma_load_2d_pair(rb + 2048, &maps.right[sg], 8, y, bar);
          } else {
            const int x = static_cast<int>(o0 + rank * 128);
            tma_load_2d_pair(rb, &maps.right[0], x, 0, bar);
            tma_load_2d_pair(rb + 2048, &maps.right[0], x + 64, 0, bar);
          }
        }
        ++n;
      };
      bool waited = false;
      auto wait_inputs = [&]() { if (!waited) { pdl_wait(); pdl_launch_dependents(); waited = true; } };
      if (lora_part) wait_inputs();
      if (premask && tile0 < p.end_tile) load_lora(tile0);
      for (int tile = tile0; ok && tile < p.end_tile; tile += step) {
        int tm, to;
        dense_tile_pos(p, tile, tm, to);
        const int m0 = tm * 512 + static_cast<int>(rank) * 128;
        int oh;                // first weight row (forward) / column (backward) of this CTA's half
        if (MODE == kFwd && p.gu_inter) oh = to * 128 + (rank ? static_cast<int>(p.gu_inter) : 0);
        else oh = to * 256 + static_cast<int>(rank) * 128;
        if (!premask && lora_part) load_lora(tile);
        int ahead = 0;         // stages whose activation boxes were requested before the weight was ready
        if (!waited) {
          for (; ahead < S && kb0 + ahead < kb1; ++ahead) {
            if (rank == 0) mbar_arrive_expect_tx(smem_u32(full + ahead), 2 * kDnStageBytes);
            const uint32_t bar = map_to_cta(smem_u32(full + ahead), lead), base = smem_u32(smem) + ahead * kDnStageBytes;
            tma_load_2d_pair(base, &maps.act, (kb0 + ahead) * 64, m0, bar);
            tma_load_2d_pair(base + 16384, &maps.act, (kb0 + ahead) * 64, m0 + 256, bar);
          }
          wait_inputs();
        }
#pragma unroll 1
        for (int kb = kb0; kb < kb1; ++kb) {
          uint32_t bar;
          const uint32_t base = smem_u32(smem) + (n % S) * kDnStageBytes;
          if (kb - kb0 < ahead) {
            bar = map_to_cta(smem_u32(full + n % S), lead);
          } else {
            bar = acquire(kDnStageBytes);
            if (!ok) break;
            tma_load_2d_pair(base, &maps.act, kb * 64, m0, bar);
            tma_load_2d_pair(base + 16384, &maps.act, kb * 64, m0 + 256, bar);
          }
          if (MODE == kFwd) {
            tma_load_2d_pair(base + kDnABytes, &maps.w, kb * 64, oh, bar);
          } else {
            tma_load_2d_pair(base + kDnABytes, &maps.w, oh, kb * 64, bar);
            tma_load_2d_pair(base + kDnABytes + 8192, &maps.w, oh + 64, kb * 64, bar);
          }
          ++n;
        }
        if (ok && premask && tile + step < p.end_tile) load_lora(tile + step);
      }
      wait_inputs();           // a pair without tiles still counts for the dependent launch
      if (*abort_flag && rank == 0) {
        // give copies still in flight a bounded chance to land before the CTA goes away
        for (int i = (n > S ? n - S : 0); i < n; ++i)
          for (int spin = 0; spin < (1 << 16) && !mbar_try_wait(smem_u32(full + (i % S)), (i / S) & 1); ++spin) {}
      }
    }
  } else if (warp == 1) {
    // ----------------------------------------------------------------------------- MMA issuer
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = make_idesc_f16(256, 256, 0, MODE == kBwd ? 1 : 0), idesc_half = make_idesc_f16(256, 128, 0, 0);
      const int G = premask ? 3 : 2;             // k-blocks the accumulators run apart at the ends of a tile
      const int cnt = kb1 - kb0;
      int n = 0, i = 0;                          // stages consumed by accumulator 0, tiles started
      int lora_at = 0;                           // ring position of the current tile's rank-16 operands
      DenseLora lora;
      lora.n = 0;
      bool ok = true;
      auto stage_base = [&](int at) { return smem_u32(smem) + (at % S) * kDnStageBytes; };
      auto wait_stage = [&](int at) -> bool {
        if (!dense_wait(smem_u32(full + at % S), (at / S) & 1, ab, 0x0203)) { ok = false; return false; }
        tc_fence_after();
        return true;
      };
      auto wait_acc = [&](int mt, int item) -> bool {
        if (!dense_wait(smem_u32(acc_empty + mt), (item & 1) ^ 1, ab, 0x0204)) { ok = false; return false; }
        tc_fence_after();
        return true;
      };
      auto find_lora = [&](int tile) {
        if (!lora_part) return;
        int tm, to;
        dense_tile_pos(p, tile, tm, to);
        lora = dense_lora<MODE>(p, static_cast<int64_t>(to) * (p.gu_inter ? 128 : 256));
      };
      // the rank-16 steps as the first products of accumulator mt
      auto mma_lora = [&](int mt) {
        const bool halves = MODE == kFwd && lora.n == 2;
#pragma unroll 1
        for (int k = 0; k < lora.n; ++k) {
          const uint32_t kb = stage_base(lora_at) + k * 3 * kDnLoraStep, rb = kb + 2 * kDnLoraStep;
          const uint64_t ad = make_smem_desc(halves && lora.seg[k] < 0 ? rb : kb + mt * kDnLoraStep, 2048, 128, kSwizzleNone);
          const uint64_t bd = (MODE == kFwd) ? make_smem_desc(rb, 2048, 128, kSwizzleNone) : make_smem_desc(rb, 2048, 1024, kSwizzle128B);
          tc_mma2_f16(tmem_base + mt * 256 + (halves ? k * 128 : 0), ad, bd, halves ? idesc_half : idesc, 0u);
        }
      };
      auto b_desc = [&](uint32_t b_base, int kk) {
        return (MODE == kFwd) ? make_smem_desc(b_base + kk * 32, 16, 1024, kSwizzle128B) : make_smem_desc(b_base + kk * 2048, 8192, 1024, kSwizzle128B);
      };
      auto mma_block = [&](int mt, int at, bool fresh) {
        const uint32_t a_base = stage_base(at) + mt * 16384, b_base = stage_base(at) + kDnABytes;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          tc_mma2_f16(tmem_base + mt * 256, make_smem_desc(a_base + kk * 32, 16, 1024, kSwizzle128B), b_desc(b_base, kk), idesc,
                      (!fresh || kk > 0) ? 1u : 0u);
      };
      int pre_n[2] = {0, 0};                     // masked LoRA products per accumulator so far
      auto wait_pre = [&](int mt) -> bool {
        if (!dense_wait(smem_u32(pre_done + mt), pre_n[mt] & 1, ab, 0x0202)) { ok = false; return false; }
        ++pre_n[mt];
        tc_fence_after();
        return true;
      };

      if (tile0 < p.end_tile) {
        find_lora(tile0);
        if (premask) {
          lora_at = n++;
          if (wait_stage(lora_at)) { mma_lora(0); tc_commit2_mask(smem_u32(pre_full), both); }
        }
      }
      for (int tile = tile0; ok && tile < p.end_tile; tile += step) {
        const bool has_lora = lora.n > 0;
        const bool next_pre = premask && tile + step < p.end_tile;
        if (premask) {
          if (!wait_pre(0)) break;
        } else {
          if (!wait_acc(0, i)) break;
          if (has_lora) {
            lora_at = n++;
            if (!wait_stage(lora_at)) break;
            mma_lora(0);
          }
        }
        int done = 0;
#pragma unroll 1
        while (ok && done < cnt) {
          // the first and the last G blocks in one go per accumulator, single blocks in between
          const int left = cnt - done;
          const bool first = done == 0;
          int g = 1;
          if (first) g = left < G ? left : G;
          else if (left <= G) g = left;
          const bool last = g == left;
          if (!first && !last) {
            // both accumulators step by step: consecutive MMAs share the weight operand
            if (!wait_stage(n)) break;
            const uint32_t a_base = stage_base(n), b_base = a_base + kDnABytes;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
              const uint64_t bd = b_desc(b_base, kk);
              tc_mma2_f16(tmem_base, make_smem_desc(a_base + kk * 32, 16, 1024, kSwizzle128B), bd, idesc, 1u);
              tc_mma2_f16(tmem_base + 256, make_smem_desc(a_base + 16384 + kk * 32, 16, 1024, kSwizzle128B), bd, idesc, 1u);
            }
            tc_commit2_mask(smem_u32(empty + n % S), both);
            ++n;
            ++done;
            continue;
          }
#pragma unroll 1
          for (int j = 0; j < g; ++j) {
            if (!wait_stage(n + j)) break;
            mma_block(0, n + j, first && j == 0 && !has_lora);
            if (first && j == 0 && premask) {
              // accumulator 1's LoRA product as soon as it is drained, so that the mask pass on it is over in time
              if (!wait_acc(1, i)) break;
              mma_lora(1);
              tc_commit2_mask(smem_u32(empty + lora_at % S), both);
              tc_commit2_mask(smem_u32(pre_full + 1), both);
            }
          }
          if (!ok) break;
          if (last) tc_commit2_mask(smem_u32(acc_full), both);
          if (first) {
            if (premask) {
              if (!wait_pre(1)) break;
            } else {
              if (!wait_acc(1, i)) break;
              if (has_lora) { mma_lora(1); tc_commit2_mask(smem_u32(empty + lora_at % S), both); }
            }
          }
#pragma unroll 1
          for (int j = 0; j < g; ++j) {
            if (last && j == g - 1 && next_pre) {
              // the next tile's LoRA product on accumulator 0, before this tile's last block on accumulator 1
              find_lora(tile + step);
              lora_at = n + g;
              if (!wait_acc(0, i + 1) || !wait_stage(lora_at)) break;
              mma_lora(0);
              tc_commit2_mask(smem_u32(pre_full), both);
            }
            mma_block(1, n + j, first && j == 0 && !has_lora);
            tc_commit2_mask(smem_u32(empty + (n + j) % S), both);
          }
          if (!ok) break;
          n += g;
          done += g;
          if (last) tc_commit2_mask(smem_u32(acc_full + 1), both);
        }
        if (!ok) break;
        if (next_pre) ++n;                       // its rank-16 operands took a stage
        else if (tile + step < p.end_tile) find_lora(tile + step);
        ++i;
      }
      if (!ok) {
        // nothing may still run on the tensor core when tensor memory is freed: this commit covers all MMAs so far. The
        // barrier may lie one phase behind or ahead of the tile; either parity ends the (bounded) wait at worst late
        tc_commit2_mask(smem_u32(acc_full + 1), both);
        for (int spin = 0; spin < (1 << 16) && !mbar_try_wait(smem_u32(acc_full + 1), i & 1); ++spin) {}
      }
    }
  } else {
    // ----------------------------------------------------------------------------- epilogue
    const int ew = warp - 2, grp = ew >> 2, q = warp & 3;
    const int r_in = q * 32 + lane;                      // this thread's accumulator row (tensor-memory lane)
    const uint32_t stage = smem_u32(sStaging) + ew * 4096;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t acc_empty0 = map_to_cta(smem_u32(acc_empty), lead), pre_done0 = map_to_cta(smem_u32(pre_done), lead);
    int pre_n[2] = {0, 0};
    bool ok = true;

    // multiply the LoRA product in accumulator mt by keep_scale * mask, in tensor memory (this group: columns 128 grp ..)
    auto apply_mask = [&](int tile, int mt) {
      int tm, to;
      dense_tile_pos(p, tile, tm, to);
      const int64_t row = static_cast<int64_t>(tm) * 512 + mt * 256 + rank * 128 + r_in;
      const int64_t o0 = static_cast<int64_t>(to) * 256 + grp * 128;
      uint4 m[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {              // in flight while the rank-16 MMA is awaited
        m[u] = make_uint4(0, 0, 0, 0);
        if (row < p.M && o0 + u * 16 < p.NO) m[u] = __ldg(reinterpret_cast<const uint4*>(p.mask + row * p.ld_mask + o0 + u * 16));
      }
      if (!dense_wait(smem_u32(pre_full + mt), pre_n[mt] & 1, ab, 0x0301)) { ok = false; return; }
      ++pre_n[mt];
      tc_fence_after();
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t taddr = lane_base + mt * 256 + grp * 128 + u * 32;
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(taddr, v);
        tmem_ld_wait();
        const uint32_t mk[8] = {m[2 * u].x, m[2 * u].y, m[2 * u].z, m[2 * u].w, m[2 * u + 1].x, m[2 * u + 1].y, m[2 * u + 1].z, m[2 * u + 1].w};
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const bool keep = ((mk[j >> 2] >> ((j & 3) * 8)) & 0xffu) != 0;
          v[j] = keep ? __float_as_uint(__uint_as_float(v[j]) * p.keep_scale) : 0u;
        }
        tmem_st32(taddr, v);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(pre_done0 + mt * 8);
    };
    // 64 columns of an accumulator, plus bias, rounded
    auto round64 = [&](const uint32_t (&v0)[32], const uint32_t (&v1)[32], const __half* bias, uint4 (&h)[8]) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float f[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] = __uint_as_float(j < 4 ? v0[8 * (j & 3) + k] : v1[8 * (j & 3) + k]);
        if (MODE == kFwd && bias) {
          float b[8];
          unpack8(__ldg(reinterpret_cast<const uint4*>(bias) + j), b);
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] += b[k];
        }
        h[j] = pack8(f);
      }
    };
    // this warp's 32 rows x 64 columns through its staging box to TMA
    auto put_box = [&](const void* map, const uint4 (&h)[8], int col, int row0) {
      if (lane == 0) bulk_wait_read_all();
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j) sts128(stage + lane * 128 + ((j ^ (lane & 7)) << 4), h[j]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (MODE == kBwd && p.accumulate) tma_reduce_add_2d(map, stage, col, row0);
        else tma_store_2d(map, stage, col, row0);
        bulk_commit();
      }
    };

    if (premask && tile0 < p.end_tile) { apply_mask(tile0, 0); if (ok) apply_mask(tile0, 1); }
    int i = 0;
    for (int tile = tile0; ok && tile < p.end_tile; tile += step, ++i) {
      int tm, to;
      dense_tile_pos(p, tile, tm, to);
#pragma unroll 1
      for (int mt = 0; mt < 2; ++mt) {
        if (!dense_wait(smem_u32(acc_full + mt), i & 1, ab, 0x0303)) { ok = false; break; }
        tc_fence_after();
        if (PARTS > 1) continue;                 // finished below, together with the other parts
        const int row0 = tm * 512 + mt * 256 + static_cast<int>(rank) * 128 + q * 32;      // of this warp's rows
        const uint32_t tacc = lane_base + mt * 256;
        // all of this thread's 128 columns at once, then the accumulator is free: the next tile's MMAs wait for it
        const bool gu = MODE == kFwd && p.gu_inter;
        const uint32_t t0 = tacc + (gu ? grp * 64 : grp * 128), t1 = gu ? t0 + 128 : t0 + 64;
        uint32_t v[4][32];
        __syncwarp();
        tmem_ld32(t0, v[0]);
        tmem_ld32(t0 + 32, v[1]);
        tmem_ld32(t1, v[2]);
        tmem_ld32(t1 + 32, v[3]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(acc_empty0 + mt * 8);
        const int col = gu ? to * 128 + grp * 64 : to * 256 + grp * 128;
        const __half* bias = p.bias ? p.bias + col : nullptr;
        uint4 h0[8], h1[8];
        if (col < p.NO) {
          round64(v[0], v[1], bias, h0);
          put_box(&maps.out, h0, col, row0);
        }
        if (gu) {
          // columns 64 grp .. +63 of gate and of up, then silu(gate) * up from the rounded values
          round64(v[2], v[3], nullptr, h1);
          put_box(&maps.out_u, h1, col, row0);
#pragma unroll
          for (int j = 0; j < 8; ++j) h1[j] = swiglu_fwd8(h0[j], h1[j]);
          put_box(&maps.out_h, h1, col, row0);
        } else if (col + 64 < p.NO) {
          round64(v[2], v[3], bias ? bias + 64 : nullptr, h1);
          put_box(&maps.out, h1, col + 64, row0);
        }
        if (premask && tile + step < p.end_tile) { apply_mask(tile + step, mt); if (!ok) break; }
      }
    }
    if (lane == 0) bulk_wait_all();
  }

  if constexpr (PARTS > 1) {
    // ----------------------------------------------------------------------------- the parts of a tile share its reduction
    // Unit u = accumulator u >> 2, columns 32 (u & 3) .. of an epilogue group's 128; part u % PARTS finishes it. Everybody
    // sends the other parts' units to their CTA of the same rank: block [source][unit / PARTS][group] of 128 rows x 32
    // fp32 in the operand ring, which no MMA reads any more once the whole cluster has got here.
    constexpr int kOwn = (8 + PARTS - 1) / PARTS;
    static_assert((PARTS - 1) * kOwn * 2 * 16384 <= S * kDnStageBytes, "exchange must fit the operand ring");
    __syncwarp();
    cluster_sync_all();
    const int grp = (warp - 2) >> 2, q = warp & 3, r_in = q * 32 + lane;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + grp * 128;
    const bool live = warp >= 2 && !*abort_flag;
    if (live) {
      tc_fence_after();
#pragma unroll 1
      for (int u = 0; u < 8; ++u) {
        const int d = u % PARTS;
        if (d == part) continue;
        const int src = part < d ? part : part - 1;
        const uint32_t dst = map_to_cta(smem_u32(smem) + ((src * kOwn + u / PARTS) * 2 + grp) * 16384 + r_in * 16, 2 * d + rank);
        uint32_t v[32];
        __syncwarp();
        tmem_ld32(lane_base + (u >> 2) * 256 + (u & 3) * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) st_cluster128(dst + j * 2048, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (live) {
      int tm, to;
      dense_tile_pos(p, tile0, tm, to);
#pragma unroll 1
      for (int u = part; u < 8; u += PARTS) {
        uint32_t own[32];
        __syncwarp();
        tmem_ld32(lane_base + (u >> 2) * 256 + (u & 3) * 32, own);
        tmem_ld_wait();
        const int64_t row = static_cast<int64_t>(tm) * 512 + (u >> 2) * 256 + rank * 128 + r_in;
        const int64_t col = static_cast<int64_t>(to) * 256 + grp * 128 + (u & 3) * 32;
        const bool store = row < p.M && col < p.NO;
        __half* dst = p.out + row * p.ldo + col;
        const uint4* more16 = nullptr;           // what is added before the one rounding: bias, or the output's previous value
        if (MODE == kFwd) { if (p.bias && store) more16 = reinterpret_cast<const uint4*>(p.bias + col); }
        else if (p.accumulate && store) more16 = reinterpret_cast<const uint4*>(dst);
        uint4 h[4];
#pragma unroll
        for (int j8 = 0; j8 < 4; ++j8) {
          float f[8];
#pragma unroll
          for (int k = 0; k < PARTS; ++k) {      // part order
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
              uint4 w = make_uint4(own[j8 * 8 + hh * 4], own[j8 * 8 + hh * 4 + 1], own[j8 * 8 + hh * 4 + 2], own[j8 * 8 + hh * 4 + 3]);
              if (k != part)
                w = lds128(smem_u32(smem) + (((k < part ? k : k - 1) * kOwn + u / PARTS) * 2 + grp) * 16384 + r_in * 16 + (j8 * 2 + hh) * 2048);
              const float t[4] = {__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w)};
#pragma unroll
              for (int e = 0; e < 4; ++e) f[hh * 4 + e] = (k == 0) ? t[e] : f[hh * 4 + e] + t[e];
            }
          }
          if (more16) {
            float b[8];
            unpack8(more16[j8], b);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] += b[e];
          }
          h[j8] = pack8(f);
        }
        if (store) {
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(dst + 8 * j) = h[j];
        }
      }
    }
  }

  // ------------------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncwarp();
  __syncthreads();
  cluster_sync_all();        // no CTA may free tensor memory or leave while another still uses its resources
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------------------
// Plan and launch
// ---------------------------------------------------------------------------------------------
template <int MODE>
static auto dense_kernel(int parts) {
  return parts == 1 ? dense_gemm_kernel<MODE, 1> : (parts == 2 ? dense_gemm_kernel<MODE, 2>
                                                  : (parts == 3 ? dense_gemm_kernel<MODE, 3> : dense_gemm_kernel<MODE, 4>));
}

// Clusters of 2 * parts CTAs of this kernel that the current device holds at once (it depends on how many SMs each of its
// GPCs has: 33 / 22 / 15 for 2 / 3 / 4 parts where measured). Asked once per device.
static int dense_clusters(int parts) {
  constexpr int kMaxDevices = 64;
  static int cached[kMaxDevices][3];             // 0: not asked yet; written with the same value by any thread
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  int n = __atomic_load_n(&cached[dev][parts - 2], __ATOMIC_RELAXED);
  if (n == 0) {
    auto kernel = dense_kernel<kFwd>(parts);
    PdlLaunch probe(dim3(static_cast<unsigned>(2 * parts)), dim3(kDnThreads), kDnSmemBytes, nullptr, 2 * parts, 1, false, false);
    probe.cfg.numAttrs = 1;                      // the cluster dimension only
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDnSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &probe.cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = -1;
    }
    __atomic_store_n(&cached[dev][parts - 2], n, __ATOMIC_RELAXED);
  }
  return n;
}

DensePlan dense_plan(int64_t M, int64_t NO, int64_t KC, int64_t gu_inter, int sms) {
  DensePlan d{};
  const int64_t pairs = sms / 2;
  d.tiles_m = (M + 511) / 512;
  d.tiles_o = gu_inter ? (gu_inter + 127) / 128 : (NO + 255) / 256;
  d.tiles = d.tiles_m * d.tiles_o;
  d.nkb = static_cast<int>(KC / 64);
  d.whole = d.tiles;
  d.parts = 1;
  // A last wave of at most half the pairs: cut its tiles. Costs in k-blocks of time: the exchange 7 and 2 per part, a second
  // launch 8. Cut / whole in us, forward: 16 k-blocks, 12 tiles in 4 parts 27.6 / 23.6 (not cut); 24, 12 in 4 27.6 / 29.7;
  // 64, 5 in 4 34 / 54; with whole waves before them 24, 6 in 4 54 / 50 (not cut); 40, 12 in 4 101 / 103; 56, 4 in 4 298 / 310.
  // gate|up pairs columns of both halves of a tile in its epilogue and is not cut.
  const int64_t rest = d.tiles % pairs;
  if (rest > 0 && rest * 2 <= pairs && !gu_inter) {
    int64_t best = d.nkb;
    for (int s = 2; s <= 4; ++s) {
      if (d.nkb < 4 * s || rest > dense_clusters(s)) continue;
      const int64_t cost = (d.nkb + s - 1) / s + kDnExchange(s) + (d.tiles > rest ? kDnSecondLaunch : 0);
      if (cost < best) { best = cost; d.parts = s; }
    }
    if (d.parts > 1) d.whole = d.tiles - rest;
  }
  return d;
}

int dense_launch(int mode, const DenseMaps& maps, const DenseParams& p_in, const DensePlan& d, int sms, cudaStream_t stream) {
  DenseParams p = p_in;
  if (d.whole > 0) {
    auto kernel = mode == kFwd ? dense_kernel<kFwd>(1) : dense_kernel<kBwd>(1);
    NF4LL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDnSmemBytes));
    p.first_tile = 0; p.end_tile = static_cast<int>(d.whole);
    const int64_t pairs = d.whole < sms / 2 ? d.whole : sms / 2;
    PdlLaunch lc(dim3(static_cast<unsigned>(2 * pairs)), dim3(kDnThreads), kDnSmemBytes, stream, 2, 1);
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, kernel, maps, p));
  }
  if (d.whole < d.tiles) {
    auto kernel = mode == kFwd ? dense_kernel<kFwd>(d.parts) : dense_kernel<kBwd>(d.parts);
    NF4LL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDnSmemBytes));
    p.first_tile = static_cast<int>(d.whole); p.end_tile = static_cast<int>(d.tiles);
    PdlLaunch lc(dim3(static_cast<unsigned>(2 * d.parts * (d.tiles - d.whole))), dim3(kDnThreads), kDnSmemBytes, stream, 2 * d.parts, 1);
    NF4LL_CUDA(cudaLaunchKernelEx(&lc.cfg, kernel, maps, p));
  }
  return NF4LL_OK;
}

}  // namespace nf4ll
