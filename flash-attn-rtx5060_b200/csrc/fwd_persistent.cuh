// Warp-specialised persistent attention-forward kernel for sm_100a.
//
// One CTA per SM walks a list of work items (work_items.h); a work item is a pair of adjacent 128-row q tiles of one
// (batch, head), one for each of the two stages, or a single q tile whose kv tiles the stages take in turn. The kv
// tiles are walked from the last visible one to the first. Roles (16 warps):
//   warps 0-3   softmax of stage 0: one thread per score row (TMEM lane), exp2 online softmax
//   warps 4-7   softmax of stage 1
//   warps 8-11  epilogue (O / l, or for a single q tile the sum of both stages' O over the sum of their l, -> fp16 ->
//               the warp's staging area in shared memory -> one TMA store)
//   warp 12     tensor-core issuer: the warp walks the schedule, one elected lane issues tcgen05.mma
//   warp 13     TMA producer: Q tiles and the K/V tile ring
//   warp 14     Q of the CTA's first item, beside the producer's first K/V tiles; else idle, as warp 15 (they only donate
//               registers)
// TMEM columns: S0 [0,128) S1 [128,256) O0 [256,256+D) O1 [384,384+D); the fp16 P tile of a
// stage overwrites the first 64 columns of its own S and is handed to the tensor pipe in two
// parts of 96 and 32 keys, so that most of P.V runs while the last keys are still being exponentiated and little of it
// stands between the last of P and the stage's next score tile.
//
// What sets the pace of a long sequence is the loop of one stage, softmax tile -> rest of P.V -> next score tile ->
// softmax, together with the issue slots of the four SM sub-partitions, each of which runs one softmax warp of either
// stage. Shortening the issuer alone or the softmax alone gained nothing or lost: a faster issuer only made the two
// stages' tiles overlap more. Done together (B200, us): the issuer's products in branch-free groups (umma_pv64 and the
// like) without a vote behind each wait; O rescaled by the softmax warps themselves, which took a hand-over per tile to
// the warps 8-11 off the path; a fifth of the exponentials on the FMA pipe (exp2_poly); what is fixed for an item
// computed once per item. (Short runs at the full clock and scores of spread 1; in rows of calls at the power cap the first and
// third of these gain 3-5 %, and less the wider the scores spread.) B2 H32 N8192 d128 causal 1085 -> 971, B2 H16 N4096 d128 268 -> 237, B4 H16 N16384 d128 window
// 1024 690 -> 613, 24 heads x 4001 rows d128 with log-sum-exp 120 -> 109, 32 heads x 8192 rows d64 761 -> 675, B8 H12
// N1000 d64 50.0 -> 47.4, B4 H16 N2048 d64 causal 66.5 -> 62.8, with dropout 97.2 -> 94.5, ALiBi B2 H16 N4096 d64 128.9
// -> 121.0. Of a round of two tiles at head_dim 128, 2725 clocks of 3050 before, 2370 remain without any products.
//
// Replaces the reference's forward_kernel, Schedule and SMem (src/flash_forward.h:22-366),
// apply_mask (src/mask.h:10-84) and apply_softmax (src/softmax.h:9-86): same function, but
// the contractions run on tcgen05 with TMEM accumulators, the two stages ping-pong so that
// the tensor pipe works on one while the other is in softmax, masks touch only boundary
// tiles, kv tiles outside a q tile's visible range are never loaded for it, and the output
// is rescaled lazily.
#pragma once
#include <type_traits>

#include "fwd_params.h"
#include "ptx.cuh"
#include "work_items.h"


namespace fa {

template <int D>
struct PersistentCfg {
  static constexpr int kThreads = 512;
  static constexpr int kTileBytes = kBlockN * D * 2;
  static constexpr int kPanelBytes = kBlockN * kPanel * 2;
  static constexpr int kStages = (D == 128) ? 4 : 8;  // ring slots, each one K or one V tile
  static constexpr int kOffQ = 0;
  static constexpr int kOffKV = 2 * kTileBytes;
  // Output staging: each epilogue warp owns 32 rows, laid out [panel][row][64] with the 128-byte swizzle, the
  // source of its TMA store.
  static constexpr int kOffOut = kOffKV + kStages * kTileBytes;
  static constexpr int kOutWarpBytes = 32 * D * 2;
  static constexpr int kOffAlpha = kOffOut + 4 * kOutWarpBytes;  // float[2][128]: references of a split item; drop_blocks
  static constexpr int kOffRowSum = kOffAlpha + 2 * kBlockM * 4;   // float[2][128]
  static constexpr int kOffBars = kOffRowSum + 2 * kBlockM * 4;
  static constexpr int kNumBars = 22 + 2 * kStages;
  static constexpr int kOffMisc = kOffBars + kNumBars * 8;
  static constexpr int kOffGeom = kOffMisc + 16;     // TMEM base, abort flag (+ 8 spare bytes)
  static constexpr int kSmemBytes = kOffGeom + 2 * 64;  // two work-item slots: the item's decoded geometry and its id
  static constexpr uint32_t kTmemCols = 512;
  static constexpr uint32_t kColS0 = 0, kColS1 = 128, kColO0 = 256, kColO1 = 384;
  static constexpr uint32_t kOwnPFromS = 320;  // kOwnP: P in columns 320 and 448, beside an O of 64 columns
  // Lazy rescale, in log2 units: a row's reference (the score that its exponentials are taken against) stays where it is
  // until a tile's row max passes it by more than kLazyLog2, so P stays below 2^8, well inside fp16, and l and O, held
  // in fp32, have the room. The key that sets the reference has P = 1 exactly; a key above it has a P rounded to 11 bits,
  // which O keeps while l takes the unrounded exponential, so a row that one such key dominates loses the exactness of
  // its main term. Two rules keep that rare. Once a warp acts for one of its rows, all its rows whose max has grown move
  // along: the cost, 32 exponentials taken again and a rescale of O, is the warp's anyway. And on the first keys of the
  // sequence, which the walk visits last and which many rows of a trained causal model look at, any growth moves it.
  // Error against 64 bits (2-norm, 1e-4; 4 heads x 4096 rows d64; one early key 8 and 12 log2 units above the others;
  // scores of spread 4; of spread 2): 2.14 2.08 2.60 2.84. With 2^14 and neither rule: 2.94 2.93 2.88 2.88; with 2^8
  // and a walk from the first tile to the last: 2.14 2.08 2.63 2.88.
  // What it costs against 2^14 alone (us): B4 H16 N2048 d64 causal 64.7 -> 66.4, B8 H16 N1024 d128 causal 56.8 -> 58.7,
  // 24 heads x 4001 rows d128 causal, log-sum-exp, spread 2 115.9 -> 116.7, B2 H32 N8192 d128 causal 1041 -> 1045 (the
  // running max as such is no longer kept; with ALiBi the register it took matters more: B2 H16 N4096 d64 131.8 -> 128.7).
  static constexpr float kLazyLog2 = 8.f;
  // One pair of exponentials in kPolyOf is taken on the FMA pipe (keys 32-63, 64-95, 96-127 of a tile that is not cut; the
  // first 32 keys share their time with the row max). A softmax tile alone takes 1336 clocks, two at once on a
  // sub-partition 2275; with one pair in four 1243 and 2063. Nearly all at once the special-function unit is no longer the
  // limit, so more does not help: against these fractions (us; B2 H32 N8192 d128 causal, 32 heads x 8192 rows d64, B8 H12
  // N1000 d64: 969, 672, 47.2), half as many 972, 692, 48.4; twice as many in the second part of d128 1061; in the last
  // part 1059, 705, 48.4; one pair in four of the first 32 keys too 991, 745, 51.0. None with dropout, whose mask fills
  // the same pipes (103 -> 101).
  static constexpr int kPolyOf1 = D == 64 ? 2 : 4, kPolyOf2 = 4, kPolyOf3 = 4;
  // Registers per thread after setmaxnreg: 8 softmax warps, 4 epilogue warps, 4 others; 256 * softmax + 128 * epilogue +
  // 128 * others <= 65536. At head_dim 64, where the exponentials are the limit, 200 let more of them be in flight (32
  // heads x 8192 rows 719 -> 680 us); at head_dim 128 it costs 2-4 %. The short build has fewer values live.
  // Columns that the epilogue takes at a time: 8 fit the 40 registers of head_dim 64 (16 spill, 3 % of the smallest calls);
  // at head_dim 128 16 are 3 % faster than 8.
  static constexpr int kEpilogueCols = D == 64 ? 8 : 16;
  static constexpr int kRegSoftmax = D == 64 ? 200 : 184, kRegEpilogue = D == 64 ? 40 : 72, kRegOthers = 72;
  static constexpr int kRegSoftmaxShort = 184, kRegEpilogueShort = 72;
};

// 2^x of two values on the FMA pipe: x = n + f with n the nearest integer (the usual addition of 1.5 * 2^23 rounds x to
// one), 2^f a polynomial, 2^n by way of the exponent field. The polynomial is the minimax approximation of 2^f in
// relative error on [-1/2, 1/2] among those of degree 5 with constant term 1 (Remez exchange): 1.6e-7 in fp32
// arithmetic, where ex2.approx states 2.4e-7. 2^0 is exactly 1; below 2^-126.5, down to -infinity, the result is 0; NaN
// stays NaN (a product, not an addition to the exponent field, and a maximum that keeps it).
__device__ __forceinline__ void exp2_poly(float x0, float x1, float& e0, float& e1) {
  const uint64_t x = f2_pack(max_nan(x0, -127.f), max_nan(x1, -127.f));
  const uint64_t magic = f2_pack(12582912.f, 12582912.f);
  const uint64_t t = f2_add(x, magic);
  const uint64_t f = f2_add(x, f2_fma(t, f2_pack(-1.f, -1.f), magic));
  uint64_t p = f2_fma(f2_pack(0x1.5bba14p-10f, 0x1.5bba14p-10f), f, f2_pack(0x1.3cea88p-7f, 0x1.3cea88p-7f));
  p = f2_fma(p, f, f2_pack(0x1.c6b752p-5f, 0x1.c6b752p-5f));
  p = f2_fma(p, f, f2_pack(0x1.ebf9bcp-3f, 0x1.ebf9bcp-3f));
  p = f2_fma(p, f, f2_pack(0x1.62e42ap-1f, 0x1.62e42ap-1f));
  p = f2_fma(p, f, f2_pack(1.f, 1.f));
  float t0, t1;
  f2_unpack(t, t0, t1);
  const float s0 = __uint_as_float((__float_as_uint(t0) << 23) + 0x3f800000u);
  const float s1 = __uint_as_float((__float_as_uint(t1) << 23) + 0x3f800000u);
  f2_unpack(f2_mul(p, f2_pack(s0, s1)), e0, e1);
}

// exp2 of 2 * kPairs scores -> packed fp16x2 words; adds the exponentials into two (even, odd) pairs of partial row sums.
// Of every kPolyOf pairs one takes exp2_poly instead of the special-function unit (0: none).
template <int kPairs, int kPolyOf>
__device__ __forceinline__ void exp_tile(const float* sc, uint64_t scale2, uint64_t negms2, uint32_t* pk, uint64_t& lsum_a,
                                         uint64_t& lsum_b) {
#pragma unroll
  for (int c = 0; c < kPairs; ++c) {
    float x0, x1, e0, e1;
    f2_unpack(f2_fma(f2_pack(sc[2 * c], sc[2 * c + 1]), scale2, negms2), x0, x1);
    if (kPolyOf > 0 && c % (kPolyOf > 0 ? kPolyOf : 1) == 1) {
      exp2_poly(x0, x1, e0, e1);
    } else {
      e0 = ex2_approx(x0);
      e1 = ex2_approx(x1);
    }
    if (c & 1) lsum_b = f2_add(lsum_b, f2_pack(e0, e1));
    else lsum_a = f2_add(lsum_a, f2_pack(e0, e1));
    pk[c] = pack_f16x2(e0, e1);
  }
}

// Philox-4x32 with 10 rounds (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3"): a keyed bijection of a
// 128-bit counter. Stateless, so the keep mask of dropout depends only on (seed, head, row, column) and is the same
// whatever tile shape or schedule computes it. (The reference keeps ONE generator state per q tile, copies it into
// every thread of the CTA, so all threads draw the same numbers, and stores it back: src/flash_forward.h:185-186,
// :248-265, :361-363. That flaw is not reproduced.)
// The counter is {column block, row, head, 0}, so what the first rounds multiply depends on the row alone or on the block
// alone: DropRow holds the row's part, DropBlock the block's, which 8 lanes of a warp compute for the 8 blocks of a tile
// (they are the same for all rows) and leave in shared memory. Of a block's 20 wide products 15 remain per row.
constexpr uint32_t kPhiloxM0 = 0xD2511F53u, kPhiloxM1 = 0xCD9E8D57u, kPhiloxW0 = 0x9E3779B9u, kPhiloxW1 = 0xBB67AE85u;
struct DropRow { uint32_t hi, lo; };  // second round: product of the row's word
__device__ __forceinline__ DropRow drop_row(const FwdParams& p, int bh, int row) {
  const uint32_t c0 = __umulhi(kPhiloxM1, bh) ^ static_cast<uint32_t>(row) ^ p.seed_lo;
  return {__umulhi(kPhiloxM0, c0), kPhiloxM0 * c0};
}
// Words of the third round that the block alone decides, keys included: {c2, c0, c2 of the next round, c3}
__device__ __forceinline__ uint4 drop_block(const FwdParams& p, int bh, uint32_t block) {
  const uint32_t c2 = __umulhi(kPhiloxM0, block) ^ p.seed_hi;
  const uint32_t c0 = __umulhi(kPhiloxM1, c2) ^ (kPhiloxM1 * static_cast<uint32_t>(bh)) ^ (p.seed_lo + kPhiloxW0);
  return make_uint4((kPhiloxM0 * block) ^ (p.seed_hi + kPhiloxW1), (kPhiloxM1 * c2) ^ (p.seed_lo + 2u * kPhiloxW0),
                    __umulhi(kPhiloxM0, c0) ^ (p.seed_hi + 2u * kPhiloxW1), kPhiloxM0 * c0);
}
__device__ __forceinline__ void drop_words(const FwdParams& p, const DropRow& row, const uint4& blk, uint32_t (&out)[4]) {
  uint32_t c2 = row.hi ^ blk.x;
  uint32_t c0 = __umulhi(kPhiloxM1, c2) ^ blk.y, c1 = kPhiloxM1 * c2, c3 = blk.w;
  c2 = row.lo ^ blk.z;
#pragma unroll
  for (uint32_t r = 3; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(kPhiloxM0, c0), lo0 = kPhiloxM0 * c0;
    const uint32_t hi1 = __umulhi(kPhiloxM1, c2), lo1 = kPhiloxM1 * c2;
    c0 = hi1 ^ c1 ^ (p.seed_lo + r * kPhiloxW0);
    c1 = lo1;
    c2 = hi0 ^ c3 ^ (p.seed_hi + r * kPhiloxW1);
    c3 = lo0;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// Zeroes the dropped elements of kBlocks * 8 packed fp16 pairs (16 columns per block). Byte t of a block's 16 random bytes
// (little endian over the four words) decides column t: kept when below the threshold. Two bytes at a time are compared
// as the fp16 values 1024 + byte, which are exact, and the comparison leaves a mask over the pair.
template <int kBlocks>
__device__ __forceinline__ void dropout_mask(uint32_t* pk, const FwdParams& p, const DropRow& row, const uint4* blocks) {
  const uint32_t limit = 0x64006400u + p.drop_keep_thr * 0x00010001u;
#pragma unroll
  for (int blk = 0; blk < kBlocks; ++blk) {
    uint32_t r[4];
    drop_words(p, row, blocks[blk], r);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      pk[blk * 8 + 2 * w] &= f16x2_less_mask(__byte_perm(r[w], 0x64646464u, 0x4140), limit);      // columns 4w, 4w+1
      pk[blk * 8 + 2 * w + 1] &= f16x2_less_mask(__byte_perm(r[w], 0x64646464u, 0x4342), limit);  // columns 4w+2, 4w+3
    }
  }
}

// kShort: the build for launches whose q tiles see few kv tiles (short_items() in work_items.h). There an item's code comes
// from cold instruction caches as often as not and the time between items weighs as much as the rounds, so what counts is
// how little code there is: cut tiles are blanked in tensor memory by a small loop and go through the same body as all
// others, the row max comes before any exponential (no second copy of the first ones), the issuer has no rounds of its
// own for the inside of an item, and at head_dim 128, where these launches are not bound by the exponentials, none are
// taken on the FMA pipe. ALiBi comes here under a causal mask only: a key left of the diagonal has a bias that is linear in
// the column, and what lies right of it is hidden. (With a body per kind of tile, one of them blanked: nothing gained. In
// long sequences one body costs 3-6 %.)
// kOwnP (own_p_columns() in work_items.h; head_dim 64, short build): P has columns of its own instead of S's, and the next
// score tile is issued ahead of the rest of P.V, so a stage waits for one hand-over and 96 keys' products less per tile.
template <int D, bool kAlibi, bool kLse = false, bool kDropout = false, bool kShort = false, bool kOwnP = false>
__global__ void __launch_bounds__(512, 1)
fwd_persistent_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                      const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapO,
                      const FwdParams p) {
  using Cfg = PersistentCfg<D>;
  constexpr bool kLateO = kShort && !kDropout && !kAlibi;
  static_assert(!kOwnP || (D == 64 && kShort), "columns of P's own lie beside an O of 64 columns");
  extern __shared__ __align__(1024) uint8_t smem[];

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;

  if ((smem_u32(smem) & 1023u) != 0) {  // swizzled tiles need a 1024-byte aligned base
    if (tid == 0) atomicExch(p.status, 2);
    return;
  }

  uint8_t* sQ = smem + Cfg::kOffQ;
  uint8_t* sKV = smem + Cfg::kOffKV;
  float* sAlpha = reinterpret_cast<float*>(smem + Cfg::kOffAlpha);
  float* sRowSum = reinterpret_cast<float*>(smem + Cfg::kOffRowSum);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::kOffBars);
  uint64_t* q_full = bars;            // [2] TMA -> MMA
  uint64_t* q_empty = bars + 2;       // [2] MMA -> TMA
  uint64_t* s_full = bars + 4;        // [2] MMA -> softmax: S tile in TMEM
  uint64_t* p_full = bars + 6;        // [2] softmax -> MMA: P of the first 96 keys written, O rescaled
  uint64_t* o_empty = bars + 8;       // [2] epilogue -> MMA, softmax: O and the row sums of the item have been read
  uint64_t* l_ready = bars + 10;      // [2] softmax -> epilogue: final row sums in smem
  uint64_t* o_full = bars + 12;       // [2] MMA -> epilogue: last P.V of the item landed
  uint64_t* p_full2 = bars + 14;      // [2] softmax -> MMA: rest of P written
  uint64_t* item_full = bars + 16;    // [2] producer -> all roles: next work item id published
  uint64_t* item_empty = bars + 18;   // [2] all roles -> producer: id slot read
  uint64_t* kv_full = bars + 20;      // [kStages] TMA -> MMA
  uint64_t* kv_empty = bars + 20 + Cfg::kStages;  // [kStages] MMA -> TMA
  uint64_t* p_empty = bars + 20 + 2 * Cfg::kStages;  // [2] MMA -> softmax: P.V of the tile complete (kOwnP)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // [2][16]: ItemGeom of the published item in words 0..11, its id (-1: no more items) in word 12, `split` in word 13
  volatile int* s_geom = reinterpret_cast<volatile int*>(smem + Cfg::kOffGeom);
  constexpr uint32_t kItemReaders = 13;  // 8 softmax warps + 4 epilogue warps + the MMA warp

  if (warp == 12) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&q_empty[s], 1);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 4);
      mbar_init(&p_full2[s], 4);
      mbar_init(&o_empty[s], 4);
      mbar_init(&l_ready[s], 4);
      mbar_init(&o_full[s], 1);
      if (kOwnP) mbar_init(&p_empty[s], 1);
      mbar_init(&item_full[s], 1);
      mbar_init(&item_empty[s], kItemReaders);
    }
    for (int i = 0; i < Cfg::kStages; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  // Work item in slot `slot` of s_geom
  auto write_item = [&](uint32_t slot, const ItemGeom& g, int item) {
    volatile int* w = s_geom + slot * 16;
    if (item >= 0) {
      w[0] = g.bh; w[1] = g.pair;
      w[2] = g.r0[0]; w[3] = g.r0[1]; w[4] = g.r1[0]; w[5] = g.r1[1];
      w[6] = g.lo[0]; w[7] = g.lo[1]; w[8] = g.hi[0]; w[9] = g.hi[1];
      w[10] = g.top; w[11] = g.steps; w[13] = g.split;
    }
    w[12] = item;
  };
  ItemGeom g_first;
  g_first.steps = 0;
  if ((warp == 13 || warp == 14) && lane == 0) {
    prefetch_tensormap(&mapK);
    prefetch_tensormap(&mapQ);
    prefetch_tensormap(&mapV);
    prefetch_tensormap(&mapO);
    g_first = decode_item(static_cast<int>(blockIdx.x), p);
    if (warp == 13 && g_first.steps > 0) write_item(0, g_first, static_cast<int>(blockIdx.x));
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Everything above overlaps the end of the kernel in front in the stream, the first item's geometry included. Nothing
  // touches global memory (inputs, outputs, scheduler words, status) before that kernel is complete: every role waits for
  // it at its beginning. The issuer, which works on what the producer loads, does so because the limit of its bounded
  // waits is meant for this launch: a kernel in front that lets this one in early may go on for longer. (Its cost: none in the
  // cases measured, up to 1.4 % for long rows with the log-sum-exp at head_dim 128, 245 -> 248 us for 32 x 4096.)
  // A short launch is one chain of latencies: with the first item decoded here, the next launch let in at once where each
  // CTA has one item, the first loads without waits, and the last CTA found by the producers instead of at the very end,
  // calls in a row take (us, B200): 1 head x 64 rows d64 6.8 -> 5.0, 4 x 512 d64 9.4 -> 7.2, 8 x 333 d128 causal
  // 10.4 -> 8.1, 16 x 256 d128 8.3 -> 6.2, 8 x 1024 d128 causal 13.8 -> 11.9. With a warp of its own for the first Q tiles
  // and the next launch let in behind the first loads: 4.5, 6.8, 7.9, 5.9, 11.9. (Running a tile's code once on nothing
  // while the first loads are under way, so that it comes from the instruction caches, gained nothing in a row of calls
  // and cost a lone one up to 2 us.)

  const int N = p.seqlen;
  const int wl = p.window_left;
  const int wr = eff_window_right(p.causal, p.window_right);

  // Every consuming warp reads the k-th work item (id and geometry, decoded once by the producer) from slot
  // k & 1 once the producer has published it, and releases the slot. -1 ends the walk (also after a give-up).
  auto take_item = [&](uint32_t& n_items, ItemGeom& g) -> int {
    const uint32_t slot = n_items & 1u;
    if (!mbar_wait_warp(&item_full[slot], (n_items >> 1) & 1u, abort_flag)) return -1;
    const volatile int* w = s_geom + slot * 16;
    const int it = w[12];
    g.bh = w[0]; g.pair = w[1];
    g.r0[0] = w[2]; g.r0[1] = w[3]; g.r1[0] = w[4]; g.r1[1] = w[5];
    g.lo[0] = w[6]; g.lo[1] = w[7]; g.hi[0] = w[8]; g.hi[1] = w[9];
    g.top = w[10]; g.steps = w[11]; g.split = w[13];
    __syncwarp();
    if (lane == 0) mbar_arrive(&item_empty[slot]);
    ++n_items;
    return it;
  };

  if (warp < 8) {
    // =====================================================================================
    // softmax: stage s = warp / 4, row = tid % 128
    // =====================================================================================
    reg_inc<kShort ? Cfg::kRegSoftmaxShort : Cfg::kRegSoftmax>();
    const int s = warp >> 2;
    const int row_l = tid & 127;
    const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
    const uint32_t tS = tmem_addr(tmem_base, lane_base, s == 0 ? Cfg::kColS0 : Cfg::kColS1);
    // With ALiBi the scores are moved to the biased log2 domain right after the TMEM load, and
    // everything downstream works with a unit scale.
    const float sl2 = kAlibi ? 1.f : p.scale_log2;
    const uint64_t scale2 = f2_pack(sl2, sl2);
    const uint32_t tO = tmem_addr(tmem_base, lane_base, s == 0 ? Cfg::kColO0 : Cfg::kColO1);
    const uint32_t tP = tS + (kOwnP ? Cfg::kOwnPFromS : 0);
    uint32_t par_s = 0;  // parity of the next s_full phase
    griddep_wait();
    const float lazy = Cfg::kLazyLog2 / sl2;
    uint32_t n_items = 0;
    uint32_t par_e = 1;  // parity of the o_empty phase of this stage's previous item
    uint4* drop_blocks = reinterpret_cast<uint4*>(sAlpha + warp * 32);
    bool after_split = false;
    bool ok = true;
    while (ok) {
      ItemGeom g;
      const int item = take_item(n_items, g);
      if (item < 0) break;
      const int q_r0 = s ? g.r0[1] : g.r0[0];
      const int q_r1 = s ? g.r1[1] : g.r1[0];
      const int j_lo = s ? g.lo[1] : g.lo[0];
      const int j_hi = s ? g.hi[1] : g.hi[0];
      if (q_r1 < q_r0) continue;
      const int row = q_r0 + row_l;
      DropRow drow = {0u, 0u};
      if (kDropout) {
        drow = drop_row(p, g.bh, row);
        // (the references of a split item lie where this warp's drop_blocks do)
        if (after_split && !mbar_wait_warp(&o_empty[s], par_e, abort_flag)) break;
        after_split = g.split;
      }
      float slope_l2 = 0.f;
      if (kAlibi) slope_l2 = p.alibi_slopes[g.bh % p.heads] * 1.4426950408889634f;
      float m_used = 0.f;  // the row's reference: the score that its exponentials are taken against
      float m_limit = -INFINITY;  // a tile max above this moves the reference
      float l_run = 0.f;   // 0 until the row has seen a finite score, at least about 1 from then on
      const int kv_step = g.split ? 2 * kBlockN : kBlockN;
      int kv0 = (g.split ? g.top - 2 * j_lo - s : g.top - j_lo) * kBlockN;
      const int kv_end = kv0 - (j_hi - j_lo) * kv_step, kv_first = kv0;
      // Tiles with kv_a <= kv0 <= kv_b are not cut (see kv_tile_needs_mask).
      const int kv_a = wl >= 0 ? q_r1 - wl : 0;
      const int kv_b = wr >= 0 ? min(N, q_r0 + wr + 1) - kBlockN : N - kBlockN;
      for (; kv0 != kv_end && ok; kv0 -= kv_step) {
        ok = mbar_wait(&s_full[s], par_s, abort_flag);
        par_s ^= 1u;
        tc_fence_after();
        // One body, instantiated twice: tiles cut by a mask boundary (or by the end of the sequence) take the
        // per-element predicate, all others carry none of that code. (Blanking a cut tile in tensor memory first
        // and sharing one body, as the short build does, makes every tile 3-6 % slower: the body then starts behind a
        // merge point instead of directly behind the wait.)
        // Visible columns of this row: c_lo <= c <= c_hi, i.e. |c - mid| <= half. The predicate is applied on the
        // FMA pipe, which the softmax leaves nearly idle, instead of as two integer compares and a select per
        // element: t = saturate(|c - mid| - half) is 0 for a visible column and 1 for a hidden one (both
        // operands are multiples of 1/2, so the difference is exact), and sc - 3e38 * t leaves a visible
        // score bit for bit as it is and puts a hidden one near -3e38, where its exponential is 0 for any scale the
        // host accepts.
        auto visible_columns = [&](float& mid, float& half) {
          const int c_lo = (wl >= 0) ? row - wl - kv0 : -(1 << 20);
          int c_hi = N - 1 - kv0;
          if (wr >= 0) c_hi = min(c_hi, row + wr - kv0);
          mid = 0.5f * static_cast<float>(c_lo + c_hi);
          half = 0.5f * static_cast<float>(c_hi - c_lo);  // negative: no visible column at all
        };
        auto hide = [](float score, float c, float mid, float half) {
          return fmaf(__saturatef(fabsf(c - mid) - half), -3.0e38f, score);
        };
        auto blank_hidden = [&]() {
          float mid, half;
          visible_columns(mid, half);
#pragma unroll 1
          for (int c0 = 0; c0 < kBlockN; c0 += 32) {
            uint32_t r[32];
            tmem_ld32(tS + c0, r);
            tmem_wait_ld();
            tmem_ld_fence(r);
            const float m0 = mid - static_cast<float>(c0);
#pragma unroll
            for (int c = 0; c < 32; ++c)
              r[c] = __float_as_uint(hide(__uint_as_float(r[c]), static_cast<float>(c), m0, half));
            tmem_st32(tS + c0, r);
          }
          tmem_wait_st();
        };
        // O of this warp's rows times the rows' factors. s_full for this tile was committed behind the previous tile's P.V
        // (kOwnP: behind its first 96 keys), so O is at rest.
        // It has to be done before P is handed over, and the short build does it last, with 96 keys' scores gone from the
        // registers: 64 columns a turn instead of 16, one or two waits instead of four or eight. A warp moves a row in
        // every few tiles where scores spread widely. us before -> after, scores of spread 1 / 4: B4 H16 N2048 d64 causal
        // 62.9 -> 62.2 / 68.1 -> 63.5, B8 H12 N1000 d64 45.2 -> 44.6 / 50.2 -> 45.6, d128 61.7 -> 61.6 / 69.1 -> 63.2, with
        // log-sum-exp 46.9 -> 45.4 / 49.7 -> 45.7, window 512 B4 H16 N8192 d64 154.9 -> 154.3 / 164.9 -> 155.2. In the
        // long build the factor is a register too many through the exponentials: B2 H16 N4096 d128 241 -> 248 / 277 -> 269,
        // and 32 columns a turn at the old place spill (252 / 284); dropout 84.8 -> 86.3 / 87.8 -> 87.8.
        auto rescale_o = [&](float alpha) {
          constexpr int kW = kLateO ? 64 : 16;  // columns at a time
          if (kOwnP) {
            ok &= mbar_wait(&p_empty[s], par_s, abort_flag);
            tc_fence_after();
          }
#pragma unroll 1
          for (int c = 0; c < D; c += kW) {
            uint32_t r[kW / 16][16];
#pragma unroll
            for (int x = 0; x < kW / 16; ++x) tmem_ld16(tO + c + x * 16, r[x]);
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < kW / 16; ++x) {
              tmem_ld_fence16(r[x]);
#pragma unroll
              for (int i = 0; i < 16; ++i) r[x][i] = __float_as_uint(__uint_as_float(r[x][i]) * alpha);
              tmem_st16(tO + c + x * 16, r[x]);
            }
          }
        };
        auto tile_body = [&](auto masked_tag) {
          constexpr bool kMasked = decltype(masked_tag)::value;
          constexpr bool kPoly = !kMasked && !kDropout && !(kShort && D == 128);
          if (kDropout) {
            if (lane < 8) drop_blocks[lane] = drop_block(p, g.bh, static_cast<uint32_t>(kv0 / 16 + lane));
            __syncwarp();
          }
          uint32_t r0[32], r1[32], r2[32], r3[32];
          tmem_ld32(tS + 0, r0);
          tmem_ld32(tS + 32, r1);
          tmem_ld32(tS + 64, r2);
          tmem_ld32(tS + 96, r3);
          tmem_wait_ld();
          tmem_ld_fence(r0);
          tmem_ld_fence(r1);
          tmem_ld_fence(r2);
          tmem_ld_fence(r3);
          float sc[kBlockN];
  #pragma unroll
          for (int i = 0; i < 32; ++i) {
            sc[i] = __uint_as_float(r0[i]);
            sc[32 + i] = __uint_as_float(r1[i]);
            sc[64 + i] = __uint_as_float(r2[i]);
            sc[96 + i] = __uint_as_float(r3[i]);
          }
          if (kAlibi) {  // s * scale - slope * |i - j|, in log2 units (reference: src/mask.h:21-26, src/main.cu:200-207)
            const float rel = static_cast<float>(row - kv0);
            if (kMasked) {
  #pragma unroll
              for (int c = 0; c < kBlockN; ++c)
                sc[c] = fmaf(sc[c], p.scale_log2, -slope_l2 * fabsf(rel - static_cast<float>(c)));
            } else {
              // All keys of the tile lie on one side of all rows, so the bias is linear in the column and costs one
              // scalar FMA and half a two-wide one per element instead of a subtraction, a product and an FMA:
              // B2 H16 N4096 causal, d64 177.5 -> 159 us, d128 199 -> 171 (without ALiBi d64 runs in 133.5). Folding
              // the bias into the exponent's FMA with a bound in place of the max was no faster on these (156, 173)
              // and slower without a mask (292 -> 331).
              const uint64_t biasscale2 = f2_pack(p.scale_log2, p.scale_log2);
              const float step = rel > 0.f ? slope_l2 : -slope_l2;
              const float base = -slope_l2 * fabsf(rel);
  #pragma unroll
              for (int c = 0; c < kBlockN; c += 2) {
                const float b0 = fmaf(step, static_cast<float>(c), base), b1 = fmaf(step, static_cast<float>(c + 1), base);
                f2_unpack(f2_fma(f2_pack(sc[c], sc[c + 1]), biasscale2, f2_pack(b0, b1)), sc[c], sc[c + 1]);
              }
            }
          }
          if (kMasked) {
            float mid, half;
            visible_columns(mid, half);
  #pragma unroll
            for (int c = 0; c < kBlockN; ++c) sc[c] = hide(sc[c], static_cast<float>(c), mid, half);
          }
          // The exponentials of the first 32 keys are taken against the reference the previous tile left while
          // the row max of this tile is still being reduced: nearly always the reference stays where it is (lazy
          // rescale), so the max leaves the critical path. When a row of the warp does move its reference
          // (always on the first tile of an item), the 32 exponentials are taken again. Cut tiles do not
          // speculate: most of them are the first tile of their walk.
          uint64_t lsum_a = 0ull, lsum_b = 0ull;
          uint32_t pk0[32];
          if (!kMasked && !kShort) {
            const float neg_ms0 = -m_used * sl2;
            exp_tile<16, 0>(sc, scale2, f2_pack(neg_ms0, neg_ms0), pk0, lsum_a, lsum_b);
          }
          float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
  #pragma unroll
          for (int c = 0; c < kBlockN; c += 8) {
            mx0 = max3(mx0, sc[c], sc[c + 1]);
            mx1 = max3(mx1, sc[c + 2], sc[c + 3]);
            mx2 = max3(mx2, sc[c + 4], sc[c + 5]);
            mx3 = max3(mx3, sc[c + 6], sc[c + 7]);
          }
          float m_new = max3(mx0, mx1, fmaxf(mx2, mx3));
          if ((kMasked || kShort) && m_new < -1.0e37f) m_new = -INFINITY;  // nothing visible (hidden scores sit near -3e38)
          // The reference moves when the tile's max has grown past it (see kLazyLog2), and always on the first tile that
          // shows a finite score: the reference then IS the row max, so the largest term of the row is exactly 1 in
          // fp16 (a row with a single visible key returns that key's V bit for bit). A cut tile over the first keys is
          // the only tile of its walk (with ALiBi it may be the last), or the far edge of a left window lies in it.
          const bool first_keys = (!kMasked || kAlibi) && kv0 == 0;
          float alpha_o = 1.f;  // kLateO: the factor for this row's O
          if (__any_sync(0xffffffffu, m_new > (first_keys ? fminf(m_used, m_limit) : m_limit))) {
            const bool fresh = l_run == 0.f;
            float alpha = 1.f;
            if (fresh || m_new > m_used) {
              const float m_next = (m_new == -INFINITY) ? 0.f : m_new;
              alpha = fresh ? 1.f : ex2_approx((m_used - m_next) * sl2);
              m_used = m_next;
            }
            m_limit = l_run == 0.f && m_new == -INFINITY ? -INFINITY : m_used + lazy;
            l_run *= alpha;
            if (kLateO) alpha_o = kv0 == kv_first ? 1.f : alpha;
            else if (kv0 != kv_first && __any_sync(0xffffffffu, alpha != 1.f)) rescale_o(alpha);
            if (!kMasked && !kShort) {
              lsum_a = 0ull;
              lsum_b = 0ull;
              const float neg_ms1 = -m_used * sl2;
              exp_tile<16, 0>(sc, scale2, f2_pack(neg_ms1, neg_ms1), pk0, lsum_a, lsum_b);
            }
          }
          if (kMasked || kShort) {
            const float neg_ms1 = -m_used * sl2;
            exp_tile<16, 0>(sc, scale2, f2_pack(neg_ms1, neg_ms1), pk0, lsum_a, lsum_b);
          }
          const float neg_ms = -m_used * sl2;
          const uint64_t negms2 = f2_pack(neg_ms, neg_ms);
          exp_tile<16, kPoly ? Cfg::kPolyOf1 : 0>(sc + 32, scale2, negms2, pk0 + 16, lsum_a, lsum_b);
          if (kDropout) dropout_mask<4>(pk0, p, drow, drop_blocks);  // the row sum keeps every exponential
          tmem_st32(tP + 0, pk0);  // (kOwnP: s_full says that the previous tile's first 96 keys have been read)
          uint32_t pk1[16], pk2[16];
          exp_tile<16, kPoly ? Cfg::kPolyOf2 : 0>(sc + 64, scale2, negms2, pk1, lsum_a, lsum_b);
          if (kDropout) dropout_mask<2>(pk1, p, drow, drop_blocks + 4);
          tmem_st16(tP + 32, pk1);
          if (kLateO && __any_sync(0xffffffffu, alpha_o != 1.f)) rescale_o(alpha_o);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          mbar_arrive_lane0(&p_full[s], lane);  // P of keys 0..95 is in TMEM
          exp_tile<16, kPoly ? Cfg::kPolyOf3 : 0>(sc + 96, scale2, negms2, pk2, lsum_a, lsum_b);
          if (kDropout) dropout_mask<2>(pk2, p, drow, drop_blocks + 6);
          if (kOwnP) {
            ok &= mbar_wait(&p_empty[s], par_s, abort_flag);
            tc_fence_after();
          }
          tmem_st16(tP + 48, pk2);
          float l0, l1;
          f2_unpack(f2_add(lsum_a, lsum_b), l0, l1);
          l_run += l0 + l1;
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          mbar_arrive_lane0(&p_full2[s], lane);  // P of keys 96..127
        };
        const bool cut = kv0 < kv_a || kv0 > kv_b;
        if (kShort) {
          if (cut) blank_hidden();
          tile_body(std::false_type{});
        } else if (cut || (kAlibi && kv0 + kBlockN - 1 > q_r0 && kv0 < q_r1)) {
          // (ALiBi: a tile that the diagonal crosses takes the cut tiles' body, whose bias has the absolute value)
          tile_body(std::true_type{});
        } else {
          tile_body(std::false_type{});
        }
        ok = __all_sync(0xffffffffu, ok);
      }
      if (!ok) break;
      // the epilogue warps have read the row sums of the previous item
      if (!mbar_wait_warp(&o_empty[s], par_e, abort_flag)) break;
      par_e ^= 1u;
      sRowSum[s * kBlockM + row_l] = l_run;
      // a split item's epilogue also needs the reference the sums are taken against
      if (g.split) sAlpha[s * kBlockM + row_l] = m_used * sl2;
      __syncwarp();
      if (lane == 0) mbar_arrive(&l_ready[s]);
      // l_run = sum over visible keys of 2^((score - m_used) * sl2), so the natural-log sum of exponentials is
      // ln2 * (m_used * sl2 + log2(l_run)).
      if (kLse && !g.split && row < N)
        p.lse[static_cast<size_t>(g.bh) * N + row] =
            (l_run > 0.f) ? 0.6931471805599453f * fmaf(m_used, sl2, __log2f(l_run)) : -INFINITY;
    }
  } else if (warp < 12) {
    // =====================================================================================
    // epilogue: row = tid % 128 of both stages
    // =====================================================================================
    reg_dec<kShort ? Cfg::kRegEpilogueShort : Cfg::kRegEpilogue>();
    griddep_wait();
    const int row_l = tid & 127;
    const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
    uint8_t* out_stage = smem + Cfg::kOffOut + (warp & 3) * Cfg::kOutWarpBytes;
    // Columns 8u .. 8u+7 of the lane's row are 16-byte unit u%8 of panel u/8; unit x of row r sits at x ^ (r%8).
    auto out_row = [&](int u) { return out_stage + (u >> 3) * (32 * 128) + lane * 128 + ((u & 7) ^ (lane & 7)) * 16; };
    constexpr int kCols = kShort ? 16 : Cfg::kEpilogueCols;
    // Bit s: phase parity of stage s's barriers. The stages share one copy of this code (rolled loops, state in bit
    // masks): with copies for both and the epilogue in four places it was 38 KB, mostly run from cold instructions.
    uint32_t par_l = 0, par_o = 0;
    uint32_t n_items = 0;
    bool ok = true;
    while (ok) {
      ItemGeom g;
      const int item = take_item(n_items, g);
      if (item < 0) break;
      // O / l -> fp16 -> global for stage s, then the next item's first product may overwrite O
      auto epilogue = [&](int s) {
        if (!mbar_wait_warp(&l_ready[s], (par_l >> s) & 1, abort_flag)) { ok = false; return; }
        par_l ^= 1u << s;
        const float l = sRowSum[s * kBlockM + row_l];
        if (!mbar_wait_warp(&o_full[s], (par_o >> s) & 1, abort_flag)) { ok = false; return; }
        par_o ^= 1u << s;
        tc_fence_after();
        const float inv_l = ((l > 0.f) ? 1.f / l : 0.f) * (kDropout ? p.drop_scale : 1.f);
        const uint32_t tO = tmem_addr(tmem_base, lane_base, s == 0 ? Cfg::kColO0 : Cfg::kColO1);
        // The rows go to the warp's staging area and from there to global memory as one TMA store: issued as plain
        // stores (each lane its own row, 16 bytes at a time) they kept the load/store unit busy for about 2000
        // clocks per tile, and the barrier traffic of every other warp of the SM queued behind them.
        if (lane == 0) tma_store_wait_read();  // the previous store of this warp has read the staging area
        __syncwarp();
        // kCols columns at a time, the load of the next chunk in flight while this one is converted and stored.
        // (Rolled up: this path runs once per item and stage, and instructions that are rarely executed are
        // fetched slowly; unrolling it eightfold made the change-over between items slower, not faster.)
        uint32_t ra[kCols], rb[kCols];
        tmem_ld_cols(tO, ra);
  #pragma unroll 2
        for (int c = 0; c < D / kCols; ++c) {
          uint32_t (&cur)[kCols] = (c & 1) ? rb : ra;
          uint32_t (&nxt)[kCols] = (c & 1) ? ra : rb;
          tmem_wait_ld();
          tmem_ld_fence_cols(cur);
          if (c + 1 < D / kCols) tmem_ld_cols(tO + (c + 1) * kCols, nxt);
#pragma unroll
          for (int i = 0; i < kCols / 8; ++i) {
            uint4 v;
            v.x = pack_f16x2(__uint_as_float(cur[i * 8 + 0]) * inv_l, __uint_as_float(cur[i * 8 + 1]) * inv_l);
            v.y = pack_f16x2(__uint_as_float(cur[i * 8 + 2]) * inv_l, __uint_as_float(cur[i * 8 + 3]) * inv_l);
            v.z = pack_f16x2(__uint_as_float(cur[i * 8 + 4]) * inv_l, __uint_as_float(cur[i * 8 + 5]) * inv_l);
            v.w = pack_f16x2(__uint_as_float(cur[i * 8 + 6]) * inv_l, __uint_as_float(cur[i * 8 + 7]) * inv_l);
            *reinterpret_cast<uint4*>(out_row(c * (kCols / 8) + i)) = v;
          }
        }
        fence_proxy_async_smem();
        // O of this stage has been read: let the next item's first product overwrite it
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          const int row0 = (s ? g.r0[1] : g.r0[0]) + static_cast<int>(lane_base);
          if (row0 < N) {  // rows of the box beyond the sequence are clipped by the store
            tma_store_4d(&mapO, out_stage, 0, row0, 0, g.bh);
            tma_store_commit();
          }
          mbar_arrive(&o_empty[s]);
        }
      };
      // Split item: O = (O_0 2^(m_0 - m) + O_1 2^(m_1 - m)) / (l_0 2^(m_0 - m) + l_1 2^(m_1 - m)), m the larger of the
      // two stages' references; then as above.
      auto epilogue_split = [&]() {
        float l[2], m[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (!mbar_wait_warp(&l_ready[s], (par_l >> s) & 1, abort_flag)) { ok = false; return; }
          l[s] = sRowSum[s * kBlockM + row_l];
          m[s] = l[s] > 0.f ? sAlpha[s * kBlockM + row_l] : -INFINITY;
          if (!mbar_wait_warp(&o_full[s], (par_o >> s) & 1, abort_flag)) { ok = false; return; }
        }
        par_l ^= 3u;
        par_o ^= 3u;
        tc_fence_after();
        const float m_all = fmaxf(fmaxf(m[0], m[1]), -3.0e38f);  // (a row without visible keys: both factors are 0)
        float f0 = ex2_approx(m[0] - m_all), f1 = ex2_approx(m[1] - m_all);
        const float l_all = l[0] * f0 + l[1] * f1;
        const float inv_l = ((l_all > 0.f) ? 1.f / l_all : 0.f) * (kDropout ? p.drop_scale : 1.f);
        f0 *= inv_l;
        f1 *= inv_l;
        const int row0 = g.r0[0] + static_cast<int>(lane_base);
        if (kLse && row0 + lane < N)
          p.lse[static_cast<size_t>(g.bh) * N + row0 + lane] =
              (l_all > 0.f) ? 0.6931471805599453f * (m_all + __log2f(l_all)) : -INFINITY;
        const uint32_t tO0 = tmem_addr(tmem_base, lane_base, Cfg::kColO0);
        const uint32_t tO1 = tmem_addr(tmem_base, lane_base, Cfg::kColO1);
        if (lane == 0) tma_store_wait_read();
        __syncwarp();
#pragma unroll 1
        for (int c = 0; c < D / kCols; ++c) {
          uint32_t ra[kCols], rb[kCols];
          tmem_ld_cols(tO0 + c * kCols, ra);
          tmem_ld_cols(tO1 + c * kCols, rb);
          tmem_wait_ld();
          tmem_ld_fence_cols(ra);
          tmem_ld_fence_cols(rb);
#pragma unroll
          for (int i = 0; i < kCols / 8; ++i) {
            uint32_t v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int e = i * 8 + 2 * k;
              v[k] = pack_f16x2(fmaf(__uint_as_float(ra[e]), f0, __uint_as_float(rb[e]) * f1),
                                fmaf(__uint_as_float(ra[e + 1]), f0, __uint_as_float(rb[e + 1]) * f1));
            }
            *reinterpret_cast<uint4*>(out_row(c * (kCols / 8) + i)) = make_uint4(v[0], v[1], v[2], v[3]);
          }
        }
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (row0 < N) {
            tma_store_4d(&mapO, out_stage, 0, row0, 0, g.bh);
            tma_store_commit();
          }
          mbar_arrive(&o_empty[0]);
          mbar_arrive(&o_empty[1]);
        }
      };
      if (g.split) {
        epilogue_split();
      } else {
        // the stage that runs out of tiles first is finished first
        const int first = g.hi[1] < g.hi[0] ? 1 : 0;
#pragma unroll 1
        for (int k = 0; k < 2 && ok; ++k) {
          const int s = first ^ k;
          if ((s ? g.r1[1] : g.r1[0]) >= (s ? g.r0[1] : g.r0[0])) epilogue(s);
        }
      }
    }
    if (lane == 0) tma_store_wait_read();  // also on the give-up path: stores in flight read this CTA's shared memory
  } else {
    reg_dec<Cfg::kRegOthers>();
    if (warp == 12) {
      // ===================================================================================
      // tensor-core issuer. The whole warp walks the schedule and waits, so that addresses and
      // descriptors are warp-uniform values; one elected lane issues the tcgen05 instructions. The
      // verdicts of the waits are gathered and looked at once per round: products issued behind a wait
      // that gave up stay inside the CTA's own memory, and the round's results are discarded.
      // ===================================================================================
      constexpr uint32_t idesc_qk = umma_idesc_f16(kBlockM, kBlockN, 0, 0);
      constexpr uint32_t idesc_pv = umma_idesc_f16(kBlockM, D, 0, 1);
      // Descriptors are built once; per instruction only the 16-byte-unit start address moves.
      const uint32_t kdesc0 = static_cast<uint32_t>(umma_desc_sw128(0, 16, 1024));  // K-major tiles (Q, K), low word
      const uint32_t vdesc0 = static_cast<uint32_t>(umma_desc_sw128(0, Cfg::kPanelBytes, 1024));  // MN-major tile (V)
      constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // row stride, version, 128-byte swizzle
      const uint32_t q_addr = smem_u32(sQ);
      const uint32_t kv_addr = smem_u32(sKV);
      const uint32_t qdesc[2] = {kdesc0 + (q_addr >> 4), kdesc0 + ((q_addr + Cfg::kTileBytes) >> 4)};
      uint32_t pos = 0;               // ring position (tiles since the start) of the first K tile of the current item
      uint32_t par_p = 0, par_q = 0, par_e = 3;  // bit s: phase parity of stage s's barriers
      uint32_t n_items = 0;
      bool ok = true;
      griddep_wait();
      // (Every published item has rows, so the loop ends on its first pass. Written without it the compiler's code for the
      // rounds ran 3 % slower at head_dim 64: B8 H12 N1000 48.7 -> 50.0 us, B4 H16 N2048 causal 64.7 -> 67.1.)
      auto take_nonempty = [&](ItemGeom& g) {
        while (take_item(n_items, g) >= 0)
          if (g.steps > 0) return true;
        g.steps = g.split = g.lo[0] = g.lo[1] = g.hi[0] = g.hi[1] = 0;
        return false;
      };
      // Head_dim 64: the round between two items issues the last P.V of item `a`, whose tiles end at ring position `end`,
      // and behind each stage's the first score tile of item `b`, so that a stage's softmax goes on while the other
      // stage's last tile is still under way. Either may be missing (no steps). B200, us: B8 H12 N1000 50.6 -> 49.3,
      // 32 heads of 8192 rows 748 -> 737 without a mask, ALiBi B2 H16 N4096 133.0 -> 131.3, B4 H16 N2048 causal
      // 65.2 -> 64.7. At head_dim 128 long sequences do not change and B8 H16 N1024 causal loses 2.6 %, so there an
      // item's rounds end before the next item's begin.
      constexpr bool kJoin = D == 64;
      auto join = [&](const ItemGeom& a, const ItemGeom& b, uint32_t end) {
        const int j = a.steps - 1;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int alo = s ? a.lo[1] : a.lo[0], ahi = s ? a.hi[1] : a.hi[0];
          const int blo = s ? b.lo[1] : b.lo[0], bhi = s ? b.hi[1] : b.hi[0];
          const uint32_t tS = tmem_base + (s ? Cfg::kColS1 : Cfg::kColS0);
          const uint32_t tP = tS + (kOwnP ? Cfg::kOwnPFromS : 0);
          auto rest_of_pv = [&](uint32_t tO, uint32_t slot, uint32_t vdesc) {
            ok &= mbar_wait(&p_full2[s], (par_p >> s) & 1, abort_flag);
            par_p ^= 1u << s;
            tc_fence_after();
            umma_pv32(tO, tP + 48, vdesc + 6 * (2048 >> 4), kDescHi, idesc_pv);
            umma_commit_warp(&kv_empty[slot], a.split || s == 1 || j < a.lo[1] || j >= a.hi[1]);
            if (kOwnP) umma_commit_warp(&p_empty[s]);
            umma_commit_warp(&o_full[s]);
          };
          const bool has_pv = j >= alo && j < ahi;
          uint32_t tO = 0, slot_pv = 0, vdesc_pv = 0;
          if (has_pv) {  // O_s += P_s V
            tO = tmem_base + (s ? Cfg::kColO1 : Cfg::kColO0);
            const uint32_t pv = end - ((a.split && s == 0 && j < a.hi[1]) ? 2 : 1);
            slot_pv = pv % Cfg::kStages;
            vdesc_pv = vdesc0 + ((kv_addr + slot_pv * Cfg::kTileBytes) >> 4);
            ok &= mbar_wait(&kv_full[slot_pv], (pv / Cfg::kStages) & 1, abort_flag);
            if (j == alo) {  // the previous item's O has been read
              ok &= mbar_wait(&o_empty[s], (par_e >> s) & 1, abort_flag);
              par_e ^= 1u << s;
            }
            ok &= mbar_wait(&p_full[s], (par_p >> s) & 1, abort_flag);
            tc_fence_after();
            umma_pv96(tO, tP, vdesc_pv, kDescHi, idesc_pv, j > alo ? 1u : 0u);
            if (!kOwnP) rest_of_pv(tO, slot_pv, vdesc_pv);
          }
          if (blo == 0 && bhi > 0) {  // S_s = Q_s K^T
            const uint32_t pk = end + (b.split ? s : 0);
            const uint32_t slot = pk % Cfg::kStages;
            ok &= mbar_wait(&q_full[s], (par_q >> s) & 1, abort_flag);
            par_q ^= 1u << s;
            ok &= mbar_wait(&kv_full[slot], (pk / Cfg::kStages) & 1, abort_flag);
            tc_fence_after();
            const uint32_t kdesc = kdesc0 + ((kv_addr + slot * Cfg::kTileBytes) >> 4);
            const uint32_t qd = s ? qdesc[1] : qdesc[0];
#pragma unroll
            for (int h = 0; h < D / 64; ++h)
              umma_qk64(tS, qd + h * (Cfg::kPanelBytes >> 4), kdesc + h * (Cfg::kPanelBytes >> 4), kDescHi, idesc_qk, h);
            umma_commit_warp(&s_full[s]);
            umma_commit_warp(&kv_empty[slot], b.split || s == 1 || b.lo[1] > 0 || b.hi[1] == 0);
            umma_commit_warp(&q_empty[s], bhi == 1);
          }
          if (kOwnP && has_pv) rest_of_pv(tO, slot_pv, vdesc_pv);
        }
      };
      ItemGeom g;
      if (kJoin) {
        ItemGeom none;
        none.steps = none.split = none.lo[0] = none.lo[1] = none.hi[0] = none.hi[1] = 0;
        if (take_nonempty(g)) join(none, g, 0);
        ok = __all_sync(0xffffffffu, ok);
      }
      while (ok) {
        if (kJoin ? g.steps == 0 : take_item(n_items, g) < 0) break;
        const int j_first = kJoin ? 0 : -1, j_end = kJoin ? g.steps - 1 : g.steps;
        // Ring positions are carried along instead of recomputed: (slot_v, par_v) is where V_j lives,
        // (slot_k, par_k) where K_{j+1} lives. Rounds in which both stages have a P.V for tile j and a
        // score tile j+1 ("interior", nearly all of a long sequence) take a branch-free body; the first
        // and last rounds of an item take the general one.
        // (split items: slot_k is the next tile in the ring)
        const uint32_t pos0 = pos + 1, pos1 = kJoin ? pos + 2 : pos;
        uint32_t slot_v = pos0 % Cfg::kStages, par_v = (pos0 / Cfg::kStages) & 1;
        uint32_t slot_k = pos1 % Cfg::kStages, par_k = (pos1 / Cfg::kStages) & 1;
        auto advance = [](uint32_t& slot, uint32_t& par, uint32_t n) {
          slot += n;
          if (slot >= static_cast<uint32_t>(Cfg::kStages)) { slot -= Cfg::kStages; par ^= 1u; }
        };
        // interior rounds in_lo <= j < in_hi: for both stages tile j is neither the first (its P.V accumulates)
        // nor among the last two (no Q release, no final commit), and tile j+1 exists
        const int in_lo = max(g.lo[0], g.lo[1]) + 1;
        const int in_hi = min(g.hi[0], g.hi[1]) - 2;
        // In a split item every product has a kv tile of its own: the tiles lie in the ring in the order of their use,
        // and slot_k is the next one.
        auto wait_next_v = [&]() {  // V_{j+1} lies behind K_{j+1}
          uint32_t slot = slot_k, par = par_k;
          advance(slot, par, 1);
          return mbar_wait(&kv_full[slot], par, abort_flag);
        };
        auto round_body = [&](auto interior_tag, auto split_tag, int j) {
          constexpr bool kInterior = decltype(interior_tag)::value;
          constexpr bool kSplit = decltype(split_tag)::value;
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const bool act_j = kInterior || (j >= g.lo[s] && j < g.hi[s]);
            const bool act_n = kInterior || (j + 1 >= g.lo[s] && j + 1 < g.hi[s]);
            const bool other_j = !kSplit && (s == 0) && (kInterior || (j >= g.lo[1] && j < g.hi[1]));          // stage 1 still needs V_j
            const bool other_n = !kSplit && (s == 0) && (kInterior || (j + 1 >= g.lo[1] && j + 1 < g.hi[1]));  // stage 1 still needs K_j+1
            // stage 0 already waited for this tile in the same round
            const bool v_seen = !kSplit && (s == 1) && (kInterior || (j >= g.lo[0] && j < g.hi[0]));
            const bool k_seen = !kSplit && (s == 1) && (kInterior || (j + 1 >= g.lo[0] && j + 1 < g.hi[0]));
            const uint32_t colS = (s == 0) ? Cfg::kColS0 : Cfg::kColS1;
            const uint32_t colO = (s == 0) ? Cfg::kColO0 : Cfg::kColO1;
            const uint32_t colP = colS + (kOwnP ? Cfg::kOwnPFromS : 0);
            auto rest_of_pv = [&](uint32_t slot, uint32_t vdesc) {
              ok &= mbar_wait(&p_full2[s], (par_p >> s) & 1, abort_flag);
              par_p ^= 1u << s;
              tc_fence_after();
              umma_pv32(tmem_base + colO, tmem_base + colP + 48, vdesc + 6 * (2048 >> 4), kDescHi, idesc_pv);
              if (!kInterior || !other_j) umma_commit_warp(&kv_empty[slot], !other_j);
              if (kOwnP) umma_commit_warp(&p_empty[s]);
              if (!kInterior) umma_commit_warp(&o_full[s], j + 1 == g.hi[s]);
            };
            uint32_t slot_pv = 0, vdesc_pv = 0;
            if (act_j) {  // O_s += P_s(j) V_j, 96 keys and 32 as P arrives
              if (kSplit) {
                slot_v = slot_k;
                par_v = par_k;
                advance(slot_k, par_k, 1);
              }
              slot_pv = slot_v;
              vdesc_pv = vdesc0 + ((kv_addr + slot_v * Cfg::kTileBytes) >> 4);
              if (!kInterior && !v_seen) ok &= mbar_wait(&kv_full[slot_v], par_v, abort_flag);
              if (!kInterior && j == g.lo[s]) {  // the previous item's O has been read
                ok &= mbar_wait(&o_empty[s], (par_e >> s) & 1, abort_flag);
                par_e ^= 1u << s;
              }
              ok &= mbar_wait(&p_full[s], (par_p >> s) & 1, abort_flag);
              tc_fence_after();
              umma_pv96(tmem_base + colO, tmem_base + colP, vdesc_pv, kDescHi, idesc_pv, (kInterior || j > g.lo[s]) ? 1u : 0u);
              if (!kOwnP) rest_of_pv(slot_pv, vdesc_pv);
            }
            if (act_n) {  // S_s = Q_s K_{j+1}^T
              if (!kInterior && j + 1 == g.lo[s]) {
                ok &= mbar_wait(&q_full[s], (par_q >> s) & 1, abort_flag);
                par_q ^= 1u << s;
              }
              if (!k_seen) ok &= mbar_wait(&kv_full[slot_k], par_k, abort_flag);
              // Inner rounds wait for V here, one round ahead: every group of instructions then has one wait in front
              // of it, about as long as the tensor pipe has work queued (two waits in a row let it run dry).
              if (kInterior && s == 1) ok &= wait_next_v();
              tc_fence_after();
              const uint32_t kdesc = kdesc0 + ((kv_addr + slot_k * Cfg::kTileBytes) >> 4);
#pragma unroll
              for (int h = 0; h < D / 64; ++h)
                umma_qk64(tmem_base + colS, qdesc[s] + h * (Cfg::kPanelBytes >> 4), kdesc + h * (Cfg::kPanelBytes >> 4), kDescHi, idesc_qk, h);
              umma_commit_warp(&s_full[s]);
              if (!kInterior || !other_n) umma_commit_warp(&kv_empty[slot_k], !other_n);
              if (!kInterior) umma_commit_warp(&q_empty[s], j + 2 == g.hi[s]);
              if (kSplit) advance(slot_k, par_k, 1);
            }
            if (kOwnP && act_j) rest_of_pv(slot_pv, vdesc_pv);
          }
        };
        if (g.split) {
          for (int j = j_first; j < j_end && ok; ++j) {
            round_body(std::false_type{}, std::true_type{}, j);
            ok = __all_sync(0xffffffffu, ok);
          }
          pos += 2u * static_cast<uint32_t>(g.hi[0] + g.hi[1]);
        } else {
          for (int j = j_first; j < j_end && ok; ++j) {
            if (!kShort && j == in_lo && in_lo < in_hi) ok &= mbar_wait(&kv_full[slot_v], par_v, abort_flag);
            if (!kShort && j >= in_lo && j < in_hi) round_body(std::true_type{}, std::false_type{}, j);
            else round_body(std::false_type{}, std::false_type{}, j);
            // V_{j+1} sits right after K_{j+1}; K_{j+2} two positions after K_{j+1}
            slot_v = slot_k;
            par_v = par_k;
            advance(slot_v, par_v, 1);
            advance(slot_k, par_k, 2);
            ok = __all_sync(0xffffffffu, ok);
          }
          pos += 2u * static_cast<uint32_t>(g.steps);
        }
        if (!ok) break;
        if (kJoin) {
          ItemGeom nx;
          take_nonempty(nx);
          join(g, nx, pos);
          ok = __all_sync(0xffffffffu, ok);
          g = nx;
        }
      }
      if (!ok) {
        // give-up path: let products that are still in flight end before the CTA retires
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
      }
    } else if (warp == 14 && lane == 0) {
      // Q of the CTA's first item, beside the producer's first K/V tiles
      griddep_wait();
      if (g_first.steps > 0) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (g_first.r1[s] < g_first.r0[s]) continue;
          mbar_arrive_expect_tx(&q_full[s], Cfg::kTileBytes);
          tma_load_4d(sQ + s * Cfg::kTileBytes, &mapQ, &q_full[s], 0, g_first.r0[s], 0, g_first.bh);
        }
      }
    } else if (warp == 13 && lane == 0) {
      // ===================================================================================
      // TMA producer
      // ===================================================================================
      uint32_t it = 0;
      uint32_t n_q[2] = {0, 0};
      uint32_t n_pub = 0;
      bool ok = true;
      bool first = g_first.steps > 0;
      // The first item was decoded in front of the CTA's first barrier. (It may be without rows: then it is none.)
      ItemGeom g = g_first;
      int item = -1, claimed = -1;
      if (g.steps > 0) {
        mbar_arrive(&item_full[0]);
        n_pub = 1;
        item = static_cast<int>(blockIdx.x);
      }
      griddep_wait();
      if (p.status_per_launch && blockIdx.x == 0) {  // (a wait that gives up sets the status much later than this)
        *p.status = 0;
        p.sched[p.clear_at] = 0;
        p.sched[p.clear_at + 1] = 0;
      }
      while (ok) {
        if (item < 0) {
          const int next = static_cast<int>(gridDim.x) + (claimed >= 0 ? claimed : atomicAdd(p.sched, 1));
          item = next_item(next, p, g, [&] { return static_cast<int>(gridDim.x) + atomicAdd(p.sched, 1); });
          if (item < 0) griddep_launch();  // no further item
          const uint32_t slot = n_pub & 1u;
          if (!mbar_wait(&item_empty[slot], ((n_pub >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
          write_item(slot, g, item);
          mbar_arrive(&item_full[slot]);
          ++n_pub;
          if (item < 0) break;
        }
        auto load_q = [&](int s) {
          if (g.r1[s] < g.r0[s]) return;
          if (n_q[s] > 0 && !mbar_wait(&q_empty[s], (n_q[s] & 1) ^ 1, abort_flag)) ok = false;
          if (!ok) return;
          ++n_q[s];
          mbar_arrive_expect_tx(&q_full[s], Cfg::kTileBytes);
          tma_load_4d(sQ + s * Cfg::kTileBytes, &mapQ, &q_full[s], 0, g.r0[s], 0, g.bh);
        };
        auto load_tile = [&](const CUtensorMap* map, int tile) {
          const uint32_t slot = it % Cfg::kStages;
          if (it >= static_cast<uint32_t>(Cfg::kStages) &&
              !mbar_wait(&kv_empty[slot], ((it / Cfg::kStages) & 1) ^ 1, abort_flag))
            ok = false;
          if (!ok) return;
#ifdef FA_TEST_WITHHOLD_LOAD  // test build only: CTA 0 never loads its fourth tile, so that a bounded wait runs out
          if (blockIdx.x == 0 && (p.variant & 2) != 0 && it == 3) {
            ++it;
            return;
          }
#endif
          mbar_arrive_expect_tx(&kv_full[slot], Cfg::kTileBytes);
          tma_load_4d(sKV + slot * Cfg::kTileBytes, map, &kv_full[slot], 0, tile * kBlockN, 0, g.bh);
          ++it;
        };
        // The Q tiles of the previous item are released one after the other, stage 0 first; the ring slots of the
        // first kv tiles usually before either.
        load_tile(&mapK, g.top);
        if (it == 1 && first) {  // (warp 14 loads the first item's)
          for (int s = 0; s < 2; ++s) n_q[s] += g.r1[s] >= g.r0[s] ? 1 : 0;
        } else {
          load_q(0);
          load_q(1);
        }
        first = false;
        // Claim the following item; the answer is looked at behind this item's loads.
        claimed = atomicAdd(p.sched, 1);
        // One item per CTA: the next kernel of the stream may take up the free SMs at once.
        if (p.num_items <= static_cast<int>(gridDim.x)) griddep_launch();
        if (g.split) {  // in the order of use
          load_tile(&mapK, g.top - 1);
          for (int j = 0; j < g.steps && ok; ++j) {
#pragma unroll 1
            for (int s = 0; s < 2; ++s) {
              const int hi = s ? g.hi[1] : g.hi[0], tile = g.top - 2 * j - s;
              if (j < hi) load_tile(&mapV, tile);
              if (j + 1 < hi) load_tile(&mapK, tile - 2);
            }
          }
        } else {
          for (int j = 0; j < g.steps && ok; ++j) {
            load_tile(&mapV, g.top - j);
            if (j + 1 < g.steps) load_tile(&mapK, g.top - j - 1);
          }
        }
        item = -1;
      }
      // This CTA claims no more: the last one to come here puts the scheduler words back to zero for the next launch.
      if (atomicAdd(p.sched + 1, 1) + 1 == static_cast<int>(gridDim.x)) {
        p.sched[0] = 0;
        p.sched[1] = 0;
      }
      if (!ok) {
        // Give-up path: let loads that are still in flight land before the CTA retires. (Where only the issuer gives up, it
        // sleeps as long. A look at the flag here costs long rows with the log-sum-exp 2 %.)
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_flag != 0) atomicExch(p.status, 1);
  if (warp == 12) tmem_dealloc(tmem_base, Cfg::kTmemCols);
}

}  // namespace fa
