// Warp-specialised persistent attention-forward kernel for sm_100a.
//
// One CTA per SM walks a list of work items (work_items.h); a work item is a pair of adjacent 128-row q tiles of one
// (batch, head), one for each of the two stages, or a single q tile whose kv tiles the stages take in turn. The kv
// tiles are walked from the last visible one to the first. Roles (16 warps):
//   warps 0-3   softmax of stage 0: one thread per score row (TMEM lane), exp2 online softmax
//   warps 4-7   softmax of stage 1
//   warps 8-11  correction: rescales the running output in TMEM when a row max moved, and the
//               epilogue (O / l, or for a single q tile the sum of both stages' O over the sum of their l, -> fp16 ->
//               the warp's staging area in shared memory -> one TMA store)
//   warp 12     tensor-core issuer: the warp walks the schedule, one elected lane issues tcgen05.mma
//   warp 13     TMA producer: Q tiles and the K/V tile ring
//   warps 14-15 idle (they only donate registers)
// TMEM columns: S0 [0,128) S1 [128,256) O0 [256,256+D) O1 [384,384+D); the fp16 P tile of a
// stage overwrites the first 64 columns of its own S and is handed to the tensor pipe in two
// halves of 64 keys, so that P.V starts while the second half is still being exponentiated.
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

// Registers per thread after setmaxnreg: 8 softmax warps, 4 correction warps, 4 others; the three
// numbers must satisfy 256 * softmax + 128 * correction + 128 * others <= 65536.
#ifndef FA_REG_SOFTMAX
#define FA_REG_SOFTMAX 184
#define FA_REG_CORR 72
#define FA_REG_MISC 72
#endif



namespace fa {

template <int D>
struct PersistentCfg {
  static constexpr int kThreads = 512;
  static constexpr int kTileBytes = kBlockN * D * 2;
  static constexpr int kPanelBytes = kBlockN * kPanel * 2;
  static constexpr int kStages = (D == 128) ? 4 : 8;  // ring slots, each one K or one V tile
  static constexpr int kOffQ = 0;
  static constexpr int kOffKV = 2 * kTileBytes;
  // Output staging: each correction warp owns 32 rows, laid out [panel][row][64] with the 128-byte swizzle, the
  // source of its TMA store.
  static constexpr int kOffOut = kOffKV + kStages * kTileBytes;
  static constexpr int kOutWarpBytes = 32 * D * 2;
  static constexpr int kOffAlpha = kOffOut + 4 * kOutWarpBytes;  // float[2][128]
  static constexpr int kOffRowSum = kOffAlpha + 2 * kBlockM * 4;   // float[2][128]
  static constexpr int kOffBars = kOffRowSum + 2 * kBlockM * 4;
  static constexpr int kNumBars = 20 + 2 * kStages;
  static constexpr int kOffMisc = kOffBars + kNumBars * 8;
  static constexpr int kOffGeom = kOffMisc + 16;     // TMEM base, abort flag (+ 8 spare bytes)
  static constexpr int kSmemBytes = kOffGeom + 2 * 64;  // two work-item slots: the item's decoded geometry and its id
  static constexpr uint32_t kTmemCols = 512;
  static constexpr uint32_t kColS0 = 0, kColS1 = 128, kColO0 = 256, kColO1 = 384;
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
};

// exp2 of 64 scores (32 pairs) -> 32 packed fp16x2 words; adds the exponentials into two
// (even, odd) pairs of partial row sums.
__device__ __forceinline__ void exp_half_tile(const float* sc, uint64_t scale2, uint64_t negms2, uint32_t (&pk)[32],
                                              uint64_t& lsum_a, uint64_t& lsum_b) {
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    float x0, x1, e0, e1;
    f2_unpack(f2_fma(f2_pack(sc[2 * c], sc[2 * c + 1]), scale2, negms2), x0, x1);
    e0 = ex2_approx(x0);
    e1 = ex2_approx(x1);
    if (c & 1) lsum_b = f2_add(lsum_b, f2_pack(e0, e1));
    else lsum_a = f2_add(lsum_a, f2_pack(e0, e1));
    pk[c] = pack_f16x2(e0, e1);
  }
}

// Same for 32 scores (16 pairs) -> the first 16 words of pk.
__device__ __forceinline__ void exp_quarter_tile(const float* sc, uint64_t scale2, uint64_t negms2, uint32_t* pk,
                                                 uint64_t& lsum_a, uint64_t& lsum_b) {
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    float x0, x1, e0, e1;
    f2_unpack(f2_fma(f2_pack(sc[2 * c], sc[2 * c + 1]), scale2, negms2), x0, x1);
    e0 = ex2_approx(x0);
    e1 = ex2_approx(x1);
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
__device__ __forceinline__ void philox4x32_10(uint32_t k0, uint32_t k1, uint32_t c0, uint32_t c1, uint32_t c2,
                                              uint32_t c3, uint32_t (&out)[4]) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    c0 = hi1 ^ c1 ^ k0;
    c1 = lo1;
    c2 = hi0 ^ c3 ^ k1;
    c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// Zeroes the dropped elements of 32 packed fp16 pairs (64 consecutive columns starting at global column `col0`, a
// multiple of 16) of query row `row` of head `bh`. One Philox call serves 16 columns: byte t of its 16 output bytes
// (little endian over the four words) decides column 16 * block + t.
__device__ __forceinline__ void dropout_mask_64(uint32_t (&pk)[32], const FwdParams& p, int bh, int row, int col0) {
  constexpr uint32_t kHigh = 0x80808080u;
  const uint32_t thr4 = p.drop_keep_thr * 0x01010101u;
#pragma unroll
  for (int blk = 0; blk < 4; ++blk) {
    uint32_t r[4];
    philox4x32_10(p.seed_lo, p.seed_hi, static_cast<uint32_t>(col0 / 16 + blk), static_cast<uint32_t>(row),
                  static_cast<uint32_t>(bh), 0u, r);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      // High bit of each byte of `ge`: the byte is not below the threshold (a subtraction that borrows within bytes).
      // A byte permute with the sign-replicating selectors 8 + b spreads these bits over the halves of two words.
      const uint32_t diff = (r[w] | kHigh) - (thr4 & ~kHigh);
      const uint32_t ge = (r[w] & ~thr4) | (~(r[w] ^ thr4) & diff);
      uint32_t lo, hi;
      asm("prmt.b32 %0, %1, 0, 0x9988;" : "=r"(lo) : "r"(ge));
      asm("prmt.b32 %0, %1, 0, 0xBBAA;" : "=r"(hi) : "r"(ge));
      pk[blk * 8 + 2 * w] &= ~lo;      // columns 4w, 4w+1
      pk[blk * 8 + 2 * w + 1] &= ~hi;  // columns 4w+2, 4w+3
    }
  }
}

template <int D, bool kAlibi, bool kLse = false, bool kDropout = false>
__global__ void __launch_bounds__(512, 1)
fwd_persistent_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                      const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapO,
                      const FwdParams p) {
  using Cfg = PersistentCfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
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
  uint64_t* p_full = bars + 6;        // [2] softmax (first half of P) + correction (O rescaled) -> MMA
  uint64_t* alpha_ready = bars + 8;   // [2] softmax -> correction: rescale factors in smem
  uint64_t* l_ready = bars + 10;      // [2] softmax -> correction: final row sums in smem
  uint64_t* o_full = bars + 12;       // [2] MMA -> correction: last P.V of the item landed
  uint64_t* p_full2 = bars + 14;      // [2] softmax -> MMA: second half of P written
  uint64_t* item_full = bars + 16;    // [2] producer -> all roles: next work item id published
  uint64_t* item_empty = bars + 18;   // [2] all roles -> producer: id slot read
  uint64_t* kv_full = bars + 20;      // [kStages] TMA -> MMA
  uint64_t* kv_empty = bars + 20 + Cfg::kStages;  // [kStages] MMA -> TMA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // [2][16]: ItemGeom of the published item in words 0..11, its id (-1: no more items) in word 12, `split` in word 13
  volatile int* s_geom = reinterpret_cast<volatile int*>(smem + Cfg::kOffGeom);
  constexpr uint32_t kItemReaders = 13;  // 8 softmax warps + 4 correction warps + the MMA warp

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
      mbar_init(&p_full[s], 8);  // one arrival per softmax warp and per correction warp
      mbar_init(&p_full2[s], 4);
      mbar_init(&alpha_ready[s], 4);
      mbar_init(&l_ready[s], 4);
      mbar_init(&o_full[s], 1);
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
  if (warp == 13 && lane == 0) {
    prefetch_tensormap(&mapQ);
    prefetch_tensormap(&mapK);
    prefetch_tensormap(&mapV);
    prefetch_tensormap(&mapO);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Everything above overlaps the end of the kernel in front in the stream; nothing below this line has touched
  // global memory (inputs, outputs, scheduler words, status) before that kernel is complete.
  griddep_wait();

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
    reg_inc<FA_REG_SOFTMAX>();
    const int s = warp >> 2;
    const int row_l = tid & 127;
    const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
    const uint32_t tS = tmem_addr(tmem_base, lane_base, s == 0 ? Cfg::kColS0 : Cfg::kColS1);
    // With ALiBi the scores are moved to the biased log2 domain right after the TMEM load, and
    // everything downstream works with a unit scale.
    const float sl2 = kAlibi ? 1.f : p.scale_log2;
    const uint64_t scale2 = f2_pack(sl2, sl2);
    uint32_t n_s = 0;  // completed s_full phases
    uint32_t n_items = 0;
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
      float slope_l2 = 0.f;
      if (kAlibi) slope_l2 = p.alibi_slopes[g.bh % p.heads] * 1.4426950408889634f;
      float m_used = 0.f;  // the row's reference: the score that its exponentials are taken against
      float l_run = 0.f;   // 0 until the row has seen a finite score, at least about 1 from then on
      for (int j = j_lo; j < j_hi; ++j) {
        if (!mbar_wait_warp(&s_full[s], n_s & 1, abort_flag)) { ok = false; break; }
        ++n_s;
        tc_fence_after();
        const int kv0 = (g.split ? g.top - 2 * j - s : g.top - j) * kBlockN;
        // One body, instantiated twice: tiles cut by a mask boundary (or by the end of the sequence) take the
        // per-element predicate, all others carry none of that code. (Blanking a cut tile in tensor memory first
        // and sharing one body saved 10 KB of instructions but made every tile 4 % slower: the body then
        // starts behind a merge point instead of directly behind the wait.)
        auto tile_body = [&](auto masked_tag) {
          constexpr bool kMasked = decltype(masked_tag)::value;
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
            // Visible columns of this row: c_lo <= c <= c_hi, i.e. |c - mid| <= half. The predicate is applied on the
            // FMA pipe, which the softmax leaves nearly idle, instead of as two integer compares and a select per
            // element: t = saturate(|c - mid| - half) is 0 for a visible column and 1 for a hidden one (both
            // operands are multiples of 1/2, so the difference is exact), and sc - kHidden * t leaves a visible
            // score bit for bit as it is and puts a hidden one near -3e38, where its exponential is 0 for any scale the
            // host accepts.
            const int c_lo = (wl >= 0) ? row - wl - kv0 : -(1 << 20);
            int c_hi = N - 1 - kv0;
            if (wr >= 0) c_hi = min(c_hi, row + wr - kv0);
            const float mid = 0.5f * static_cast<float>(c_lo + c_hi);
            const float half = 0.5f * static_cast<float>(c_hi - c_lo);  // negative: no visible column at all
            constexpr float kHidden = 3.0e38f;
  #pragma unroll
            for (int c = 0; c < kBlockN; ++c) {
              const float t = __saturatef(fabsf(static_cast<float>(c) - mid) - half);
              sc[c] = fmaf(t, -kHidden, sc[c]);
            }
          }
          // The exponentials of the first 32 keys are taken against the reference the previous tile left while
          // the row max of this tile is still being reduced: nearly always the reference stays where it is (lazy
          // rescale), so the max leaves the critical path. When a row of the warp does move its reference
          // (always on the first tile of an item), the 32 exponentials are taken again. Cut tiles do not
          // speculate: most of them are the first tile of their walk.
          uint64_t lsum_a = 0ull, lsum_b = 0ull;
          uint32_t pk0[32], pk1[32];
          if (!kMasked) {
            const float neg_ms0 = -m_used * sl2;
            exp_quarter_tile(sc, scale2, f2_pack(neg_ms0, neg_ms0), pk0, lsum_a, lsum_b);
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
          if (kMasked && m_new < -1.0e37f) m_new = -INFINITY;  // nothing visible (hidden scores sit near -3e38)
          // The reference moves when the tile's max has grown past it (see kLazyLog2), and always on the first tile that
          // shows a finite score: the reference then IS the row max, so the largest term of the row is exactly 1 in
          // fp16 (a row with a single visible key returns that key's V bit for bit). A cut tile over the first keys is
          // the only tile of its walk (with ALiBi it may be the last), or the far edge of a left window lies in it.
          const bool fresh = l_run == 0.f;
          const bool first_keys = (!kMasked || kAlibi) && kv0 == 0;
          float alpha = 1.f;
          if (__any_sync(0xffffffffu, fresh || (m_new - m_used) * sl2 > (first_keys ? 0.f : Cfg::kLazyLog2))) {
            if (fresh || m_new > m_used) {
              const float m_next = (m_new == -INFINITY) ? 0.f : m_new;
              alpha = fresh ? 1.f : ex2_approx((m_used - m_next) * sl2);
              m_used = m_next;
            }
            if (!kMasked) {
              lsum_a = 0ull;
              lsum_b = 0ull;
              const float neg_ms1 = -m_used * sl2;
              exp_quarter_tile(sc, scale2, f2_pack(neg_ms1, neg_ms1), pk0, lsum_a, lsum_b);
            }
          }
          if (kMasked) {
            const float neg_ms1 = -m_used * sl2;
            exp_quarter_tile(sc, scale2, f2_pack(neg_ms1, neg_ms1), pk0, lsum_a, lsum_b);
          }
          // (no hand-over on the first tile of an item: there is nothing to rescale yet, and the correction warps
          // may still be in the previous item's epilogue)
          if (j != j_lo) sAlpha[s * kBlockM + row_l] = alpha;
          __syncwarp();
          if (lane == 0 && j != j_lo) mbar_arrive(&alpha_ready[s]);
          const float neg_ms = -m_used * sl2;
          const uint64_t negms2 = f2_pack(neg_ms, neg_ms);
          exp_quarter_tile(sc + 32, scale2, negms2, pk0 + 16, lsum_a, lsum_b);
          if (kDropout) dropout_mask_64(pk0, p, g.bh, row, kv0);  // the row sum keeps every exponential
          tmem_st32(tS + 0, pk0);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[s]);  // P of keys 0..63 is in TMEM
          exp_half_tile(sc + 64, scale2, negms2, pk1, lsum_a, lsum_b);
          if (kDropout) dropout_mask_64(pk1, p, g.bh, row, kv0 + 64);
          tmem_st32(tS + 32, pk1);
          float l0, l1;
          f2_unpack(f2_add(lsum_a, lsum_b), l0, l1);
          l_run = l_run * alpha + (l0 + l1);
          tmem_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full2[s]);  // P of keys 64..127
        };
        // (ALiBi: a tile that the diagonal crosses takes the cut tiles' body, whose bias has the absolute value)
        if (kv_tile_needs_mask(kv0, q_r0, q_r1, wl, wr, N) ||
            (kAlibi && kv0 + kBlockN - 1 > q_r0 && kv0 < q_r1))
          tile_body(std::true_type{});
        else tile_body(std::false_type{});
      }
      if (!ok) break;
      // The row sums of the previous item may still be unread when this item is a single tile. The last tile's
      // p_full phase completes only after the correction warps have arrived on it, and on an item's first tile
      // they do that after their epilogue of the previous item, which reads the sums first.
      if (!mbar_wait_warp(&p_full[s], (n_s - 1) & 1, abort_flag)) break;
      sRowSum[s * kBlockM + row_l] = l_run;
      // a split item's epilogue also needs the reference the sums are taken against; the rescale factors of this item
      // have all been read, and the next item's first factor is written after its first P.V, i.e. after that epilogue
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
    // correction + epilogue: row = tid % 128 of both stages
    // =====================================================================================
    reg_dec<FA_REG_CORR>();
    const int row_l = tid & 127;
    const uint32_t lane_base = static_cast<uint32_t>(warp & 3) * 32u;
    uint8_t* out_stage = smem + Cfg::kOffOut + (warp & 3) * Cfg::kOutWarpBytes;
    // Bit s: phase parity of stage s's barriers. The stages share one copy of this code (rolled loops, state in bit
    // masks): with copies for both and the epilogue in four places it was 38 KB, mostly run from cold instructions.
    uint32_t par_alpha = 0, par_l = 0, par_o = 0;
    uint32_t n_items = 0;
    // The first P.V product of an item overwrites O, so it has to wait until the epilogue of the previous item
    // has read O. That hand-off is the correction warps' arrival on p_full for the item's first tile; it is made
    // right after the epilogue (there is nothing to rescale on a first tile), so the next item's first product
    // does not wait for these warps to come round to it.
    uint32_t arrived_early = 0;  // bit s
    bool ok = true;
    while (ok) {
      ItemGeom g;
      const int item = take_item(n_items, g);
      if (item < 0) break;
      uint32_t epi_pending = g.split ? 0u : (g.r1[0] >= g.r0[0] ? 1u : 0u) | (g.r1[1] >= g.r0[1] ? 2u : 0u);  // bit s
      // O / l -> fp16 -> global for stage s, then the early arrival for the next item's first tile
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
        // 16 columns at a time, the load of the next chunk in flight while this one is converted and stored.
        // (Rolled up: this path runs once per item and stage, and instructions that are rarely executed are
        // fetched slowly; unrolling it eightfold made the change-over between items slower, not faster.)
        uint32_t ra[16], rb[16];
        tmem_ld16(tO, ra);
  #pragma unroll 2
        for (int c = 0; c < D / 16; ++c) {
          uint32_t (&cur)[16] = (c & 1) ? rb : ra;
          uint32_t (&nxt)[16] = (c & 1) ? ra : rb;
          tmem_wait_ld();
          tmem_ld_fence16(cur);
          if (c + 1 < D / 16) tmem_ld16(tO + (c + 1) * 16, nxt);
          // columns 16c .. 16c+15 are 16-byte units 2(c%4), 2(c%4)+1 of panel c/4; unit u of row r sits at u ^ (r%8)
          uint8_t* prow = out_stage + (c >> 2) * (32 * 128) + lane * 128;
  #pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint4 v;
            v.x = pack_f16x2(__uint_as_float(cur[i * 8 + 0]) * inv_l, __uint_as_float(cur[i * 8 + 1]) * inv_l);
            v.y = pack_f16x2(__uint_as_float(cur[i * 8 + 2]) * inv_l, __uint_as_float(cur[i * 8 + 3]) * inv_l);
            v.z = pack_f16x2(__uint_as_float(cur[i * 8 + 4]) * inv_l, __uint_as_float(cur[i * 8 + 5]) * inv_l);
            v.w = pack_f16x2(__uint_as_float(cur[i * 8 + 6]) * inv_l, __uint_as_float(cur[i * 8 + 7]) * inv_l);
            const int unit = ((c & 3) * 2 + i) ^ (lane & 7);
            *reinterpret_cast<uint4*>(prow + unit * 16) = v;
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
          mbar_arrive(&p_full[s]);
        }
        arrived_early |= 1u << s;
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
        for (int c = 0; c < D / 16; ++c) {
          uint32_t ra[16], rb[16];
          tmem_ld16(tO0 + c * 16, ra);
          tmem_ld16(tO1 + c * 16, rb);
          tmem_wait_ld();
          tmem_ld_fence16(ra);
          tmem_ld_fence16(rb);
          uint8_t* prow = out_stage + (c >> 2) * (32 * 128) + lane * 128;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            uint32_t v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int e = i * 8 + 2 * k;
              v[k] = pack_f16x2(fmaf(__uint_as_float(ra[e]), f0, __uint_as_float(rb[e]) * f1),
                                fmaf(__uint_as_float(ra[e + 1]), f0, __uint_as_float(rb[e + 1]) * f1));
            }
            const int unit = ((c & 3) * 2 + i) ^ (lane & 7);
            *reinterpret_cast<uint4*>(prow + unit * 16) = make_uint4(v[0], v[1], v[2], v[3]);
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
          mbar_arrive(&p_full[0]);
          mbar_arrive(&p_full[1]);
        }
        arrived_early = 3u;
      };
      for (int j = 0; j <= g.steps && ok; ++j) {
#pragma unroll 1
        for (int s = 0; s < 2 && ok; ++s) {
          const int lo = s ? g.lo[1] : g.lo[0], hi = s ? g.hi[1] : g.hi[0];
          // a stage that has run out of tiles is finished at once, while the other stage may still be in its softmax
          if (((epi_pending >> s) & 1) && j >= hi) {
            epi_pending &= ~(1u << s);
            epilogue(s);
            continue;
          }
          if (j < lo || j >= hi) continue;
          if (j == lo) {  // first tile of the item: nothing to rescale, and no factors are handed over
            const bool done = (arrived_early >> s) & 1;
            arrived_early &= ~(1u << s);
            if (done) continue;
          } else {
            if (!mbar_wait_warp(&alpha_ready[s], (par_alpha >> s) & 1, abort_flag)) { ok = false; break; }
            par_alpha ^= 1u << s;
            const float alpha = sAlpha[s * kBlockM + row_l];
            if (__any_sync(0xffffffffu, alpha != 1.f)) {
              tc_fence_after();
              const uint32_t tO = tmem_addr(tmem_base, lane_base, s == 0 ? Cfg::kColO0 : Cfg::kColO1);
#pragma unroll 1
              for (int c = 0; c < D / 32; ++c) {
                uint32_t r[32];
                tmem_ld32(tO + c * 32, r);
                tmem_wait_ld();
                tmem_ld_fence(r);
#pragma unroll
                for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
                tmem_st32(tO + c * 32, r);
              }
              tmem_wait_st();
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[s]);
        }
      }
      if (ok && g.split) epilogue_split();
    }
    if (lane == 0) tma_store_wait_all();  // also on the give-up path: stores in flight read this CTA's shared memory
  } else {
    reg_dec<FA_REG_MISC>();
    if (warp == 12) {
      // ===================================================================================
      // tensor-core issuer. The whole warp walks the schedule and waits, so that addresses and
      // descriptors are warp-uniform values; one elected lane issues the tcgen05 instructions.
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
      uint32_t par_p = 0, par_q = 0;  // bit s: phase parity of stage s's barriers
      uint32_t n_items = 0;
      bool ok = true;
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
          if (j >= alo && j < ahi) {  // O_s += P_s V
            const uint32_t tO = tmem_base + (s ? Cfg::kColO1 : Cfg::kColO0);
            const uint32_t pv = end - ((a.split && s == 0 && j < a.hi[1]) ? 2 : 1);
            const uint32_t slot = pv % Cfg::kStages;
            const uint32_t vdesc = vdesc0 + ((kv_addr + slot * Cfg::kTileBytes) >> 4);
            if (!mbar_wait_warp(&kv_full[slot], (pv / Cfg::kStages) & 1, abort_flag)) { ok = false; return; }
            if (!mbar_wait_warp(&p_full[s], (par_p >> s) & 1, abort_flag)) { ok = false; return; }
            tc_fence_after();
            if (elect_one()) {
              umma_ts_lo(tO, tS, vdesc, kDescHi, idesc_pv, j > alo ? 1u : 0u);
#pragma unroll
              for (int kk = 1; kk < 4; ++kk) umma_ts_lo(tO, tS + kk * 8, vdesc + kk * (2048 >> 4), kDescHi, idesc_pv, 1u);
            }
            __syncwarp();
            if (!mbar_wait_warp(&p_full2[s], (par_p >> s) & 1, abort_flag)) { ok = false; return; }
            par_p ^= 1u << s;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int kk = 4; kk < 8; ++kk) umma_ts_lo(tO, tS + kk * 8, vdesc + kk * (2048 >> 4), kDescHi, idesc_pv, 1u);
              if (a.split || s == 1 || j < a.lo[1] || j >= a.hi[1]) umma_commit(&kv_empty[slot]);
              umma_commit(&o_full[s]);
            }
            __syncwarp();
          }
          if (blo == 0 && bhi > 0) {  // S_s = Q_s K^T
            const uint32_t pk = end + (b.split ? s : 0);
            const uint32_t slot = pk % Cfg::kStages;
            if (!mbar_wait_warp(&q_full[s], (par_q >> s) & 1, abort_flag)) { ok = false; return; }
            par_q ^= 1u << s;
            if (!mbar_wait_warp(&kv_full[slot], (pk / Cfg::kStages) & 1, abort_flag)) { ok = false; return; }
            tc_fence_after();
            const uint32_t kdesc = kdesc0 + ((kv_addr + slot * Cfg::kTileBytes) >> 4);
            const uint32_t qd = s ? qdesc[1] : qdesc[0];
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < D / 16; ++k) {
                const uint32_t off = ((k / 4) * Cfg::kPanelBytes + (k % 4) * 32) >> 4;
                umma_ss_lo(tS, qd + off, kdesc + off, kDescHi, idesc_qk, k > 0 ? 1u : 0u);
              }
              umma_commit(&s_full[s]);
              if (b.split || s == 1 || b.lo[1] > 0 || b.hi[1] == 0) umma_commit(&kv_empty[slot]);
              if (bhi == 1) umma_commit(&q_empty[s]);
            }
            __syncwarp();
          }
        }
      };
      ItemGeom g;
      if (kJoin) {
        ItemGeom none;
        none.steps = none.split = none.lo[0] = none.lo[1] = none.hi[0] = none.hi[1] = 0;
        if (take_nonempty(g)) join(none, g, 0);
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
          return mbar_wait_warp(&kv_full[slot], par, abort_flag);
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
            if (act_j) {  // O_s += P_s(j) V_j, in two halves of 64 keys as P arrives
              if (kSplit) {
                slot_v = slot_k;
                par_v = par_k;
                advance(slot_k, par_k, 1);
              }
              const uint32_t vdesc = vdesc0 + ((kv_addr + slot_v * Cfg::kTileBytes) >> 4);
              if (!kInterior && !v_seen && !mbar_wait_warp(&kv_full[slot_v], par_v, abort_flag)) { ok = false; return; }
              if (!mbar_wait_warp(&p_full[s], (par_p >> s) & 1, abort_flag)) { ok = false; return; }
              tc_fence_after();
              if (elect_one()) {
                umma_ts_lo(tmem_base + colO, tmem_base + colS, vdesc, kDescHi, idesc_pv, (kInterior || j > g.lo[s]) ? 1u : 0u);
#pragma unroll
                for (int kk = 1; kk < 4; ++kk)
                  umma_ts_lo(tmem_base + colO, tmem_base + colS + kk * 8, vdesc + kk * (2048 >> 4), kDescHi, idesc_pv, 1u);
              }
              __syncwarp();
              if (!mbar_wait_warp(&p_full2[s], (par_p >> s) & 1, abort_flag)) { ok = false; return; }
              par_p ^= 1u << s;
              tc_fence_after();
              if (elect_one()) {
#pragma unroll
                for (int kk = 4; kk < 8; ++kk)
                  umma_ts_lo(tmem_base + colO, tmem_base + colS + kk * 8, vdesc + kk * (2048 >> 4), kDescHi, idesc_pv, 1u);
                if (!other_j) umma_commit(&kv_empty[slot_v]);
                if (!kInterior && j + 1 == g.hi[s]) umma_commit(&o_full[s]);
              }
              __syncwarp();
            }
            if (act_n) {  // S_s = Q_s K_{j+1}^T
              if (!kInterior && j + 1 == g.lo[s]) {
                if (!mbar_wait_warp(&q_full[s], (par_q >> s) & 1, abort_flag)) { ok = false; return; }
                par_q ^= 1u << s;
              }
              if (!k_seen && !mbar_wait_warp(&kv_full[slot_k], par_k, abort_flag)) { ok = false; return; }
              // Inner rounds wait for V here, one round ahead: every group of instructions then has one wait in front
              // of it, about as long as the tensor pipe has work queued (two waits in a row let it run dry).
              if (kInterior && s == 1 && !wait_next_v()) { ok = false; return; }
              tc_fence_after();
              const uint32_t kdesc = kdesc0 + ((kv_addr + slot_k * Cfg::kTileBytes) >> 4);
              if (elect_one()) {
#pragma unroll
                for (int k = 0; k < D / 16; ++k) {
                  const uint32_t off = ((k / 4) * Cfg::kPanelBytes + (k % 4) * 32) >> 4;
                  umma_ss_lo(tmem_base + colS, qdesc[s] + off, kdesc + off, kDescHi, idesc_qk, k > 0 ? 1u : 0u);
                }
                umma_commit(&s_full[s]);
                if (!other_n) umma_commit(&kv_empty[slot_k]);
                if (!kInterior && j + 2 == g.hi[s]) umma_commit(&q_empty[s]);
              }
              __syncwarp();
              if (kSplit) advance(slot_k, par_k, 1);
            }
          }
        };
        if (g.split) {
          for (int j = j_first; j < j_end && ok; ++j) round_body(std::false_type{}, std::true_type{}, j);
          pos += 2u * static_cast<uint32_t>(g.hi[0] + g.hi[1]);
        } else {
          for (int j = j_first; j < j_end && ok; ++j) {
            if (j == in_lo && in_lo < in_hi) ok = mbar_wait_warp(&kv_full[slot_v], par_v, abort_flag);
            if (j >= in_lo && j < in_hi) round_body(std::true_type{}, std::false_type{}, j);
            else round_body(std::false_type{}, std::false_type{}, j);
            // V_{j+1} sits right after K_{j+1}; K_{j+2} two positions after K_{j+1}
            slot_v = slot_k;
            par_v = par_k;
            advance(slot_v, par_v, 1);
            advance(slot_k, par_k, 2);
          }
          pos += 2u * static_cast<uint32_t>(g.steps);
        }
        if (!ok) break;
        if (kJoin) {
          ItemGeom nx;
          take_nonempty(nx);
          join(g, nx, pos);
          g = nx;
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
      int next = static_cast<int>(blockIdx.x);
      while (ok) {
        ItemGeom g;
        const int item =
            next_item(next, p, g, [&] { return static_cast<int>(gridDim.x) + atomicAdd(p.sched, 1); });
        if (item < 0) griddep_launch();  // no further item: the next kernel of the stream may take up free SMs
        {  // publish the item to the other roles
          const uint32_t slot = n_pub & 1u;
          if (!mbar_wait(&item_empty[slot], ((n_pub >> 1) & 1u) ^ 1u, abort_flag)) { ok = false; break; }
          volatile int* w = s_geom + slot * 16;
          if (item >= 0) {
            w[0] = g.bh; w[1] = g.pair;
            w[2] = g.r0[0]; w[3] = g.r0[1]; w[4] = g.r1[0]; w[5] = g.r1[1];
            w[6] = g.lo[0]; w[7] = g.lo[1]; w[8] = g.hi[0]; w[9] = g.hi[1];
            w[10] = g.top; w[11] = g.steps; w[13] = g.split;
          }
          w[12] = item;
          mbar_arrive(&item_full[slot]);
          ++n_pub;
        }
        if (item < 0) break;
        // Claim the following item now; the answer is looked at behind this item's loads.
        const int claimed = atomicAdd(p.sched, 1);
        auto load_q = [&](int s) {
          if (g.r1[s] < g.r0[s]) return;
          if (!ok || !mbar_wait(&q_empty[s], (n_q[s] & 1) ^ 1, abort_flag)) { ok = false; return; }
          ++n_q[s];
          mbar_arrive_expect_tx(&q_full[s], Cfg::kTileBytes);
          tma_load_4d(sQ + s * Cfg::kTileBytes, &mapQ, &q_full[s], 0, g.r0[s], 0, g.bh);
        };
        auto load_tile = [&](const CUtensorMap* map, int tile) {
          const uint32_t slot = it % Cfg::kStages;
          if (!ok || !mbar_wait(&kv_empty[slot], ((it / Cfg::kStages) & 1) ^ 1, abort_flag)) { ok = false; return; }
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
        load_q(0);
        load_q(1);
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
        next = static_cast<int>(gridDim.x) + claimed;
      }
      if (!ok) {
        // give-up path: let loads that are still in flight land before the CTA retires
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (tid == 0) {
    const int gave_up = *abort_flag != 0 ? 1 : 0;
    if (gave_up) atomicExch(p.status, 1);
    if (p.status_per_launch && blockIdx.x == 0) {
      p.sched[p.clear_at] = 0;
      p.sched[p.clear_at + 1] = 0;
    }
    // the last CTA to finish puts the scheduler words back to zero for the next launch
    const int ended = atomicAdd(p.sched + 1, 1 + (gave_up << 16)) + 1 + (gave_up << 16);
    if ((ended & 0xffff) == static_cast<int>(gridDim.x)) {
      if (p.status_per_launch) *p.status = (ended >> 16) != 0 ? 1 : 0;
      p.sched[0] = 0;
      p.sched[1] = 0;
      __threadfence();
    }
  }
  if (warp == 12) tmem_dealloc(tmem_base, Cfg::kTmemCols);
}

}  // namespace fa
