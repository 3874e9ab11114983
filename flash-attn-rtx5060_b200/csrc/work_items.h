// Work items of the one-CTA persistent kernel: the host's plan (which pairs of q tiles are taken apart), the geometry of
// an item and the walk over the items that a CTA claims. Plain C++ as well as device code, so that the walk can be
// checked without a GPU.
#pragma once
#include "fwd_params.h"

#ifdef __CUDA_ARCH__
#define FA_UNROLL _Pragma("unroll")
#else
#define FA_UNROLL
#endif

namespace fa {

__host__ __device__ inline int min_int(int a, int b) { return a < b ? a : b; }

// Heads per scheduling group of the persistent kernel. Without a mask all items cost the same and head-major
// order (1) shares K/V best. With a causal mask or a window the item costs differ, and interleaving the heads of
// a group pair-major makes the order of the group longest first (causal masks). Measured constraints (B200): the K and V
// rows that a group keeps live (the whole head, or the window span) should stay within ~64 MB (the 126 MB L2 holds two copies of
// what both dies read: the long-context workload read K/V from DRAM 2.2 times with 96 MB in flight, 1.5 times
// with 64 MB, 1.1 times with 48 MB, at the same speed; the 8192-row config is 0.6 % faster with 64 MB than
// with 48); a group needs about two items per CTA to balance; and the groups must be of even size (64 heads in
// groups of 12 leave a last group of 4 heads, too few items for 148 CTAs: -4 %). Within those limits a group is as
// large as it can be: with one group for all heads the whole launch is handed out longest first and ends on its
// cheapest items. Against groups of at most 16 heads: B4 H16 N2048 d64 causal 82.4 -> 72.8 us, 24 heads of 4001 rows
// d128 with log-sum-exp 132 -> 116, B2 H16 N4096 d64 ALiBi 161 -> 136, B8 H16 N1024 d128 70 -> 58.
inline int pick_head_group(int bh, int seqlen, int head_dim, int causal, int window_left, int window_right,
                           int num_q_pairs, int num_sms, int most = 0x7fffffff) {
  if (!causal && window_left < 0 && window_right < 0) return 1;
  const int wr = causal ? 0 : window_right;
  long long span = seqlen;
  if (window_left >= 0 && wr >= 0) {
    span = (long long)window_left + wr + 2 * kBlockM;
    if (span > seqlen) span = seqlen;
  }
  const double span_bytes = 4.0 * (double)span * head_dim;  // K and V rows, fp16
  int grp_l2 = (int)(64.0 * 1024 * 1024 / span_bytes);
  const int grp_bal = (2 * num_sms + num_q_pairs - 1) / num_q_pairs;
  int grp = grp_l2;
  if (grp < grp_bal) grp = grp_bal;
  if (grp > most) grp = most;
  if (grp < 1) grp = 1;
  if (grp > bh) grp = bh;
  const int groups = (bh + grp - 1) / grp;
  return (bh + groups - 1) / groups;
}

// Takes some of the pairs of q tiles apart into single q tiles whose kv tiles the two stages of a CTA share out
// (ItemGeom::split). Per unit of work a single costs more than a pair (where balance
// no longer matters about 1.05 times, 48x1536 and 60x1024 below: every product fetches a kv tile of its own, and
// the epilogue merges two outputs), but there are twice as many items of half the length.
// - Items of about equal cost (no mask, a short window): the last, partial wave is split when its halves still make
//   one wave. 32x4096 d128: 3.46 waves of 32 steps, 246 -> 220 us; 40x1000 d64 31.3 -> 25.3 us.
// - Under a causal mask items are handed out longest first, and what decides is how they fill the waves. Let r be the
//   pairs per CTA (tiles / 2, so that an unfilled last pair counts half). Up to r = 1 pairs are one wave that lasts as
//   long as the longest of them; singles are two waves of half the length, which pays off while they fill little of the
//   second or a head has many pairs of different lengths. From r = 1 on pairs need a second wave and singles balance
//   better, until there are so many items of either kind that balance matters less than the cost of a single. Below, the
//   lines in percent of r by a head's tiles t. The same rule serves a window bounded on one side without a causal mask,
//   whose items differ likewise. Time of pairs over singles, d64 / d128 (heads x rows; r):
//   20x640 (0.3) 1.03 / 1.08, 32x640 (0.5) 0.85 / 0.92, 28x768 (0.6) 1.04 / 1.02, 36x768 (0.7) 0.96 / 1.03, 20x896 (0.5)
//   1.12 / 1.14, 28x896 (0.7) 0.89 / 1.03, 24x1000 (0.6) 1.11 / 1.09, 32x1000 (0.9) 0.94 / 1.03, 40x1024 (1.1) 1.09 / 1.12,
//   60x1024 (1.6) 0.95 / 1.01, 24x1280 (0.8) 1.05 / 1.08, 32x1280 (1.1) 1.14 / 1.19, 48x1280 (1.6) 1.01 / 1.03, 24x1536
//   (1.0) 1.08 / 1.08, 32x1536 (1.3) 1.15 / 1.16, 48x1536 (1.9) 0.96 / 1.00, 22x2048 (1.2) 1.24 / 1.26, 36x2048 (1.9) 1.05
//   / 1.05, 48x2048 (2.6) 0.92 / 0.95, 20x3000 (1.6) 1.10 / 1.11, 26x3000 (2.1) 0.98 / 0.99, 18x4096 (1.9) 1.07 / 1.05,
//   24x4096 (2.6) 0.92 / 0.93, 10x8192 (2.2) 1.16 / 1.08, 14x8192 (3.0) 0.98 / 0.94, 6x16384 (2.6) 1.11 / 1.01, 8x16384
//   (3.5) 1.00 / 0.98, 4x32768 (3.5) 1.03 / 1.05. With dropout 30x768 1.08 / 1.06, 40x1024 1.11 / 1.10, 36x1536 1.14 / 1.10,
//   32x2048 1.14 / 1.12; with ALiBi 28x768 1.04 / 1.06, 40x1024 1.07 / 1.11, 32x1536 1.15 / 1.15, 34x2048 1.04 / 1.07, 12x4096
//   1.31 / 1.29, 10x8192 1.05 / 1.08.
inline long long pairs_to_split(long long heads, int num_q_pairs, int seqlen, int window_left, int window_right,
                                int num_sms) {
  const long long pairs = heads * num_q_pairs;
  if (seqlen <= kBlockM || pairs >= (1 << 30)) return 0;
  const bool even = (window_left < 0 && window_right < 0) || (window_left >= 0 && window_right >= 0 &&
                                                               window_left < seqlen / 4 && window_right < seqlen / 4);
  if (even) {
    const long long tail = pairs % num_sms;
    return 2 * tail <= num_sms ? tail : 0;
  }
  const int t = (seqlen + kBlockM - 1) / kBlockM;
  const long long r100 = 50 * heads * t / num_sms;
  constexpr int kOneWave[] = {61, 50, 66, 64, 85, 80};  // t = 6 .. 11
  const int one_wave = t <= 5 ? 50 : t >= 12 ? 100 : kOneWave[t - 6];
  const int most = t < 8 ? 0 : t < 10 ? 135 : t < 12 ? 160 : t < 14 ? 175 : t < 48 ? 200 : t < 96 ? 240 : t < 192 ? 280 : 350;
  return r100 <= one_wave || (r100 > 100 && r100 <= most) ? pairs : 0;
}

// Whether a launch takes the kernel's short build: q tiles that see few kv tiles, most of all where some of them are cut,
// since the other build has a body of code for either kind. It depends on the shape of a head alone, so chunks and slabs
// of a problem take the build that the whole would. Time of the other build over the short one's, head_dim 64 / 128
// (batch x heads x rows):
//   no mask        16x16x128 1.08 / 1.16, 16x16x256 1.08 / 1.07, 8x16x640 1.05 / 1.08, 8x16x768 0.98 / 1.01,
//                  8x16x1024 0.98 / 1.02
//   ..., ragged    8x12x700 1.04 / 1.06, 8x12x1000 1.01 / 1.04, 8x12x1200, 1300 1.01 / 1.05, 8x12x1700 - / 1.00
//   causal         16x16x512 1.11 / 1.09, 8x16x1024 1.09 / 1.08, 4x16x2048 1.03 / 1.05, 4x16x2560 1.01 / 1.02,
//                  4x16x3072 1.00 / 1.02, 24x4001 - / 0.97
//   window (left, right) over 4x16x4096   256,0 1.09 / 1.02, 512,0 1.01 / 1.01, 768,0 0.99 / 1.00, 1024,0 0.98 / 0.96,
//                  128,128 1.10 / 1.03, 256,256 1.04 / 1.04, 512,512 1.02 / 1.00
// With dropout 16x4x256 1.24, 16x4x1024 1.07 / 1.10, 16x4x2048 1.02 / 1.06.
// With ALiBi the one body takes the bias as linear in the column, which holds where all visible keys lie on one side: under
// a causal mask. A cut tile of the other build then costs more, too: 8x16x512 1.25 / 1.23, 8x16x1024 1.13 / 1.17, 4x16x2048
// 1.08 / 1.08, 8x4096 1.15 / 1.12, 2x16x4096 1.01 / 1.04, 4x16x4096 0.98 / 1.04, 2x16x6144 0.96 / 1.02.
inline bool short_items(int seqlen, int causal, int window_left, int window_right, bool alibi) {
  const int wr = eff_window_right(causal, window_right);
  if (alibi) return causal && window_left < 0 && seqlen <= 32 * kBlockN;
  if (window_left < 0 && wr < 0) return seqlen <= (seqlen % kBlockN ? 10 : 5) * kBlockN;
  if (seqlen <= 20 * kBlockN) return true;
  return window_left >= 0 && wr >= 0 && wr <= 4 * kBlockN && window_left <= 4 * kBlockN - wr;
}

// The items of a launch on p->bh heads, the first of which is head `first_head` of a problem of `total_heads`: its order
// (head_group), and how many pairs at the end of that order are taken apart. A split q tile is summed in another order
// than a pair's, so which pairs are split is decided for the whole problem: the chunks of flash_forward_host and the slabs
// of flash_forward_multi_gpu give the bits of the call on all heads. Where only the last pairs of the problem are
// split, they must be the last ones of the slab's order as well, if it holds any of them. That is so in head-major order
// and where all heads form one group; with several groups (windows over so many heads that K and V pass L2, hence with
// many waves of items) nothing is split. (Head-major order for windows whose last pairs are split would serve too, but
// runs up to 17 % slower: 40 heads x 4096 rows d128, window 512 75 -> 84 us, 256 x 1500 d64, window 128 71 -> 83.)
inline void set_work_items(FwdParams* p, int head_dim, int num_sms, long long first_head, long long total_heads) {
  const int wl = p->window_left, wr = eff_window_right(p->causal, p->window_right), nq = p->num_q_pairs;
  auto group = [&](long long heads) {
    const int bh = heads > 0x7fffffff ? 0x7fffffff : static_cast<int>(heads);
    return pick_head_group(bh, p->seqlen, head_dim, p->causal, p->window_left, p->window_right, nq, num_sms);
  };
  const long long all = total_heads * nq, last = first_head + p->bh;
  const int pairs = p->bh * nq, group_all = group(total_heads);
  p->head_group = group(p->bh);
  long long split = pairs_to_split(total_heads, nq, p->seqlen, wl, wr, num_sms);
  if (split > 0 && split < all && group_all > 1) {
    if (group_all < total_heads) {
      split = 0;
    } else {  // one group: pairs in the order (pair, head), the first split one is `head` of pair `pr`
      const long long pr = (all - split) / total_heads, head = (all - split) % total_heads;
      split = (nq - 1 - pr) * p->bh;
      if (last > head) split += last - (first_head > head ? first_head : head);
    }
  } else {  // head-major, or all or none of the pairs
    split = last * nq - (all - split);
    split = split < 0 ? 0 : (split > pairs ? pairs : split);
  }
  p->num_pair_items = pairs - static_cast<int>(split);
  p->num_items = pairs + static_cast<int>(split);
}

// Whether a plain launch of the short build at head_dim 64 gives P tensor-memory columns of its own (kOwnP in
// fwd_persistent.cuh; the same bits either way). The turnaround that it saves is worth more than its two further waits and
// their cold code from about six rounds an item on, and nothing in single q tiles, whose stages have half the rounds. Time
// of the build without over the one with them (batch x heads x rows):
//   no mask     16x12x200 0.96, 1x4x512 0.97, 8x16x512 1.00, 16x16x640 1.00 (five tiles), 8x12x700 1.02, 8x12x1000 1.05,
//               16x12x1200 1.05, 8x16x1250 1.05, 1x8x900 1.00
//   causal      1x16x1000 0.91, 16x16x256 0.96, 8x16x1024 0.99, 16x16x1280 1.00, 8x16x1500 1.00, 8x16x2048 1.01,
//               4x16x2048 1.02, 4x16x2560 1.02; with single q tiles 2x16x1800 0.95, 1x32x2048 0.94, 2x12x2300 0.95
//   window      4x16x4096 left 256 0.97, 4x12x2000 left 128 0.96
// (In the build for long sequences it gains 0-1 % without a mask, loses 0-2 % under a causal one and 4-6 % with ALiBi.)
inline bool own_p_columns(const FwdParams& p) {
  if (p.window_left >= 0 || (!p.causal && p.window_right >= 0)) return false;
  const int t = (p.seqlen + kBlockN - 1) / kBlockN;
  return p.causal ? t >= 14 && p.num_items == p.num_pair_items : t >= 6;
}

// Work item -> geometry. Every role decodes the same item the same way.
// The kv tiles of an item are walked from the last visible one to the first. Under a causal mask (and for a ragged
// end) the tiles that carry the per-element predicate then come first, where the pipeline fills anyway, instead of
// at the item's end where nothing hides them; the two stages start one tile apart, out of phase; and with ALiBi the
// bias falls along the walk, so the row reference is found on the first tile and stays. Measured on B200, first to
// last against last to first (and no speculation in cut tiles): B4 H16 N2048 d64 causal 89.2 -> 82.4 us,
// B2 H32 N8192 d128 causal 1112 -> 1079, its 16384-row sliding window 755 -> 712, B2 H16 N4096 d64 ALiBi 217 -> 182,
// B4 H16 N2048 d64 with dropout 138 -> 125.
struct ItemGeom {
  int bh, pair;
  int r0[2], r1[2];  // first / last q row of each stage's tile (r1 < r0: stage has no rows)
  int lo[2], hi[2];  // walk steps of each stage, [lo, hi); empty when no rows. Step t works on kv tile `top - t`
  int top, steps;    // last visible kv tile of the item, number of steps
  // 0: the stages own the two q tiles of a pair and share every kv tile (both work on tile `top - t` in step t).
  // 1: both stages own the SAME q tile and take its kv tiles in turn: stage s works on tile top - 2t - s; the
  //    epilogue merges their two outputs.
  int split;
};

// Work-item order. Heads are taken in groups of `head_group` (sized on the host so that the K/V of
// a group stays in L2); inside a group the items run pair-major from the last (under a causal mask
// the longest) q pair to the first. CTAs claim items in this order from a global counter, so CTAs
// that run together read the same few heads, and under a causal mask the items handed out last are the
// cheapest ones of the last group: the tail stays short. (With a window bounded on the left only and no causal mask
// the first pairs are the longest, and come last.)
template <int BN = kBlockN>
__host__ __device__ inline ItemGeom decode_item(int item, const FwdParams& p) {
  ItemGeom g;
  const int sub = (item - p.num_pair_items) & 1;  // of a split pair: 0 the second q tile (the longer one), 1 the first
  g.split = item >= p.num_pair_items;
  if (g.split) item = p.num_pair_items + ((item - p.num_pair_items) >> 1);
  const int per_group = p.head_group * p.num_q_pairs;
  const int grp = item / per_group;
  const int r = item - grp * per_group;
  const int heads_here = min_int(p.head_group, p.bh - grp * p.head_group);
  const int pr = r / heads_here;
  g.bh = grp * p.head_group + (r - pr * heads_here);
  g.pair = p.num_q_pairs - 1 - pr;
  const int wr = eff_window_right(p.causal, p.window_right);
  int lo_all = 0x7fffffff, hi_all = 0;
FA_UNROLL
  for (int s = 0; s < 2; ++s) {
    g.r0[s] = g.pair * 2 * kBlockM + s * kBlockM;
    if (g.r0[s] >= p.seqlen) {
      g.r1[s] = g.r0[s] - 1;
      g.lo[s] = g.hi[s] = 0;
    } else {
      g.r1[s] = min_int(g.r0[s] + kBlockM, p.seqlen) - 1;
      g.lo[s] = kv_tile_begin(g.r0[s], p.window_left, BN);
      g.hi[s] = kv_tile_end(g.r1[s], wr, p.seqlen, BN);
      lo_all = min_int(lo_all, g.lo[s]);
      hi_all = hi_all > g.hi[s] ? hi_all : g.hi[s];
    }
  }
  if (g.split) {
    const int s = 1 - sub;
    const int n = s ? g.hi[1] - g.lo[1] : g.hi[0] - g.lo[0];  // kv tiles of the one q tile (0: it has no rows)
    g.top = (s ? g.hi[1] : g.hi[0]) - 1;
    g.r0[0] = g.r0[1] = s ? g.r0[1] : g.r0[0];
    g.r1[0] = s ? g.r1[1] : g.r1[0];
    g.r1[1] = n > 1 ? g.r1[0] : g.r0[0] - 1;
    g.lo[0] = g.lo[1] = 0;
    g.hi[0] = g.steps = (n + 1) >> 1;
    g.hi[1] = n >> 1;
    g.split = n > 1;
    return g;
  }
  g.top = hi_all - 1;
  g.steps = hi_all - lo_all;
FA_UNROLL
  for (int s = 0; s < 2; ++s) {  // tile range -> step range
    if (g.r1[s] < g.r0[s]) continue;
    const int lo = g.lo[s];
    g.lo[s] = hi_all - g.hi[s];
    g.hi[s] = hi_all - lo;
  }
  return g;
}

// The first item with rows, starting at `item` and going on with what `claim()` returns (the next unclaimed item);
// -1 when the items have run out. A split pair whose second q tile lies past the end of the sequence counts as two items,
// one of them without rows. Such an item is never published to the roles of the kernel: the issuing warp looks for the
// next item before it commits the last product of the current one, the epilogue warps wait for that commit before they
// free the slot of the item after next, and with two slots two row-less items in a row would close that circle.
template <typename Claim>
__host__ __device__ inline int next_item(int item, const FwdParams& p, ItemGeom& g, Claim claim) {
  while (item >= 0 && item < p.num_items) {
    g = decode_item(item, p);
    if (g.steps > 0) return item;
    item = claim();
  }
  return -1;
}

}  // namespace fa
