// Host build of the kernel's work-item code (csrc/work_items.h) for tests/test_work_items.py.
#include <cstring>

#include "work_items.h"

namespace {
fa::FwdParams params(int bh, int seqlen, int causal, int window_left, int window_right, int head_group, int num_sms) {
  fa::FwdParams p;
  std::memset(&p, 0, sizeof(p));
  p.bh = bh;
  p.seqlen = seqlen;
  p.causal = causal;
  p.window_left = window_left;
  p.window_right = window_right;
  p.head_group = head_group;
  p.num_q_pairs = (seqlen + 2 * fa::kBlockM - 1) / (2 * fa::kBlockM);
  p.num_items = bh * p.num_q_pairs;
  fa::set_work_items(&p, num_sms);
  return p;
}
}  // namespace

extern "C" {

// Number of items, and of those the pairs, that a launch hands out.
void plan(int bh, int seqlen, int causal, int window_left, int window_right, int head_group, int num_sms, int* items,
          int* pair_items) {
  const fa::FwdParams p = params(bh, seqlen, causal, window_left, window_right, head_group, num_sms);
  *items = p.num_items;
  *pair_items = p.num_pair_items;
}

// next_item() from `item` on, claims taken from the list; out[0..13] = item, head, rows and steps of both stages, top,
// steps, split. Returns the number of claims used.
int walk(int bh, int seqlen, int causal, int window_left, int window_right, int head_group, int num_sms, int item,
         const int* claims, int* out) {
  const fa::FwdParams p = params(bh, seqlen, causal, window_left, window_right, head_group, num_sms);
  fa::ItemGeom g;
  std::memset(&g, 0, sizeof(g));
  int used = 0;
  out[0] = fa::next_item(item, p, g, [&] { return claims[used++]; });
  const int rest[] = {g.bh, g.r0[0], g.r1[0], g.lo[0], g.hi[0], g.r0[1], g.r1[1], g.lo[1], g.hi[1], g.top, g.steps, g.split};
  std::memcpy(out + 1, rest, sizeof(rest));
  return used;
}
}
