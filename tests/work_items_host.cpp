// Host build of the kernel's work-item code (csrc/work_items.h) for tests/test_work_items.py.
#include <cstring>

#include "work_items.h"

namespace {
fa::FwdParams params(const int* a) {  // bh, seqlen, head_dim, causal, window_left, window_right, num_sms, first, total heads
  fa::FwdParams p;
  std::memset(&p, 0, sizeof(p));
  p.bh = a[0];
  p.seqlen = a[1];
  p.causal = a[3];
  p.window_left = a[4];
  p.window_right = a[5];
  p.num_q_pairs = (p.seqlen + 2 * fa::kBlockM - 1) / (2 * fa::kBlockM);
  fa::set_work_items(&p, a[2], a[6], a[7], a[8]);
  return p;
}
}  // namespace

extern "C" {

// out[0..2] = number of items that a launch hands out, of those the pairs, heads per scheduling group
void plan(const int* args, int* out) {
  const fa::FwdParams p = params(args);
  out[0] = p.num_items;
  out[1] = p.num_pair_items;
  out[2] = p.head_group;
}

// short_items() of a launch, with ALiBi or without
int short_build(const int* args, int alibi) { return fa::short_items(args[1], args[3], args[4], args[5], alibi != 0); }

// own_p_columns(), which plain launches of the short build at head_dim 64 ask
int own_p(const int* args) { return fa::own_p_columns(params(args)); }

// next_item() from `item` on, claims taken from the list; out[0..12] = item, head, rows and steps of both stages, top,
// steps, split. Returns the number of claims used.
int walk(const int* args, int item, const int* claims, int* out) {
  const fa::FwdParams p = params(args);
  fa::ItemGeom g;
  std::memset(&g, 0, sizeof(g));
  int used = 0;
  out[0] = fa::next_item(item, p, g, [&] { return claims[used++]; });
  const int rest[] = {g.bh, g.r0[0], g.r1[0], g.lo[0], g.hi[0], g.r0[1], g.r1[1], g.lo[1], g.hi[1], g.top, g.steps, g.split};
  std::memcpy(out + 1, rest, sizeof(rest));
  return used;
}
}
