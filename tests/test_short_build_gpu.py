"""The kernel has a build for q tiles that see few kv tiles and one for all others; which of them a launch takes depends on
the sequence length and the masks alone (short_items() in csrc/work_items.h). Both sides of every line, against the
attention of the same inputs in 64 bits."""
import ctypes
import math

import numpy as np
import pytest

from conftest import make_inputs, rules_args

pytestmark = pytest.mark.gpu

#          rows, causal, left, right
EDGES = [(640, False, -1, -1), (768, False, -1, -1), (641, False, -1, -1), (1280, False, -1, -1), (1279, False, -1, -1),
         (1281, False, -1, -1), (2560, True, -1, -1), (2561, True, -1, -1), (2688, True, -1, -1), (2900, True, 512, -1),
         (2900, True, 513, -1), (2816, False, 200, 312), (2816, False, 200, 313), (2800, False, -1, 40), (2500, False, 90, -1),
         (1, True, -1, -1), (128, False, -1, -1), (129, True, 0, -1)]


def exact(q, k, v, causal, wl, wr):
    import torch

    n, d = q.shape[2:]
    i = torch.arange(n, device="cuda")
    gap = i[None, :] - i[:, None]
    hidden = torch.zeros(n, n, dtype=torch.bool, device="cuda")
    if wl >= 0:
        hidden |= gap < -wl
    if causal:
        hidden |= gap > 0
    elif wr >= 0:
        hidden |= gap > wr
    s = (q.double() @ k.double().transpose(-1, -2) / math.sqrt(d)).masked_fill_(hidden, -math.inf)
    return torch.softmax(s, dim=-1) @ v.double(), torch.logsumexp(s, dim=-1)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n,causal,wl,wr", EDGES)
def test_both_builds_at_the_lines_between_them(pkg, d, n, causal, wl, wr):
    import torch

    q, k, v = (torch.from_numpy(a).cuda() for a in make_inputs(n + d, 1, 3, n, d))
    want, want_lse = exact(q, k, v, causal, wl, wr)
    kw = dict(causal=causal, window_left=wl, window_right=wr)
    out = pkg.attention_forward(q, k, v, **kw)
    out2, lse = pkg.attention_forward(q, k, v, return_lse=True, **kw)
    own = torch.empty_like(q)
    stream = torch.cuda.current_stream().cuda_stream
    assert pkg.lib().flash_forward_noalloc(q.data_ptr(), k.data_ptr(), v.data_ptr(), own.data_ptr(), 1, 3, n, d, 0.0,
                                           int(causal), wl, wr, stream, 0, 1) == pkg.FA_OK
    pkg.check(stream)
    for o in (out, out2, own):
        # probabilities and output rounded to fp16: 2^-11 of |v| (rows that see one key: exact) and half an ulp of the
        # output; the largest |v| is about 4.5
        assert (o.double() - want).abs().max().item() < 4e-3
        assert ((o.double() - want).norm() / want.norm()).item() < 4e-4
    assert torch.equal(own, out)                            # the same kernel behind either entry point
    assert (lse.double() - want_lse).abs().max().item() < 5e-5  # fp32 sums of up to 2900 terms
    if causal or wl == 0:
        assert torch.equal(out[:, :, 0], v[:, :, 0])        # one visible key: its value bit for bit


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n,causal,wl", [(1, True, -1), (127, True, -1), (129, True, -1), (1000, True, -1), (4096, True, -1),
                                         (4100, True, -1), (1000, True, 300), (1000, False, -1)])
def test_alibi_in_both_builds(pkg, d, n, causal, wl):
    import torch

    q, k, v = (torch.from_numpy(a).cuda() for a in make_inputs(n + d, 1, 4, n, d))
    slopes = torch.tensor([0.5, 2.0 ** -6, 0.0, -0.01], device="cuda")  # no bias, and one that grows with the distance
    i = torch.arange(n, device="cuda")
    gap = i[None, :] - i[:, None]
    s = q.double() @ k.double().transpose(-1, -2) / math.sqrt(d) - slopes.double()[:, None, None] * gap.abs()
    hidden = (gap > 0) & causal
    if wl >= 0:
        hidden |= gap < -wl
    s.masked_fill_(hidden, -math.inf)
    want, want_lse = torch.softmax(s, dim=-1) @ v.double(), torch.logsumexp(s, dim=-1)
    kw = dict(causal=causal, window_left=wl, alibi_slopes=slopes)
    out = pkg.attention_forward(q, k, v, **kw)
    out2, lse = pkg.attention_forward(q, k, v, return_lse=True, **kw)
    pkg.check(torch.cuda.current_stream().cuda_stream)
    for o in (out, out2):
        assert (o.double() - want).abs().max().item() < 4e-3
        assert ((o.double() - want).norm() / want.norm()).item() < 4e-4
    assert (lse.double() - want_lse).abs().max().item() < 1e-4  # biases of up to 60, in fp32
    if causal:
        assert torch.equal(out[:, :, 0], v[:, :, 0])


@pytest.mark.parametrize("n,d,causal", [(2500, 64, True), (2700, 64, True), (1200, 128, False), (1400, 128, False)])
def test_dropout_in_both_builds(pkg, ob, n, d, causal):
    import torch

    q, k, v = make_inputs(n, 1, 1, n, d)
    out = pkg.attention_forward(*(torch.from_numpy(a).cuda() for a in (q, k, v)), causal=causal, dropout_p=0.2, seed=5)
    pkg.check(torch.cuda.current_stream().cuda_stream)
    mx, mean, nans = ob.abs_error(out.cpu().numpy(), ob.attention_dropout(q, k, v, 0.2, 5, causal=causal))
    assert nans == 0 and mx <= 2.5e-3 and mean <= 2.5e-4, (mx, mean, nans)
    slopes = np.array([0.03125], np.float32)
    out = pkg.attention_forward(*(torch.from_numpy(a).cuda() for a in (q, k, v)), causal=causal, dropout_p=0.2, seed=5,
                                alibi_slopes=torch.from_numpy(slopes).cuda())
    want = ob.attention_dropout(q, k, v, 0.2, 5, causal=causal, alibi_slopes=slopes)
    mx, mean, nans = ob.abs_error(out.cpu().numpy(), want)
    assert nans == 0 and mx <= 4e-3 and mean <= 3e-4, (mx, mean, nans)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n,short", [(2560, True), (2688, False)])
def test_the_line_does_not_depend_on_the_number_of_heads(pkg, wi, n, short, d):
    """Last tiles on either side of the line. All pairs of q tiles are taken apart with 8 heads as with 4, so the bits are
    the same unless the builds are not: the two round some exponentials differently."""
    import torch

    for heads in (8, 4):
        plan = (ctypes.c_int * 3)()
        wi.plan(rules_args(heads, n, d, True), plan)
        assert list(plan)[:2] == [2 * heads * ((n + 255) // 256), 0]  # single q tiles alone
        assert bool(wi.short_build(rules_args(heads, n, d, True), 0)) == short
    q, k, v = (torch.from_numpy(a).cuda() for a in make_inputs(3, 1, 8, n, d))
    whole = pkg.attention_forward(q, k, v, causal=True)
    parts = [pkg.attention_forward(*(t[:, h:h + 4].contiguous() for t in (q, k, v)), causal=True) for h in (0, 4)]
    assert torch.equal(torch.cat(parts, dim=1), whole)


# Plain launches at head_dim 64 give P columns of its own in part of the short build's range (own_p_columns() in
# csrc/work_items.h); with the log-sum-exp they do not. One arithmetic: the same bits.
@pytest.mark.parametrize("rising", [False, True])
@pytest.mark.parametrize("b,h,n,causal", [(1, 1, 641, False), (2, 20, 700, False), (8, 24, 897, False), (1, 3, 1279, False),
                                          (1, 2, 640, False), (4, 16, 1665, True), (2, 48, 1664, True), (5, 30, 1793, True),
                                          (3, 32, 2560, True), (1, 16, 2048, True)])
def test_columns_of_its_own_for_p_change_no_bit(pkg, b, h, n, causal, rising):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    q, k, v = (torch.randn(b, h, n, 64, device="cuda", generator=g) for _ in range(3))
    if rising:  # kv runs from the last tile to the first: scores that grow that way move every row's reference in every tile
        q = q.abs()
        k = k * 0.1 + torch.linspace(6.0, -1.0, n, device="cuda")[:, None]
    q, k, v = q.half(), k.half(), v.half()
    out = pkg.attention_forward(q, k, v, causal=causal)
    again = pkg.attention_forward(q, k, v, causal=causal)
    want, _ = pkg.attention_forward(q, k, v, causal=causal, return_lse=True)
    own = torch.empty_like(q)
    stream = torch.cuda.current_stream().cuda_stream
    assert pkg.lib().flash_forward_noalloc(q.data_ptr(), k.data_ptr(), v.data_ptr(), own.data_ptr(), b, h, n, 64, 0.0,
                                           int(causal), -1, -1, stream, 0, 1) == pkg.FA_OK
    pkg.check(stream)
    for o in (out, again, own):
        assert torch.equal(o, want)
    exact_out, _ = exact(q[:1, :2], k[:1, :2], v[:1, :2], causal, -1, -1)
    assert (out[:1, :2].double() - exact_out).abs().max().item() < 4e-3  # as above


# Where a row's reference moves, O is rescaled; the short build does that behind the exponentials of the first 96 keys. Scores
# that grow from the last tile to the first move rows in every tile, in a spread of 4 in some.
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("n,causal,wl", [(300, False, -1), (640, False, -1), (1000, False, -1), (1024, True, -1),
                                         (2500, True, -1), (2700, True, -1), (2900, True, 500)])
@pytest.mark.parametrize("rising", [False, True])
def test_rows_whose_reference_moves(pkg, d, n, causal, wl, rising):
    import torch

    heads = 3 if n < 2000 else 40  # (whole pairs of q tiles and single ones)
    g = torch.Generator(device="cuda")
    g.manual_seed(n + d)
    q, k, v = (torch.randn(1, heads, n, d, device="cuda", generator=g) for _ in range(3))
    if rising:
        q, k = q.abs(), k * 0.1 + torch.linspace(6.0, -1.0, n, device="cuda")[:, None]
    else:
        q = q * 4
    q, k, v = q.half(), k.half(), v.half()
    kw = dict(causal=causal, window_left=wl)
    out = pkg.attention_forward(q, k, v, **kw)
    out2, lse = pkg.attention_forward(q, k, v, return_lse=True, **kw)
    pkg.check(torch.cuda.current_stream().cuda_stream)
    want, want_lse = exact(q[:, -2:], k[:, -2:], v[:, -2:], causal, wl, -1)
    for o in (out, out2):
        # P and the output rounded to fp16, 2^-11 each, where one key has all the weight
        assert ((o[:, -2:].double() - want).norm() / want.norm()).item() < 2.0 ** -10
        assert (o[:, -2:].double() - want).abs().max().item() < 6e-3  # the same of |v| < 6
    # scores of up to about 6 * d / sqrt(d) in fp32, 2^-24 of them per product and add
    assert ((lse[:, -2:].double() - want_lse).abs() / (1 + want_lse.abs())).max().item() < 2e-5
