"""The exponentials of a kv tile, column by column: some are taken on the special-function unit, some by a polynomial on
the FMA pipe, and no result may tell which. Scores are set one by one: q_i = (r_i, 0, ...), k_j = (x_j, 0, ...), so that
score (i, j) is scale * r_i * x_j exactly, and head h has its key under test in column h of the tile."""
import numpy as np
import pytest

from conftest import rules_args

pytestmark = pytest.mark.gpu

TILE = 128
# Rows, tile that holds the keys under test, and the build that the launch takes. Tiles are visited from the last to the first;
# the first keys (tile 0) have a rule of their own, and no tile under test is cut or the first that is visited.
CASES = [(256, 0, "short"), (1000, 3, "short"), (768, 0, "long"), (768, 2, "long")]


@pytest.fixture(params=[(*c, d) for c in CASES for d in (64, 128)], ids=lambda c: "n%d-tile%d-%s-d%d" % c)
def case(request, wi):
    n, tile, build_name, d = request.param
    args = rules_args(TILE, n, d)
    assert bool(wi.short_build(args, 0)) == (build_name == "short")
    if n == 1000:  # at head_dim 64 the plain launch of this one gives P columns of its own
        assert wi.own_p(args)
    return n, tile * TILE, d


def last_tile(n):
    return (n - 1) // TILE * TILE


def build(n, d, fill, set_key, rng):
    q = np.zeros((1, TILE, n, d), np.float16)
    k = np.zeros_like(q)
    q[..., 0] = rng.uniform(0.25, 1.0, (1, TILE, n)).astype(np.float16)
    k[..., 0] = fill
    for h in range(TILE):
        set_key(k[0, h, :, 0], h)
    v = rng.standard_normal(q.shape).astype(np.float16)
    return q, k, v


def run(pkg, q, k, v):
    import torch

    t = [torch.from_numpy(a).cuda() for a in (q, k, v)]
    out, lse = pkg.attention_forward(*t, softmax_scale=1.0, return_lse=True)
    plain = pkg.attention_forward(*t, softmax_scale=1.0)
    pkg.check(torch.cuda.current_stream().cuda_stream)
    # (NaN is NaN whatever its bits; the plain kernel is a build of its own)
    assert torch.equal(torch.isnan(out), torch.isnan(plain))
    assert torch.allclose(out.float(), plain.float(), rtol=1e-3, atol=1e-4, equal_nan=True)
    return out.double(), lse.double()


def exact(q, k, v):
    import torch

    q, k, v = (torch.from_numpy(a).cuda().double() for a in (q, k, v))
    s = q[..., 0][..., :, None] * k[..., 0][..., None, :]
    top = s.amax(-1, keepdim=True)
    p = s.sub_(torch.where(top.isfinite(), top, 0.0)).exp_()
    total = p.sum(-1, keepdim=True)
    return torch.where(total > 0, p @ v / total, 0.0), total.log()[..., 0] + top[..., 0]


def test_every_column_has_the_exponential_to_fp32_precision(pkg, case):
    n, first, d = case
    rng = np.random.default_rng(5 + d)

    def set_key(x, h):
        x[last_tile(n) + 7] = 0.0               # the reference
        x[first + h] = -rng.uniform(0.0, 16.0)  # the key under test, all others at e^-50 and below
    q, k, v = build(n, d, -200.0, set_key, rng)
    out, lse = run(pkg, q, k, v)
    want_out, want_lse = exact(q, k, v)
    # ln(1 + e^-f): 2.4e-7 for the exponential, as much for the logarithm and its product with ln 2, in fp32
    assert (lse - want_lse).abs().max() < 1e-6
    # P rounded to fp16 (2^-11 of a probability of at most one half) and the output rounded to fp16
    assert (out - want_out).abs().max() < np.abs(v).max() * 2.0 ** -11 + 2.0 ** -10


@pytest.mark.parametrize("hidden", ["one key", "the tile visited first", "all keys"])
def test_scores_of_minus_infinity_vanish(pkg, case, hidden):
    n, first, d = case
    rng = np.random.default_rng(9 + d)

    def set_key(x, h):
        x[:] = rng.standard_normal(n) - 40.0   # far below the reference of 0 that a row starts with
        if hidden == "one key":
            x[first + h] = -np.inf
        elif hidden == "all keys":
            x[:] = -np.inf
        else:
            x[last_tile(n):] = -np.inf
    q, k, v = build(n, d, 0.0, set_key, rng)
    out, lse = run(pkg, q, k, v)
    want_out, want_lse = exact(q, k, v)
    if hidden == "all keys":
        assert (out == 0).all() and (lse == -np.inf).all()
    else:
        assert (lse - want_lse).abs().max() < 1e-5   # fp32 sums of 128 to 999 terms, values near -15
        assert (out - want_out).abs().max() < 2e-3


def test_nan_reaches_the_output_from_every_column(pkg, case):
    n, first, d = case
    rng = np.random.default_rng(13 + d)

    def set_key(x, h):
        x[:] = rng.standard_normal(n)
        x[first + h] = np.nan
    q, k, v = build(n, d, 0.0, set_key, rng)
    out, _ = run(pkg, q, k, v)  # (a row sum of NaN gives a log-sum-exp of -inf, as one of 0 does)
    assert out.isnan().all()
