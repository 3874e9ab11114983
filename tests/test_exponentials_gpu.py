"""The exponentials of a kv tile, column by column: some are taken on the special-function unit, some by a polynomial on
the FMA pipe, and no result may tell which. Scores are set one by one: q_i = (r_i, 0, ...), k_j = (x_j, 0, ...), so that
score (i, j) is scale * r_i * x_j exactly, and head h has its key under test in column h of the tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE, N = 128, 256  # two kv tiles without a mask: keys 128..255 are visited first and set every row's reference


def build(d, fill, set_key, rng):
    q = np.zeros((1, TILE, N, d), np.float16)
    k = np.zeros_like(q)
    q[..., 0] = rng.uniform(0.25, 1.0, (1, TILE, N)).astype(np.float16)
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
    return out.cpu().numpy().astype(np.float64), lse.cpu().numpy().astype(np.float64)


def exact(q, k, v):
    s = q[..., 0].astype(np.float64)[..., :, None] * k[..., 0].astype(np.float64)[..., None, :]
    top = s.max(-1, keepdims=True)
    p = np.exp(s - np.where(np.isfinite(top), top, 0.0))
    total = p.sum(-1, keepdims=True)
    with np.errstate(divide="ignore", invalid="ignore"):
        lse = np.log(total)[..., 0] + top[..., 0]
        out = np.where(total > 0, p @ v.astype(np.float64) / total, 0.0)
    return out, lse


@pytest.mark.parametrize("d", [64, 128])
def test_every_column_has_the_exponential_to_fp32_precision(pkg, d):
    rng = np.random.default_rng(5 + d)

    def set_key(x, h):
        x[TILE + 7] = 0.0                      # the reference
        x[h] = -rng.uniform(0.0, 16.0)         # the key under test, all others at e^-50 and below
    q, k, v = build(d, -200.0, set_key, rng)
    out, lse = run(pkg, q, k, v)
    want_out, want_lse = exact(q, k, v)
    # ln(1 + e^-f): 2.4e-7 for the exponential, as much for the logarithm and its product with ln 2, in fp32
    assert np.abs(lse - want_lse).max() < 1e-6
    # P rounded to fp16 (2^-11 of a probability of at most one half) and the output rounded to fp16
    assert np.abs(out - want_out).max() < np.abs(v).max() * 2.0 ** -11 + 2.0 ** -10


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("hidden", ["one key", "the tile visited first", "all keys"])
def test_scores_of_minus_infinity_vanish(pkg, d, hidden):
    rng = np.random.default_rng(9 + d)

    def set_key(x, h):
        x[:] = rng.standard_normal(N) - 40.0   # far below the reference of 0 that a row starts with
        if hidden == "one key":
            x[h] = -np.inf
        elif hidden == "all keys":
            x[:] = -np.inf
        else:
            x[TILE:] = -np.inf
    q, k, v = build(d, 0.0, set_key, rng)
    out, lse = run(pkg, q, k, v)
    want_out, want_lse = exact(q, k, v)
    if hidden == "all keys":
        assert np.all(out == 0) and np.all(lse == -np.inf)
    else:
        assert np.abs(lse - want_lse).max() < 1e-5   # fp32 sums of 128 to 255 terms, values near -15
        assert np.abs(out - want_out).max() < 2e-3


@pytest.mark.parametrize("d", [64, 128])
def test_nan_reaches_the_output_from_every_column(pkg, d):
    rng = np.random.default_rng(13 + d)

    def set_key(x, h):
        x[:] = rng.standard_normal(N)
        x[h] = np.nan
    q, k, v = build(d, 0.0, set_key, rng)
    out, _ = run(pkg, q, k, v)  # (a row sum of NaN gives a log-sum-exp of -inf, as one of 0 does)
    assert np.isnan(out).all()
