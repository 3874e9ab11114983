"""The work this library is used for, as cases that can be timed and compared.

A case names an entry point (`call`), a problem shape and the options of the attention. `prepare` makes what a caller
holds before the call (fp16 Q, K, V on the GPU, or in pinned host memory for the host-buffer call), `run` makes one
call of the public entry point, `work` counts what the problem itself needs.

The value that a case gives as `spread` is the standard deviation of the scaled scores: 1 for i.i.d. N(0, 1) tensors,
more for the peaked rows of a trained model, where the running maximum of a row keeps moving.
"""
import importlib
import math

import torch

fa = importlib.import_module("flash-attn-rtx5060_b200")

WINDOW_NONE = -1


def _case(name, call, batch, heads, seqlen, head_dim, causal, window_left=WINDOW_NONE, window_right=WINDOW_NONE,
          dropout=0.0, chunk_heads=0, spread=1.0):
    return {"name": name, "call": call, "batch": batch, "heads": heads, "seqlen": seqlen, "head_dim": head_dim,
            "causal": causal, "window_left": window_left, "window_right": window_right, "dropout": dropout,
            "chunk_heads": chunk_heads, "spread": spread}


def listed():
    return [
        # One small layer call: latency is all that counts (the smallest configuration of the benchmark).
        _case("small_full_d64", "forward", 1, 4, 512, 64, False),
        # A short ragged prompt in a latency-critical loop that must not allocate.
        _case("prompt_noalloc_d128", "noalloc", 1, 8, 333, 128, True, spread=2.0),
        # A batch of ragged encoder inputs, no mask.
        _case("encoder_ragged_d64", "forward", 8, 12, 1000, 64, False, spread=2.0),
        # Medium decoder batch with 64-wide heads.
        _case("decoder_d64", "forward", 4, 16, 2048, 64, True),
        # Long decoder context with 128-wide heads: the library's main configuration.
        _case("decoder_d128", "forward", 2, 32, 8192, 128, True),
        # The same without a mask (encoder, diffusion transformer) at half the length.
        _case("encoder_d128", "forward", 2, 16, 4096, 128, False),
        # Sliding-window decoder.
        _case("window_d128", "forward", 4, 16, 16384, 128, True, window_left=1024),
        # Long context: one GPU's eighth of the benchmark's 512 heads of 32768 rows.
        _case("long_context_d128", "forward", 1, 64, 32768, 128, True),
        # ALiBi-biased decoder.
        _case("alibi_d64", "alibi", 2, 16, 4096, 64, True),
        # A training forward, or one part of a key-split attention: output and log-sum-exp, ragged length.
        _case("training_lse_d128", "lse", 1, 24, 4001, 128, True, spread=2.0),
        # A training forward with dropout on the probabilities.
        _case("dropout_d64", "dropout", 4, 16, 2048, 64, True, dropout=0.1),
        # Tensors that live in pinned host memory: upload, attention and download as one call.
        _case("host_buffers_d128", "host", 1, 32, 8192, 128, True, chunk_heads=8),
    ]


def _visible_pairs(case):
    """Visible (query, key) pairs of one head."""
    n, wl, wr = case["seqlen"], case["window_left"], case["window_right"]
    if case["causal"]:
        wr = 0
    if wl < 0 and wr < 0:
        return n * n
    left = n if wl < 0 else wl
    right = n if wr < 0 else wr
    pairs = n  # the diagonal
    for w in (min(left, n - 1), min(right, n - 1)):
        pairs += w * n - w * (w + 1) // 2  # sum over rows of min(rows on that side, w)
    return pairs


def work(case):
    bh, n, d = case["batch"] * case["heads"], case["seqlen"], case["head_dim"]
    nbytes = 4 * 2 * bh * n * d
    if case["call"] == "lse":
        nbytes += 4 * bh * n
    return {"bytes": nbytes, "flops": 4 * d * bh * _visible_pairs(case)}


def tolerance(case):
    # fp16 inputs, probabilities and outputs with fp32 sums: against an fp64 evaluation the outputs of the listed cases
    # differ by 2.3e-4 .. 2.9e-4 (2-norm, relative); about four times the largest of these.
    return {"rel": 1.2e-3}


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["forward", "forward", "forward", "forward", "noalloc", "alibi", "lse", "dropout", "host"])
    head_dim = rng.choice([64, 128])
    # bounds on the work of one call: the largest listed case's, less for the calls that are slower per operation
    most_flops = {"forward": 1.5e13, "noalloc": 1.5e13, "alibi": 4e12, "lse": 1.5e13, "dropout": 2e12, "host": 1.5e12}[call]
    most_bytes = 6e8 if call == "host" else 2.1e9
    while True:
        seqlen = log_int(64, 32768)
        if seqlen >= 256 and rng.random() < 0.5:
            seqlen -= seqlen % 128
        batch = log_int(1, 16)
        heads = log_int(1, 64)
        causal = rng.random() < 0.7
        window_left = window_right = WINDOW_NONE
        if call in ("forward", "noalloc", "lse") and seqlen >= 512 and rng.random() < 0.25:
            window_left = log_int(64, seqlen // 2)
            if not causal:
                window_right = window_left
        case = _case("drawn", call, batch, heads, seqlen, head_dim, causal, window_left, window_right,
                     dropout=rng.choice([0.1, 0.2]) if call == "dropout" else 0.0,
                     chunk_heads=min(8, batch * heads) if call == "host" else 0, spread=rng.choice([1.0, 1.0, 2.0]))
        w = work(case)
        if w["flops"] <= most_flops and w["bytes"] <= most_bytes:
            del case["name"]
            return case


def prepare(case, seed):
    shape = (case["batch"], case["heads"], case["seqlen"], case["head_dim"])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    q, k, v = (torch.randn(shape, generator=gen, device="cuda", dtype=torch.float16) for _ in range(3))
    if case["spread"] != 1.0:
        q *= case["spread"]
    state = {"case": case, "q": q, "k": k, "v": v}
    call = case["call"]
    if call == "alibi":  # the usual geometric slopes
        state["slopes"] = torch.tensor([2.0 ** (-8.0 * (h + 1) / case["heads"]) for h in range(case["heads"])],
                                       device="cuda", dtype=torch.float32)
    elif call == "noalloc":
        state["out"] = torch.empty_like(q)
    elif call == "dropout":
        state["seed"] = seed
    elif call == "host":
        for name in ("q", "k", "v"):
            state[name] = state[name].cpu().pin_memory()
        state["out"] = torch.empty(shape, dtype=torch.float16, pin_memory=True)
        nbytes = fa.host_workspace_bytes(case["seqlen"], case["head_dim"], case["chunk_heads"])
        state["workspace"] = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        state["workspace_bytes"] = nbytes
    return state


def run(state):
    case = state["case"]
    q, k, v = state["q"], state["k"], state["v"]
    call = case["call"]
    if call == "noalloc":
        out = state["out"]
        rc = fa.lib().flash_forward_noalloc(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), case["batch"],
                                            case["heads"], case["seqlen"], case["head_dim"], 0.0, int(case["causal"]),
                                            case["window_left"], case["window_right"],
                                            torch.cuda.current_stream().cuda_stream, 0, 0)
        if rc != fa.FA_OK:
            raise RuntimeError(fa.lib().flash_forward_last_error().decode())
        return out
    if call == "host":
        fa.flash_forward_host(q.data_ptr(), k.data_ptr(), v.data_ptr(), state["out"].data_ptr(), case["batch"],
                              case["heads"], case["seqlen"], case["head_dim"], state["workspace"].data_ptr(),
                              state["workspace_bytes"], case["chunk_heads"], is_causal=case["causal"])
        return state["out"]
    window = {"causal": case["causal"], "window_left": case["window_left"], "window_right": case["window_right"]}
    if call == "alibi":
        return fa.attention_forward(q, k, v, alibi_slopes=state["slopes"], **window)
    if call == "lse":
        return fa.attention_forward(q, k, v, return_lse=True, **window)
    if call == "dropout":
        return fa.attention_forward(q, k, v, dropout_p=case["dropout"], seed=state["seed"], **window)
    return fa.attention_forward(q, k, v, **window)


def _philox_keep(seed, head, rows, n, threshold):
    """Keep mask of the dropout call for a block of query rows: byte j % 16 of Philox-4x32-10 (key = seed,
    counter = {j / 16, row, head, 0}; Salmon et al. 2011) below `threshold`."""
    low = 0xFFFFFFFF

    def words(block, row):
        c = [block, row, torch.full_like(block, head), torch.zeros_like(block)]
        k = [seed & low, (seed >> 32) & low]
        for _ in range(10):
            a, b = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # 32 x 32 bits; the sign of the wrapped 64-bit product is masked off
            c = [((b >> 32) & low) ^ c[1] ^ k[0], b & low, ((a >> 32) & low) ^ c[3] ^ k[1], a & low]
            k = [(k[0] + 0x9E3779B9) & low, (k[1] + 0xBB67AE85) & low]
        return c

    block = torch.arange((n + 15) // 16, device=rows.device).expand(len(rows), -1)
    out = torch.stack(words(block, rows[:, None].expand_as(block)), dim=-1)  # [row][block][word]
    byte = torch.stack([(out >> (8 * t)) & 255 for t in range(4)], dim=-1)
    return byte.reshape(len(rows), -1)[:, :n] < threshold


def exact(case, seed):
    """The attention of the same inputs in 64 bits."""
    state = prepare(case, seed)
    n, d, heads, call = case["seqlen"], case["head_dim"], case["heads"], case["call"]
    q, k, v = (state[x].cuda().view(-1, n, d) for x in "qkv")
    bh = q.shape[0]
    out = torch.empty((bh, n, d), dtype=torch.float64)
    lse = torch.empty((bh, n), dtype=torch.float64)
    wl, wr = case["window_left"], 0 if case["causal"] else case["window_right"]
    threshold = int(round(256 * (1 - case["dropout"])))
    step = max(1, min(n, (1 << 27) // n))
    for h in range(bh):
        kh, vh = k[h].double(), v[h].double()
        for r0 in range(0, n, step):
            rows = torch.arange(r0, min(n, r0 + step), device="cuda")
            lo = 0 if wl < 0 else max(0, r0 - wl)
            hi = n if wr < 0 else min(n, r0 + len(rows) + wr)
            cols = torch.arange(lo, hi, device="cuda")
            s = q[h, rows].double() @ kh[lo:hi].T / math.sqrt(d)
            gap = cols[None, :] - rows[:, None]
            if call == "alibi":
                s -= state["slopes"][h % heads].double() * gap.abs()
            if wl >= 0:
                s.masked_fill_(gap < -wl, -math.inf)
            if wr >= 0:
                s.masked_fill_(gap > wr, -math.inf)
            top = s.amax(dim=1, keepdim=True)
            p = s.sub_(top).exp_()
            total = p.sum(dim=1, keepdim=True)
            lse[h, rows.cpu()] = (top + total.log()).squeeze(1).cpu()
            if case["dropout"] > 0:
                p = p * _philox_keep(seed, h, rows, n, threshold)[:, lo:hi] * (256 / threshold)
            out[h, rows.cpu()] = (p @ vh[lo:hi] / total).cpu()
    out = out.view(case["batch"], heads, n, d)
    return (out, lse.view(case["batch"], heads, n)) if call == "lse" else out
