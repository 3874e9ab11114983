"""CPU tests of the persistent kernel's work items (csrc/work_items.h, compiled here for the host): every q tile is handed
out exactly once with exactly its visible kv tiles, and the hand-over of items through the two-slot ring ends for every
order in which a CTA may claim them."""
import ctypes
import itertools
import random

import pytest

SMS = 148


class Launch:
    def __init__(self, wi, bh, n, d=64, causal=False, wl=-1, wr=-1, first=0, total=0):
        self.wi, self.args = wi, (ctypes.c_int * 9)(bh, n, d, int(causal), wl, wr, SMS, first, total or bh)
        out = (ctypes.c_int * 3)()
        wi.plan(self.args, out)
        self.items, self.pair_items, self.group = out

    def walk(self, item, claims):
        out = (ctypes.c_int * 16)()
        claims = (ctypes.c_int * (len(claims) + 1))(*claims, self.items)
        used = self.wi.walk(self.args, item, claims, out)
        keys = ("item", "head", "r0a", "r1a", "loa", "hia", "r0b", "r1b", "lob", "hib", "top", "steps", "split")
        return dict(zip(keys, out)), used

    def published(self, first, claims):
        """What one CTA publishes to its roles when it starts with `first` and its claims are answered by `claims`."""
        out, at, item = [], 0, first
        while True:
            g, used = self.walk(item, claims[at:])
            at += used
            if g["item"] < 0:
                return out
            out.append(g)
            item = claims[at] if at < len(claims) else self.items
            at += 1


SHAPES = [
    dict(bh=100, n=300), dict(bh=111, n=300), dict(bh=123, n=600), dict(bh=75, n=333), dict(bh=3, n=129),
    dict(bh=1, n=100), dict(bh=2, n=129, causal=True), dict(bh=80, n=450, causal=True, wl=60),
    dict(bh=5, n=1000, wl=100, wr=5), dict(bh=8, n=2304 + 77, causal=True),
    dict(bh=40, n=4097, causal=True), dict(bh=7, n=700, wl=50), dict(bh=96, n=1000),
    # window, last pairs split; causal with several head groups; causal, all pairs split; slabs of such problems
    dict(bh=152, n=1000, d=128, wl=100, wr=0), dict(bh=64, n=4101, d=128, causal=True), dict(bh=8, n=4096, causal=True),
    dict(bh=5, n=512, first=70, total=75), dict(bh=5, n=2048, causal=True, first=0, total=40),
]


@pytest.mark.parametrize("shape", [s for s in SHAPES if "total" not in s], ids=str)
def test_head_group_is_the_launch_s(wi, pkg, shape):
    s = {"d": 64, "causal": False, "wl": -1, "wr": -1, **shape}
    assert pkg.head_group(s["bh"], s["n"], s["d"], s["causal"], s["wl"], s["wr"], SMS) == Launch(wi, **shape).group


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_every_q_tile_once_with_its_kv_tiles(wi, pkg, shape):
    L = Launch(wi, **shape)
    n, causal = shape["n"], shape.get("causal", False)
    wl, wr = shape.get("wl", -1), shape.get("wr", -1)
    seen = {}
    for item in range(L.items):
        g, _ = L.walk(item, [])
        if g["item"] != item:  # an item without rows: skipped, and the stand-in claim ended the walk
            assert g["item"] == -1 and item >= L.pair_items
            continue
        tiles = {}
        for s, (r0, r1, lo, hi) in enumerate([(g["r0a"], g["r1a"], g["loa"], g["hia"]),
                                              (g["r0b"], g["r1b"], g["lob"], g["hib"])]):
            assert r1 >= r0 or lo == hi
            for t in range(lo, hi):
                tiles.setdefault(r0, []).append(g["top"] - 2 * t - s if g["split"] else g["top"] - t)
                assert 0 <= t < g["steps"] and r1 >= r0
        assert tiles
        for r0, js in tiles.items():
            assert (g["head"], r0) not in seen
            seen[g["head"], r0] = js
    assert set(seen) == set(itertools.product(range(shape["bh"]), range(0, n, 128)))
    for (_, r0), js in seen.items():
        lo, hi, _ = pkg.kv_range(n, causal, wl, wr, r0, min(r0 + 128, n) - 1)
        assert sorted(js) == list(range(lo, hi))


@pytest.mark.parametrize("shape", [
    dict(n=512, total=75), dict(n=333, total=75), dict(n=2048, total=40, causal=True), dict(n=4096, total=9, causal=True),
    dict(n=8192, total=32, d=128, causal=True), dict(n=1000, total=152, wl=100, wr=0),
    dict(n=4096, total=10, causal=True, wl=500),
    dict(n=900, total=41, wl=60), dict(n=4096, total=30), dict(n=4096, total=40, d=128, causal=True, wl=512),
    dict(n=2048, total=223, d=128, causal=True, wl=500), dict(n=1500, total=7, wl=128, wr=128),
], ids=str)
def test_slabs_take_the_same_pairs_apart(wi, shape):
    """Whether a q tile is summed by one stage or by two does not depend on how the heads are cut into calls that know the
    whole problem (the bits of flash_forward_host and flash_forward_multi_gpu)."""
    def split_tiles(**kw):
        L = Launch(wi, **{**shape, **kw})
        geoms = (L.walk(i, [])[0] for i in range(L.items))
        return {(kw["first"] + g["head"], g["r0a"]) for g in geoms if g["item"] >= 0 and g["split"]}

    total = shape["total"]
    whole = split_tiles(bh=total, first=0)
    for step in (1, 3, 8, total - 1):
        parts = [split_tiles(bh=min(step, total - h), first=h) for h in range(0, total, step)]
        assert set().union(*parts) == whole


def ring_ends(rows):
    """The hand-over of items between the roles of a CTA, as the kernel does it at head_dim 64. `rows[i]`: published item i
    has rows. Two slots; the producer fills one again when every reader has taken it. The issuing warp takes the next item
    with rows (or the end) before it commits the last product of the current one; the epilogue warps take an item and
    wait for that commit before they take another. Returns whether everybody reaches the end."""
    end = len(rows)  # the end marker is published like an item
    published = issuer = corr = 0  # items published / taken
    current, committed = None, set()
    issuer_done = corr_done = False
    waiting = None
    while True:
        before = (published, issuer, corr, len(committed), issuer_done, corr_done, current, waiting)
        if published <= end and min(issuer, corr) >= published - 1:  # the slot of item published - 2 has been read
            published += 1
        if not issuer_done and issuer < published:
            i = issuer
            issuer += 1
            if i == end or rows[i]:
                if current is not None:
                    committed.add(current)
                current = i
                issuer_done = i == end
        if waiting is not None and waiting in committed:
            waiting = None
        if waiting is None and not corr_done and corr < published:
            if corr == end:
                corr_done = True
            elif rows[corr]:
                waiting = corr
            corr += 1
        if (published, issuer, corr, len(committed), issuer_done, corr_done, current, waiting) == before:
            return issuer_done and corr_done


def test_ring_model_sees_the_cycle_of_row_less_items():
    assert ring_ends([True] * 5) and ring_ends([]) and ring_ends([True, False, True]) and ring_ends([False, False])
    assert not ring_ends([True, False, False]) and not ring_ends([True, False, False, True])


@pytest.mark.parametrize("shape", [s for s in SHAPES if (s["n"] - 1) % 256 < 128], ids=str)
def test_item_hand_over_ends_for_every_claim_order(wi, shape):
    """One CTA starts with any item and then gets any rising sequence of the others (the rest goes to CTAs that run beside
    it): whatever it publishes must let all its roles reach the end."""
    L = Launch(wi, **shape)
    rng = random.Random(5)
    row_less = [i for i in range(L.pair_items, L.items) if L.walk(i, [])[0]["item"] < 0]
    orders = [[]]
    if row_less:
        orders += [row_less, row_less[:2], [0] + row_less[:3] + [L.items - 1]]
    for _ in range(40):
        orders.append(sorted(rng.sample(range(L.items), min(L.items, rng.randint(1, 8)))))
    for order in orders:
        for first in {0, order[0] if order else 0}:
            pub = L.published(first, [i for i in order if i != first])
            assert ring_ends([g["steps"] > 0 for g in pub])
            assert all(g["steps"] > 0 for g in pub)
            assert [g["item"] for g in pub] == [i for i in [first] + [i for i in order if i != first] if i not in row_less]


@pytest.mark.parametrize("heads,n,causal,wl,wr,split", [
    (37, 512, True, -1, -1, True), (38, 512, True, -1, -1, False),          # half a pair per CTA
    (28, 768, True, -1, -1, True), (36, 768, True, -1, -1, False),
    (24, 1000, True, -1, -1, True), (32, 1024, True, -1, -1, False),        # one wave of pairs against two of singles
    (40, 1024, True, -1, -1, True), (60, 1024, True, -1, -1, False),        # two waves of pairs
    (36, 2048, True, -1, -1, True), (40, 2048, True, -1, -1, False), (36, 2048, False, -1, 0, True),
    (10, 8192, True, -1, -1, True), (12, 8192, True, -1, -1, False), (1, 32768, True, -1, -1, True),
    (8, 128, True, -1, -1, False),                                          # one tile
])
def test_which_launches_take_their_pairs_apart(wi, heads, n, causal, wl, wr, split):
    launch = Launch(wi, heads, n, causal=causal, wl=wl, wr=wr)
    pairs = heads * -(-n // 256)
    assert launch.items == pairs * (2 if split else 1) and launch.pair_items == (0 if split else pairs)
