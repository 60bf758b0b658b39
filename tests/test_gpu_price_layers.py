"""The pricing layers' quantization by the last CTA of each 1024-rank block, and the sums formed before the
layer waits for the one before: layers of one block, of a ragged last block and of many (n = 9, 12, 17),
lists and rows scanned, two residuals in turn on one pricer (the blocks' counters start at zero again)."""
import numpy as np
import pytest

import oracle as O
from rumb import _lib
from rumb.instances import mixture_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,density", [(9, 0.5), (12, 0.05), (17, 0.002)])
@pytest.mark.parametrize("mode", ["u16", "u24", "f32"])
def test_layers_match_oracle_in_turn(ctx, monkeypatch, n, density, mode):
    monkeypatch.setenv("RUMB_STREAM_FORM", "layer")
    m, a, p = mixture_instance(n, density, K=8, N=100, seed=n)
    menus, _, p32, offsets, _ = O.cg_layout(n, m, a, p)
    rng = np.random.default_rng(n)
    scores = [rng.normal(0, 0.1, p32.size).astype(np.float32) for _ in range(2)]
    want = [O.price_stream(n, menus, s, offsets, mode=mode) for s in scores]
    for lists in (True, False):
        pr = _lib.Pricer(ctx, n, menus, offsets, mode=mode, lists=lists, stream=mode == "f32")
        for s, (v, r, mg, steps) in (list(zip(scores, want)) * 2):
            got = pr.price(s, want_steps=True)
            assert got[0] == v and got[2] == mg
            np.testing.assert_array_equal(got[1], r)
            np.testing.assert_array_equal(got[3], steps)
        pr.close()


def test_ranking_columns_at_word_edges(ctx):
    """A ranking's column for 1, 63, 64, 65 and 2,000 rows (a lane per row, two ballots a word)."""
    n = 8
    m, a, p = mixture_instance(n, 1.0, K=5, N=50, seed=3)
    for rows in (1, 63, 64, 65, m.size):
        menus, alts, p32, offsets, _ = O.cg_layout(n, m[:rows], a[:rows], p[:rows])
        pr = _lib.Pricer(ctx, n, menus, offsets, mode="mask")
        cg = _lib.CgMaster(pr, alts, p32.astype(np.float64), 4)
        for seed in range(3):
            rank = np.random.default_rng(seed).permutation(n).astype(np.int32)
            bits = cg.add_column(rank_pos=rank)[1]
            got = np.unpackbits(bits.view(np.uint8), bitorder="little")[:rows].astype(bool)
            np.testing.assert_array_equal(got, np.asarray(O.ranking_column(n, menus, alts, rank)).astype(bool))
        cg.close()
        pr.close()


def _edge_menus(n, rng):
    """Alternatives with 0, 1, 31, 32, 33, 64 and 65 rows in turn."""
    counts = [0, 1, 31, 32, 33, 64, 65]
    menus, offsets = [], [0]
    for x in range(n):
        sets = set()
        while len(sets) < counts[x % len(counts)]:
            d = rng.random(n) < rng.choice([0.1, 0.3, 0.6])
            d[x] = True
            sets.add(int(sum(1 << int(i) for i in np.nonzero(d)[0])))
        menus += sorted(sets)
        offsets.append(len(menus))
    return np.array(menus, np.uint64), np.array(offsets, np.int64)


@pytest.mark.parametrize("n", [9, 11, 22])
def test_tile_row_pass_at_batch_edges(ctx, monkeypatch, n):
    """The tile sweep's row pass reads 32 rows at a time: alternatives with 0, 1, 31, 32, 33, 64 and 65 rows,
    few low bits and few high bits per menu, split tiles (n = 9, 11) and a warp per tile (n = 22), bit for bit
    the oracle's sweep (n <= 11) or the layer kernels' (n = 22), also with scores of one sign and with zeros."""
    rng = np.random.default_rng(n)
    menus, offsets = _edge_menus(n, rng)
    pr = {}
    for form in ("tile", "layer"):
        monkeypatch.setenv("RUMB_MASK_FORM", form)
        pr[form] = _lib.Pricer(ctx, n, menus, offsets, mode="mask")
        monkeypatch.delenv("RUMB_MASK_FORM")
    base = rng.standard_normal(menus.size).astype(np.float32)
    for s in (base, -np.abs(base), np.where(rng.random(menus.size) < 0.5, np.float32(0), base)):
        v, r, _ = pr["tile"].price(s)
        want = O.price_mask(n, menus, s, offsets) if n <= 11 else pr["layer"].price(s)[:2]
        assert v == want[0]
        np.testing.assert_array_equal(r, want[1])
    for p in pr.values():
        p.close()


@pytest.mark.parametrize("mode", ["u16", "f32"])
def test_group_row_pass_at_batch_edges(ctx, monkeypatch, mode):
    """The group sweep's row pass (32 rows at a time) on the same menus at n = 13: the layer kernels' value and
    ranking, and their float64 maximum, bit for bit."""
    n, rng, got = 13, np.random.default_rng(13), {}
    menus, offsets = _edge_menus(n, rng)
    s = rng.standard_normal(menus.size).astype(np.float32)
    for form in ("group", "layer"):
        monkeypatch.setenv("RUMB_STREAM_FORM", form)
        pr = _lib.Pricer(ctx, n, menus, offsets, mode=mode, stream=mode == "f32")
        v, r, _ = pr.price(s)
        got[form] = (v, r.tolist(), pr.max64(s.astype(np.float64)))
        pr.close()
    assert got["group"] == got["layer"]
