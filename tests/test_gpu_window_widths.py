"""Signature joins whose longest probes fill their signatures and take wider
ones (256, then 512 bits): every starting width, both verification modes, probe
ranges across the border between two widths, R-S windows, repeated calls."""
import numpy as np
import pytest

import oracle
from hyset_gb300 import synth

pytestmark = pytest.mark.gpu


def _set(pairs):
    s = oracle.as_set(pairs)
    assert len(s) == len(pairs), "duplicate pairs"
    return s


@pytest.mark.parametrize("bits", [64, 128, 256, 512])
@pytest.mark.parametrize("sim,tau", [("jaccard", 0.6), ("cosine", 0.75)])
def test_self_join_widths(ctx, bits, sim, tau):
    c = synth.generate(synth.C3, n_sets=12_001, universe=12_000, seed=5)
    coll = ctx.upload(c.tokens, c.sizes, c.starts)
    want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, tau, sim=sim))
    kw = dict(threshold=tau, sim=sim, technique="bitmap", bitmap=bits)
    one = ctx.self_join(coll, **kw)
    assert one.bitmap_bits == bits and _set(one.pairs) == want
    assert _set(ctx.self_join(coll, verify_mode=2, **kw).pairs) == want
    lo, hi = 4_003, 11_999
    assert _set(ctx.self_join(coll, probe_range=(lo, hi), **kw).pairs) == {p for p in want if lo <= p[0] < hi}


@pytest.mark.parametrize("bits", [64, 128])
def test_rs_join_widths(ctx, bits):
    c = synth.generate(synth.C3, n_sets=14_000, universe=9_000, seed=6)
    side = np.random.default_rng(1).random(c.n) < 0.4
    colls = []
    for mask in (side, ~side):
        ids = np.nonzero(mask)[0]
        tokens = np.concatenate([c.set(i) for i in ids])
        sizes = c.sizes[ids]
        starts = np.concatenate([[0], np.cumsum(sizes.astype(np.int64))])[:-1].astype(np.uint32)
        colls.append(ctx.upload(tokens, sizes, starts))
    all_pairs = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.55))
    # the self-join's pairs with one set on either side, in the halves' own numbers
    at = np.where(side, np.cumsum(side) - 1, np.cumsum(~side) - 1)
    want = set()
    for a, b in all_pairs:
        if side[a] != side[b]:
            r, s = (a, b) if side[a] else (b, a)
            want.add((int(at[s]), int(at[r])))
    got = ctx.rs_join(colls[0], colls[1], threshold=0.55, technique="bitmap", bitmap=bits)
    assert _set(got.pairs) == want
