"""The signature technique's tiled kernel (k_window) against the enumeration
kernel (which a call that collects work counters runs) and the oracle: every
signature width, both verification modes, tiles and segments with remainders,
sizes whose admissible distance takes every way of counting, R-S windows on
both sides of the probe, probe ranges."""
import numpy as np
import pytest

import oracle
from hyset_gb300 import synth

pytestmark = pytest.mark.gpu

BITS = [64, 128, 256, 512]


def _as_set(p):
    s = oracle.as_set(p)
    assert len(s) == len(p), "duplicate pairs"
    return s


@pytest.mark.parametrize("n", [1, 2, 31, 33, 63, 65, 129, 1000, 1025, 9001])
@pytest.mark.parametrize("bits", BITS)
def test_self_join_sizes(ctx, n, bits):
    c = synth.generate(synth.C1, n_sets=n, universe=300, dup_frac=0.2, dup_edit_hi=0.3, seed=n + bits)
    coll = ctx.upload(c.tokens, c.sizes, c.starts)
    want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.6))
    for mode in (1, 2):
        kw = dict(threshold=0.6, technique="bitmap", bitmap=bits, verify_mode=mode)
        assert _as_set(ctx.self_join(coll, **kw).pairs) == want
        old = ctx.self_join(coll, collect_stats=True, **kw)
        assert _as_set(old.pairs) == want
    lo, hi = n // 3, n - n // 4
    if lo < hi:
        part = ctx.self_join(coll, threshold=0.6, technique="bitmap", bitmap=bits, probe_range=(lo, hi))
        assert _as_set(part.pairs) == {p for p in want if lo <= p[0] < hi}


@pytest.mark.parametrize("sim", ["jaccard", "cosine", "dice"])
@pytest.mark.parametrize("bits", BITS)
def test_long_and_mixed_sizes(ctx, sim, bits):
    # sizes 10..2000: admissible distances from a few bits to more than the signature holds
    c = synth.generate(synth.C3, n_sets=6000, universe=20000, seed=91)
    coll = ctx.upload(c.tokens, c.sizes, c.starts)
    for tau in (0.5, 0.8, 1.0):
        kw = dict(threshold=tau, sim=sim, technique="bitmap", bitmap=bits)
        want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, tau, sim=sim))
        assert _as_set(ctx.self_join(coll, **kw).pairs) == want
        assert ctx.self_join(coll, count_only=True, **kw).count == len(want)


@pytest.mark.parametrize("sim", ["jaccard", "cosine", "dice"])
@pytest.mark.parametrize("orientation", ["as_given", "swapped"])
def test_rs_windows(ctx, sim, orientation):
    R = synth.generate(synth.C1, n_sets=1501, universe=900, dup_frac=0.0, seed=21)
    S = synth.generate(synth.C1, n_sets=777, universe=900, seed=22)
    # some of R's sets on both sides
    S_t = np.concatenate([S.tokens] + [R.set(i) for i in range(0, R.n, 7)])
    S_z = np.concatenate([S.sizes, R.sizes[::7]])
    S_s = np.concatenate([[0], np.cumsum(S_z.astype(np.int64))])[:-1]
    order = np.argsort(S_z, kind="stable")
    S_t = np.concatenate([S_t[S_s[i]:S_s[i] + S_z[i]] for i in order])
    S_z = S_z[order].astype(np.uint32)
    S_s = np.concatenate([[0], np.cumsum(S_z.astype(np.int64))])[:-1].astype(np.uint32)
    want = oracle.as_set(oracle.brute_rs((R.tokens, R.starts, R.sizes), (S_t, S_s, S_z), 0.6, sim=sim))
    r, s = ctx.upload(R.tokens, R.sizes, R.starts), ctx.upload(S_t, S_z, S_s)
    for bits in BITS:
        got = ctx.rs_join(r, s, threshold=0.6, sim=sim, technique="bitmap", bitmap=bits, orientation=orientation)
        assert _as_set(got.pairs) == want
