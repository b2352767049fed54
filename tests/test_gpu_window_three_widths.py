"""Signature joins in three launches: the probes that fill their signatures
take 256 bits, those that fill these 512.  The launches are counted against the
rule that cuts the probes, restated here, so an input that no longer reaches
all three fails; results against the oracle, over the whole range and over
probe ranges that begin and end around either border."""
import math

import numpy as np
import pytest

import oracle
from hyset_gb300 import similarity, synth

pytestmark = pytest.mark.gpu

WIDE_PAIRS = 16 << 20


def _cut(sizes, indexed, sim, tau, words, lo=0, hi=None):
    """(widths signed, probe ranges launched) of a join of `words`-word signatures."""
    hi = len(sizes) if hi is None else hi
    ranges = [(words, lo, hi)]
    while max(4, 2 * ranges[-1][0]) <= 8:
        bits, l = 64 * ranges[-1][0], int(sizes.max()) + 1
        while l > 1:  # the first size from which on all are filled
            e = 0.5 * bits * (1.0 - math.exp(-4.0 * (l - 1) / bits))
            most = 2 * (l - 1) - 2 * similarity.minoverlap(sim, l - 1, l - 1, tau)
            if most < e - 2.0 * math.sqrt(e * (1.0 - e / bits)):
                break
            l -= 1
        at = max(lo, min(hi, int(np.searchsorted(sizes, l))))
        if at >= hi:
            break
        least = similarity.minsize(sim, int(sizes[at]), tau)
        if (hi - at) * (len(indexed) - int(np.searchsorted(indexed, least))) < WIDE_PAIRS:
            break
        w, a, _ = ranges[-1]
        ranges[-1] = (w, a, at)
        ranges.append((max(4, 2 * w), at, hi))
    return len(ranges), [r for r in ranges if r[1] < r[2]]


def _set(pairs):
    s = oracle.as_set(pairs)
    assert len(s) == len(pairs), "duplicate pairs"
    return s


@pytest.mark.parametrize("bits", [64, 128, 256, 512])
@pytest.mark.parametrize("sim,tau", [("jaccard", 0.5), ("cosine", 0.7), ("dice", 0.7)])
def test_self_join_in_three_widths(ctx, bits, sim, tau):
    c = synth.generate(synth.C3, n_sets=24_001, universe=24_000, seed=5)
    coll = ctx.upload(c.tokens, c.sizes, c.starts)
    want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, tau, sim=sim))
    widths, ranges = _cut(c.sizes, c.sizes, sim, tau, bits // 64)
    assert [r[0] * 64 for r in ranges] == {64: [64, 256, 512], 128: [128, 256, 512], 256: [256, 512], 512: [512]}[bits]
    kw = dict(threshold=tau, sim=sim, technique="bitmap", bitmap=bits)
    for mode in (1, 2):
        got = ctx.self_join(coll, verify_mode=mode, **kw)
        assert got.launches == widths + len(ranges)
        assert got.bitmap_bits == bits and _set(got.pairs) == want
    for _, border, _ in ranges[1:] or [(0, 12_000, 0)]:
        for lo, hi in ((border - 3, c.n - 1), (border, c.n), (border + 1, border + 7_001), (border - 6_000, border),
                       (border - 6_000, border + 1)):
            lo, hi = max(lo, 0), min(hi, c.n)
            got = ctx.self_join(coll, probe_range=(lo, hi), **kw)
            w, parts = _cut(c.sizes, c.sizes, sim, tau, bits // 64, lo, hi)
            assert got.launches == w + len(parts)
            assert _set(got.pairs) == {p for p in want if lo <= p[0] < hi}
    coll.free()


@pytest.mark.parametrize("bits", [64, 128])
def test_rs_join_in_three_widths(ctx, bits):
    tau = 0.5
    c = synth.generate(synth.C3, n_sets=40_000, universe=30_000, seed=6)
    side = np.random.default_rng(1).random(c.n) < 0.4
    colls, sizes = [], []
    for mask in (side, ~side):
        ids = np.nonzero(mask)[0]
        sizes.append(c.sizes[ids])
        starts = np.concatenate([[0], np.cumsum(sizes[-1].astype(np.int64))])[:-1].astype(np.uint32)
        colls.append(ctx.upload(np.concatenate([c.set(i) for i in ids]), sizes[-1], starts))
    widths, ranges = _cut(sizes[1], sizes[0], "jaccard", tau, bits // 64)
    assert len(ranges) == 3
    at = np.where(side, np.cumsum(side) - 1, np.cumsum(~side) - 1)  # in the halves' own numbers
    want = {(int(at[b]), int(at[a])) if side[a] else (int(at[a]), int(at[b]))
            for a, b in oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, tau)) if side[a] != side[b]}
    got = ctx.rs_join(colls[0], colls[1], threshold=tau, technique="bitmap", bitmap=bits, orientation="as_given")
    assert got.launches == 2 * widths + len(ranges)
    assert _set(got.pairs) == want
    for x in colls:
        x.free()
