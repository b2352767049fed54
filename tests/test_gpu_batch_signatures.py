"""Signature joins of a batch on both sides of the size from which on they are
launches of their own, at every width, beside joins of the other techniques."""
import pytest

import hyset_gb300 as hs
import oracle
from hyset_gb300 import synth
from test_gpu_short_memory import failing

pytestmark = pytest.mark.gpu


def _set(pairs):
    s = oracle.as_set(pairs)
    assert len(s) == len(pairs), "duplicate pairs"
    return s


@pytest.mark.parametrize("sim,tau", [("jaccard", 0.6), ("cosine", 0.75)])
def test_small_and_large_signature_joins(ctx, sim, tau):
    sizes = (1, 33, 700, 2895, 2897, 5001)  # 2,896 sets and more: 8M pairs
    colls, want = [], []
    for k, n in enumerate(sizes):
        c = synth.generate(synth.C2, n_sets=n, universe=2_500, dup_frac=0.2 if n > 1 else 0.0, seed=40 + k)
        colls.append(ctx.upload(c.tokens, c.sizes, c.starts))
        want.append(oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, tau, sim=sim)))
    kw = dict(threshold=tau, sim=sim)
    for bits in (64, 128, 256, 512, 1024):
        joins = [(x, None, dict(kw, technique="bitmap", bitmap=bits, sort_pairs=bits == 64)) for x in colls]
        for _ in range(2):  # the second call replays the graph
            assert [_set(r.pairs) for r in ctx.batch_join(joins)] == want
    mixed = [(x, None, dict(kw, **t)) for x in colls[1:] for t in
             (dict(technique="bitmap", bitmap=128), dict(technique="direct"), dict(technique="fgss", bitmap=256),
              dict(technique="bitmap"))]
    assert [_set(r.pairs) for r in ctx.batch_join(mixed)] == [w for w in want[1:] for _ in range(4)]
    lo, hi = 1_500, 4_900  # a range of 17M pairs, and one of 5M
    ranges = [(colls[-1], None, dict(kw, technique="bitmap", bitmap=64, probe_range=r)) for r in ((lo, hi), (lo, lo + 1000))]
    for (a, b), r in zip(((lo, hi), (lo, lo + 1000)), ctx.batch_join(ranges)):
        assert _set(r.pairs) == {p for p in want[-1] if a <= p[0] < b}
    for x in colls:
        x.free()


@pytest.mark.parametrize("n_r,n_s", [(300, 900), (2_600, 3_300)])
def test_rs_signature_joins(ctx, n_r, n_s):
    c = synth.generate(synth.C2, n_sets=n_r, universe=1_500, dup_frac=0.1, seed=7)
    s = synth.generate(synth.C2, n_sets=n_s, universe=1_500, dup_frac=0.1, seed=7)  # shares c's generator: pairs across
    want = oracle.as_set(oracle.brute_rs((c.tokens, c.starts, c.sizes), (s.tokens, s.starts, s.sizes), 0.6))
    R, S = ctx.upload(c.tokens, c.sizes, c.starts), ctx.upload(s.tokens, s.sizes, s.starts)
    joins = [(R, S, dict(threshold=0.6, technique="bitmap", bitmap=b, orientation=o)) for b in (64, 256)
             for o in ("as_given", "swapped")]
    for _ in range(2):
        for r in ctx.batch_join(joins):
            assert _set(r.pairs) == want
    R.free()
    S.free()


@pytest.mark.parametrize("bits", [64, 128, 256])
def test_joins_in_three_widths(ctx, bits):
    """Long sets whose probes fill their signatures, as in test_gpu_window_three_widths.py, beside small ones."""
    tau = 0.5
    big = synth.generate(synth.C3, n_sets=24_001, universe=24_000, seed=5)
    small = synth.generate(synth.C3, n_sets=1_500, universe=3_000, seed=6)
    B, A = ctx.upload(big.tokens, big.sizes, big.starts), ctx.upload(small.tokens, small.sizes, small.starts)
    want = oracle.as_set(oracle.join(big.tokens, big.starts, big.sizes, tau))
    want_a = oracle.as_set(oracle.join(small.tokens, small.starts, small.sizes, tau))
    want_rs = oracle.as_set(oracle.brute_rs((small.tokens, small.starts, small.sizes),
                                            (big.tokens, big.starts, big.sizes), tau))
    kw = dict(threshold=tau, technique="bitmap", bitmap=bits)
    joins = [(B, None, kw), (A, None, kw), (A, B, kw), (B, None, dict(kw, probe_range=(20_000, 24_001)))]
    for _ in range(2):
        got = [_set(r.pairs) for r in ctx.batch_join(joins)]
        assert got == [want, want_a, want_rs, {p for p in want if p[0] >= 20_000}]
    wider = {64: (3, 4), 128: (3, 4), 256: (3,)}[bits]  # the allocations after the join's own signatures and its pairs
    for k in range(1, 30):
        ctx.batch_join([(A, None, dict(threshold=0.9))])  # another batch: the plan is made again
        with failing(k):
            try:
                got = ctx.batch_join([(B, None, kw)])
            except hs.HysetError as e:
                assert e.status == 3 and k not in wider
                continue
        assert _set(got[0].pairs) == want
    B.free()
    A.free()
