"""Signature joins on both sides of the number of pairs from which on the tiled
kernel takes them, by probe ranges of one collection (the bound depends on
the width and on how many probes are heavy): one probe more and one less."""
import numpy as np
import pytest

import oracle
from hyset_gb300 import synth

pytestmark = pytest.mark.gpu


def _set(p):
    s = oracle.as_set(p)
    assert len(s) == len(p), "duplicate pairs"
    return s


@pytest.mark.parametrize("bits", [64, 128, 256, 512])
@pytest.mark.parametrize("sim,tau", [("jaccard", 0.6), ("cosine", 0.8)])
def test_self_join_ranges(ctx, bits, sim, tau):
    c = synth.generate(synth.C2, n_sets=16_384, universe=9_000, dup_frac=0.2, seed=bits)
    coll = ctx.upload(c.tokens, c.sizes, c.starts)
    want = np.array(sorted(oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, tau, sim=sim))))
    bounds = [b // c.n for b in ((3 << 18,) if bits == 512 else (1 << 18, 5 << 19))]  # 48, 16 (heavy probes) and 160
    some = sorted({1, 2 * bounds[-1] + 5, 4 * bounds[-1] - 1} | {b + k for b in bounds for k in (-1, 0, 1)})
    for lo in (0, 5_001, 12_000):
        for np_ in some:
            for mode in (1, 2):
                got = ctx.self_join(coll, threshold=tau, sim=sim, technique="bitmap", bitmap=bits, verify_mode=mode,
                                    probe_range=(lo, lo + np_))
                rows = want[(want[:, 0] >= lo) & (want[:, 0] < lo + np_)]
                assert _set(got.pairs) == set(map(tuple, rows.tolist()))
    hi = c.n  # the longest sets
    for np_ in some:
        got = ctx.self_join(coll, threshold=tau, sim=sim, technique="bitmap", bitmap=bits, probe_range=(hi - np_, hi))
        assert _set(got.pairs) == set(map(tuple, want[want[:, 0] >= hi - np_].tolist()))
    coll.free()


@pytest.mark.parametrize("bits", [64, 512])
def test_rs_join_ranges(ctx, bits):
    c = synth.generate(synth.C2, n_sets=11_192, universe=5_000, dup_frac=0.3, seed=3)
    side = np.zeros(c.n, bool)
    side[np.random.default_rng(1).choice(c.n, 8_192, replace=False)] = True
    at = np.where(side, np.cumsum(side) - 1, np.cumsum(~side) - 1)  # in the halves' own numbers
    want = np.array(sorted((int(at[b]), int(at[a])) if side[a] else (int(at[a]), int(at[b]))
                           for a, b in oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.6)) if side[a] != side[b]))
    colls = []
    for ids in (np.nonzero(side)[0], np.nonzero(~side)[0]):
        colls.append(ctx.upload(np.concatenate([c.set(i) for i in ids]), c.sizes[ids]))
    R, S = colls
    bounds = [b // 8_192 for b in ((3 << 18,) if bits == 512 else (5 << 17, 3 << 20))]  # 96, 80 (heavy probes) and 384
    assert len(want) > 500
    for lo in (0, 1_001, 2_000):
        for np_ in sorted({1, 2 * bounds[-1] + 3} | {b + k for b in bounds for k in (-1, 0, 1)}):
            got = ctx.rs_join(R, S, threshold=0.6, technique="bitmap", bitmap=bits, probe_range=(lo, lo + np_),
                              orientation="as_given")
            rows = want[(want[:, 0] >= lo) & (want[:, 0] < lo + np_)]
            assert _set(got.pairs) == set(map(tuple, rows.tolist()))
    R.free()
    S.free()
