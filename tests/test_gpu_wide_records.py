"""Token records of 64 words (lists of 32 to 63 entries) on both sides of
their bounds: the collection's first build, which converts its lists, later
builds, which emit records, R-S joins whose two indexes have records of
different widths, and the host-input join, whose list can outgrow the records
it was given."""
import numpy as np
import pytest

import oracle
from hyset_gb300 import synth
from test_gpu_index_lists import _longest_list, _plant

pytestmark = pytest.mark.gpu
PIPELINED = dict(technique="fgss", probe_major=True, bitmap=256)


@pytest.mark.parametrize("k", [32, 39, 40, 62, 63, 64])
def test_lists_around_the_wide_record(ctx, k):
    c = _plant(synth.generate(synth.C2, n_sets=20000, seed=64), k, seed=k)
    assert _longest_list(c, 0.8) == k
    exp = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.8))
    coll = ctx.upload(c.tokens, c.sizes, c.starts)
    for kw in (dict(bitmap=0), dict(bitmap=256), dict(bitmap=512, verify_mode=2), dict(bitmap=0, fgss_batch=1)):
        r = ctx.self_join(coll, threshold=0.8, technique="fgss", probe_major=True, **kw)
        assert r.count == len(exp) and oracle.as_set(r.pairs) == exp, kw


@pytest.mark.parametrize("sim", ["jaccard", "cosine", "dice"])
def test_wide_records_every_similarity(ctx, sim):
    c = synth.generate(synth.C3, n_sets=30000, universe=30000, seed=5)
    exp = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.8, sim=sim))
    coll = ctx.upload(c.tokens, c.sizes, c.starts)
    for _ in range(3):
        r = ctx.self_join(coll, threshold=0.8, sim=sim, **PIPELINED)
        assert r.count == len(exp) and oracle.as_set(r.pairs) == exp


@pytest.mark.parametrize("sim", ["jaccard", "cosine"])
def test_rs_join_with_records_of_two_widths(ctx, sim):
    c = synth.generate(synth.C3, n_sets=9000, universe=9000, seed=6)
    side = np.random.default_rng(3).random(c.n) < 0.4
    parts = []
    for mask in (side, ~side):
        ids = np.nonzero(mask)[0]
        sizes = c.sizes[ids]
        starts = np.concatenate([[0], np.cumsum(sizes.astype(np.int64))])[:-1].astype(np.uint32)
        parts.append((np.concatenate([c.set(i) for i in ids]), starts, sizes))
    exp = oracle.as_set(oracle.brute_rs(parts[0], parts[1], 0.7, sim=sim))
    R, S = (ctx.upload(t, z, s) for t, s, z in parts)
    for _ in range(3):
        r = ctx.rs_join(R, S, threshold=0.7, sim=sim, **PIPELINED)
        assert r.count == len(exp) and oracle.as_set(r.pairs) == exp


@pytest.mark.parametrize("before,after", [(30, 33), (45, 63), (45, 64), (63, 63), (40, 90)])
def test_host_join_whose_lists_grow(ctx, before, after):
    base = synth.generate(synth.C2, n_sets=20000, seed=64)
    for k in (before, before, before, after, after, before):  # the same sizes every time
        c = _plant(base, k, seed=k)
        exp = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.8))
        r = ctx.self_join_host(c.tokens, c.sizes, c.starts, threshold=0.8, sort_pairs=True, **PIPELINED)
        assert r.count == len(exp) and oracle.as_set(r.pairs) == exp, k


@pytest.mark.parametrize("sim", ["jaccard", "cosine", "dice"])
def test_split_probes_of_banded_joins(ctx, sim):
    """Probes of more than 128 prefix slots go in units of 64 slots of both bands."""
    c = synth.generate(synth.C3, n_sets=1500, universe=12000, size_min=200, size_a=6.3, seed=8)
    assert c.sizes.max() > 1500
    side = np.random.default_rng(4).random(c.n) < 0.5
    parts = []
    for mask in (side, ~side):
        ids = np.nonzero(mask)[0]
        sizes = c.sizes[ids]
        starts = np.concatenate([[0], np.cumsum(sizes.astype(np.int64))])[:-1].astype(np.uint32)
        parts.append((np.concatenate([c.set(i) for i in ids]), starts, sizes))
    R, S = (ctx.upload(t, z, s) for t, s, z in parts)
    for tau in (0.6, 0.85):
        exp = oracle.as_set(oracle.brute_rs(parts[0], parts[1], tau, sim=sim))
        for kw in (dict(bitmap=0), dict(bitmap=512, fgss_batch=16), dict(bitmap=128, verify_mode=2)):
            for orientation in ("as_given", "swapped"):
                r = ctx.rs_join(R, S, threshold=tau, sim=sim, technique="fgss", probe_major=True,
                                orientation=orientation, **kw)
                assert r.count == len(exp) and oracle.as_set(r.pairs) == exp
