"""One-launch ordering of result pairs (k_sort_pairs) at the sizes where it can
go wrong: nothing and one pair, slices of 32 keys and their remainders, the
most a cluster holds, and results past it (the radix sort), on one join and
on a batch of joins sorted by one launch."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _cliques(n, extra, n_sets, seed):
    """n_sets sets of five tokens with exactly n(n-1)/2 + extra equal pairs: one
    group of n equal sets, `extra` pairs of equal sets, the rest on their own
    tokens, in a random order (all of one size, so any order is sorted)."""
    group = np.concatenate([np.zeros(n, int), 1 + np.repeat(np.arange(extra), 2)])
    group = np.concatenate([group, 1 + extra + np.arange(n_sets - group.size)])
    group = np.random.default_rng(seed).permutation(group)
    tokens = (1 + 5 * group[:, None] + np.arange(5)).astype(np.uint32)
    starts = (5 * np.arange(n_sets)).astype(np.uint32)
    return tokens.reshape(-1), starts, np.full(n_sets, 5, np.uint32)


def _expected(tokens, n):
    key = tokens.reshape(n, 5)[:, 0]
    order = np.argsort(key, kind="stable")
    pairs = []
    for ids in np.split(order, np.nonzero(np.diff(key[order]))[0] + 1):
        hi, lo = np.meshgrid(ids, ids, indexing="ij")
        pairs.append(np.stack([hi[hi > lo], lo[hi > lo]], 1))
    p = np.concatenate(pairs)
    return p[np.lexsort((p[:, 1], p[:, 0]))].astype(np.uint32)


# (clique, extra pairs): pairs = clique * (clique - 1) / 2 + extra
SIZES = [(0, 0), (0, 1), (0, 31), (0, 33), (9, 0), (23, 4), (46, 0), (91, 2), (129, 0), (362, 194), (362, 195),
         (363, 3000)]


@pytest.mark.parametrize("clique,extra", SIZES)
def test_sorted_pairs(ctx, clique, extra):
    n = clique + 2 * extra + 700
    tokens, starts, sizes = _cliques(clique, extra, n, seed=clique + extra)
    want = _expected(tokens, n)
    assert len(want) == clique * (clique - 1) // 2 + extra
    coll = ctx.upload(tokens, sizes, starts)
    for kw in (dict(technique="bitmap", bitmap=64), dict(technique="fgss", probe_major=True, pair_capacity=1000)):
        r = ctx.self_join(coll, threshold=0.9, sort_pairs=True, **kw)
        assert r.count == len(want)
        np.testing.assert_array_equal(r.pairs, want)
    plain = ctx.self_join(coll, threshold=0.9, technique="direct").pairs
    assert oracle.as_set(plain) == oracle.as_set(want)


def test_sorted_batch_of_every_size(ctx):
    joins, wants = [], []
    for clique, extra in SIZES:
        n = clique + 2 * extra + 700
        tokens, starts, sizes = _cliques(clique, extra, n, seed=7 + clique + extra)
        joins.append((ctx.upload(tokens, sizes, starts), None,
                      dict(threshold=0.9, technique="fgss", sort_pairs=True, pair_capacity=65600)))
        wants.append(_expected(tokens, n))
    for _ in range(2):
        for r, want in zip(ctx.batch_join(joins), wants):
            np.testing.assert_array_equal(r.pairs, want)
