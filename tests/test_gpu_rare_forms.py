"""Forms of a call that ordinary inputs do not take: a batch on one branch of
its graph, a handler's index range of a collection whose lists are known to be
long, a signature join without room for its wider signatures."""
import numpy as np
import pytest

import hyset_gb300 as hs
import oracle
from hyset_gb300 import synth
from hyset_gb300.handlers import FgssHandler
from test_gpu_index_lists import _plant
from test_gpu_short_memory import failing, keep  # noqa: F401  (keep: a fixture)

pytestmark = pytest.mark.gpu


def test_batch_on_one_branch(ctx, keep):  # noqa: F811
    """A universe so large that the scratch of one index build passes a gigabyte, half of what all branches may take."""
    joins, want = [], []
    for seed, tau in ((1, 0.6), (2, 0.7), (3, 0.8)):
        c = synth.generate(synth.C2, n_sets=3000, universe=2000, dup_frac=0.1, seed=seed)
        far = np.where(c.tokens == c.tokens.max(), np.uint32(300_000_000), c.tokens)  # keeps the order of all tokens
        coll = keep(ctx.upload(far, c.sizes, c.starts))
        joins.append((coll, None, dict(threshold=tau, technique="bitmap" if seed == 2 else "auto", sort_pairs=True)))
        want.append(oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, tau)))
    for _ in range(2):  # the second call replays the graph
        got = ctx.batch_join(joins)
        assert [oracle.as_set(r.pairs) for r in got] == want
        for r in got:
            p = r.pairs.astype(np.int64)
            assert (np.diff(p[:, 0] * 3000 + p[:, 1]) > 0).all()


@pytest.mark.parametrize("longest", [31, 40, 64, 65, 90])
def test_ranges_of_a_collection_whose_lists_are_known(ctx, keep, longest):  # noqa: F811
    c = _plant(synth.generate(synth.C2, n_sets=20_000, seed=64), longest, seed=longest)
    pairs = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.8))
    coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
    assert oracle.as_set(ctx.self_join(coll, threshold=0.8, technique="fgss", probe_major=True).pairs) == pairs
    blocks = list(hs.from_arrays(c.tokens, c.sizes, 2_000, 0.8).blocks)
    h = keep(FgssHandler(ctx, None, coll, 2_000, False, 0.8))
    for a, b in ((blocks, blocks), (blocks[1:4], blocks[2:]), (blocks[3:], blocks[5:7]), (blocks[:1], blocks)):
        out = hs.PairsHandler()
        h.set_output_handler(out)
        h.join(hs.Partition(0, a), hs.Partition(0, b))
        assert oracle.as_set(out.pairs) == {(p, q) for p, q in pairs if b[0].start_id <= p <= b[-1].end_id
                                            and a[0].start_id <= q <= a[-1].end_id}


def test_signature_join_without_room_for_wider_signatures(ctx, keep):  # noqa: F811
    """In three widths with room (test_gpu_window_three_widths.py), in fewer without."""
    c = synth.generate(synth.C3, n_sets=24_001, universe=24_000, seed=5)
    want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.5))
    kw = dict(threshold=0.5, technique="bitmap", bitmap=64)
    ctx.self_join(keep(ctx.upload(c.tokens, c.sizes, c.starts)), **kw)
    launches = []
    for n in range(1, 6):
        coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
        with failing(n):
            try:
                got = ctx.self_join(coll, **kw)
            except hs.HysetError as e:
                assert n == 1 and e.status == 3  # the signatures that were asked for
                continue
        assert oracle.as_set(got.pairs) == want
        launches.append(got.launches)
    assert launches == [2, 4, 6, 6]
