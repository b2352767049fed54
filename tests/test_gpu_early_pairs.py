"""The pairs that come back with their number: a sixteenth of the sets probed,
at least 2,048.  Results on both sides of that bound, where the sets probed are
a part of a larger collection: probe ranges and pairs of blocks."""
import numpy as np
import pytest

import hyset_gb300 as hs
from hyset_gb300.handlers import BitmapHandler, FgssHandler

pytestmark = pytest.mark.gpu

N, TAIL, SIZE = 60_000, 500, 12  # a sixteenth of all sets: 3,750


def _groups(groups):
    """N sets of one size, apart except for groups of equal ones among the last TAIL."""
    rows = (np.arange(N, dtype=np.uint32)[:, None] * SIZE + np.arange(SIZE, dtype=np.uint32))
    at, pairs = N - TAIL, []
    for g in groups:
        rows[at:at + g] = rows[at]
        pairs += [(at + i, at + j) for i in range(g) for j in range(i)]
        at += g
    assert at <= N
    return rows, pairs


@pytest.mark.parametrize("groups,count", [
    ((), 0), ((2,), 1), ((64, 8, 3), 2047), ((64, 8, 3, 2), 2048), ((64, 8, 3, 2, 2), 2049), ((87, 5), 3751),
])
@pytest.mark.parametrize("technique", ["bitmap", "fgss"])
def test_results_around_the_early_copy(ctx, groups, count, technique):
    rows, want = _groups(groups)
    assert len(want) == count
    sizes = np.full(N, SIZE, np.uint32)
    coll = ctx.upload(rows.reshape(-1), sizes)
    kw = dict(threshold=0.9, technique=technique, bitmap=64, probe_major=technique == "fgss")
    for opts in (dict(probe_range=(N - TAIL, N)), {}, dict(probe_range=(N - TAIL, N), sort_pairs=True)):
        got = ctx.self_join(coll, **kw, **opts)
        assert got.count == count
        np.testing.assert_array_equal(np.array(sorted(map(tuple, got.pairs.tolist()))).reshape(-1, 2),
                                      np.array(want).reshape(-1, 2))
    hc = hs.from_arrays(rows.reshape(-1), sizes, TAIL, 0.9)
    h = BitmapHandler(ctx, hc, coll, 64, TAIL, False, 0.9) if technique == "bitmap" else FgssHandler(ctx, hc, coll, TAIL, False, 0.9)
    out = hs.PairsHandler()
    h.set_output_handler(out)
    h.join(hc.blocks[-1], hc.blocks[-1])
    got = np.asarray(out.pairs, np.int64).reshape(-1, 2)
    np.testing.assert_array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], np.array(want, np.int64).reshape(-1, 2))
    h.close()
    coll.free()
