"""Collections whose sizes are on the device: those of up to 16,384 sets come
back as they are, those of more as runs, with more than 8,192 runs as they are
after all.  Both sides of either bound."""
import numpy as np
import pytest
import torch

import oracle
from hyset_gb300 import similarity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distinct,alone", [
    (1, 0), (1, 16_400), (8191, 8_190), (8191, 8_191), (8191, 9_000), (8192, 9_000), (8193, 9_000), (8200, 0), (8200, 9_000),
])
def test_sizes_read_back_from_the_device(ctx, distinct, alone):
    """Nested sets {0 .. l-1}, one of every size, the last three sizes twice, and
    sets of one token each that no other has."""
    sizes = np.sort(np.concatenate([np.arange(1, distinct + 1), np.arange(max(1, distinct - 2), distinct + 1)]))
    starts = np.concatenate([[0], np.cumsum(sizes)])[:-1]
    tokens = np.arange(sizes.sum()) - np.repeat(starts, sizes)
    tau = 0.9995
    want = set()
    for i, l in enumerate(sizes):
        for j in range(i - 1, -1, -1):
            if sizes[j] < similarity.minsize("jaccard", int(l), tau):
                break
            if similarity.minoverlap("jaccard", int(l), int(sizes[j]), tau) <= sizes[j]:
                want.add((alone + i, alone + j))
    assert len(want) >= 3 * distinct // 4 or distinct == 1
    sizes = np.concatenate([np.ones(alone, np.int64), sizes])
    tokens = np.concatenate([10_000 + np.arange(alone), tokens])
    starts = np.concatenate([[0], np.cumsum(sizes)])[:-1]
    d = [torch.from_numpy(a.astype(np.uint32).view(np.int32)).cuda() for a in (tokens, starts, sizes)]
    coll = ctx.from_device(d[0].data_ptr(), tokens.size, d[1].data_ptr(), d[2].data_ptr(), sizes.size, keep=d)
    for kw in (dict(technique="fgss", probe_major=True, bitmap=128), dict(technique="bitmap"), dict(technique="direct")):
        got = ctx.self_join(coll, threshold=tau, **kw)
        assert got.count == len(want) and oracle.as_set(got.pairs) == want
    coll.free()
