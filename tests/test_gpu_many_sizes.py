"""Collections whose sizes are on the device: up to 8,192 distinct sizes come
back as runs, more as they are.  Both sides of the bound."""
import numpy as np
import pytest
import torch

import oracle
from hyset_gb300 import similarity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distinct", [1, 8191, 8192, 8193, 8200])
def test_sizes_read_back_from_the_device(ctx, distinct):
    """Nested sets {0 .. l-1}, one of every size, the last three sizes twice."""
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
                want.add((i, j))
    assert len(want) >= 3 * distinct // 4 or distinct == 1
    d = [torch.from_numpy(a.astype(np.uint32).view(np.int32)).cuda() for a in (tokens, starts, sizes)]
    coll = ctx.from_device(d[0].data_ptr(), tokens.size, d[1].data_ptr(), d[2].data_ptr(), sizes.size, keep=d)
    for kw in (dict(technique="fgss", probe_major=True, bitmap=128), dict(technique="bitmap"), dict(technique="direct")):
        got = ctx.self_join(coll, threshold=tau, **kw)
        assert got.count == len(want) and oracle.as_set(got.pairs) == want
    coll.free()
