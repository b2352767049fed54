"""One set of millions of tokens among many of a few hundred: the split probes'
units (probes x segments of the longest prefix) would pass 32 bits."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZE, STEP, N, GIANT = 260, 15_000, 131_200, 4_200_000
HEAVY = N + 1  # at Jaccard 0.5 a set of 260 has a prefix of 131 slots, more than 128
assert HEAVY * -(-(GIANT // 2 + 1) // 64) >= 1 << 32


def _edited(rows, rng):
    """240 of a set's 260 tokens kept: Jaccard 0.857; sets drawn apart share a token in 58 sets, never 174."""
    rows = rows.copy()
    rows[:, ::13] = np.arange(0, SIZE, 13) * STEP + rng.integers(0, STEP, (len(rows), SIZE // 13))
    return rows


@pytest.fixture(scope="module")
def sets():
    rng = np.random.default_rng(3)
    rows = (np.arange(SIZE) * STEP + rng.integers(0, STEP, (N, SIZE))).astype(np.uint32)
    rows[100_000:101_000] = _edited(rows[:1000], rng)
    other = _edited(rows[5_000:6_500], rng)
    own = {(100_000 + i, i) for i in range(1000)}
    cross = {(5_000 + i, i) for i in range(1500)}
    return rows, other, own, cross


def _upload(ctx, rows, giant):
    sizes = np.full(len(rows), SIZE, np.uint32)
    if not giant:
        return ctx.upload(rows.reshape(-1), sizes)
    return ctx.upload(np.concatenate([rows.reshape(-1), np.arange(GIANT, dtype=np.uint32)]),
                      np.append(sizes, np.uint32(GIANT)))


def test_no_probe_is_left_out(ctx, sets):
    rows, other, own, cross = sets
    S, R = _upload(ctx, rows, True), _upload(ctx, other, False)
    try:
        kw = dict(threshold=0.5, technique="fgss", probe_major=True, bitmap=256)
        assert oracle.as_set(ctx.self_join(S, **kw).pairs) == own
        assert oracle.as_set(ctx.rs_join(R, S, **kw).pairs) == cross
        both = ctx.batch_join([(S, None, kw), (R, S, kw)])
        assert [oracle.as_set(r.pairs) for r in both] == [own, cross]
    finally:
        S.free()
        R.free()
