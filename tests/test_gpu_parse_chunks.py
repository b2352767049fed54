"""Host text on both sides of the size from which on it is parsed in chunks as
it lands, from pageable and pinned memory, every line's tokens compared."""
import numpy as np
import pytest
import torch

from hyset_gb300 import synth

pytestmark = pytest.mark.gpu

ROW, LIMIT = 60, 48 << 20


@pytest.fixture(scope="module")
def rows():
    rng = np.random.default_rng(8)
    n = 190_000  # about 58 MB: tokens of one to seven digits, lines of uneven length
    low = np.sort(np.argsort(rng.random((n, 40)), axis=1)[:, :6], axis=1)
    high = 40 + np.cumsum(rng.integers(1, 120_000, (n, ROW - 6)) >> rng.integers(0, 16, (n, 1)), axis=1)
    r = np.concatenate([low, high + np.arange(ROW - 6)], axis=1).astype(np.uint32)
    text = synth.format_text(r.reshape(-1), np.arange(n, dtype=np.uint32) * ROW, np.full(n, ROW, np.uint32))
    return r, np.frombuffer(text.tobytes(), np.uint8)


@pytest.mark.parametrize("over", [-4096, -1, 0, 1, 4096, 1 << 20, 5 << 20])
@pytest.mark.parametrize("pinned", [False, True])
def test_text_around_one_chunk(ctx, rows, over, pinned):
    r, text = rows
    ends = np.nonzero(text == 10)[0] + 1
    assert ends[-1] > LIMIT + (5 << 20)
    k = int(np.searchsorted(ends, LIMIT + over, side="right"))  # whole lines; the text's last one may lack its newline
    part = text[: ends[k - 1] - (1 if over % 2 else 0)]
    if pinned:
        t = torch.empty(part.size, dtype=torch.uint8, pin_memory=True)
        t.numpy()[:] = part
        part = t.numpy()
    coll = ctx.parse(part)
    tokens, starts, sizes = coll.download()
    np.testing.assert_array_equal(sizes, np.full(k, ROW, np.uint32))
    np.testing.assert_array_equal(tokens, r[:k].reshape(-1))
    np.testing.assert_array_equal(starts, np.arange(k, dtype=np.uint32) * ROW)
    coll.free()
