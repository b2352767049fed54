"""Calls that find less device memory than they would like: an allocation is
made to fail (as in test_gpu_faults.py, before CUDA is asked), and the call
either goes on with less or reports HYSET_E_NOMEM and leaves its objects fit
for the next call."""
import contextlib
import dataclasses
import itertools
import os

import numpy as np
import pytest

import hyset_gb300 as hs
import oracle
from hyset_gb300 import synth
from hyset_gb300.handlers import BitmapHandler, FgssHandler

pytestmark = pytest.mark.gpu

E_NOMEM = 3
_spelling = itertools.cycle(range(1, 30))


@contextlib.contextmanager
def failing(n):
    """The n-th device allocation of the block fails (another spelling of n starts the count again)."""
    os.environ["HYSET_FAULT_ALLOC"] = "0" * next(_spelling) + str(n)
    try:
        yield
    finally:
        os.environ.pop("HYSET_FAULT_ALLOC")


@pytest.fixture
def keep(ctx):
    """Collections and handlers given back when the test ends, whatever still refers to them."""
    held = []
    yield lambda x: held.append(x) or x
    for x in reversed(held):
        x.close() if hasattr(x, "close") else x.free()


def outcomes(op, most):
    """op(n) with the n-th allocation failing, until twelve in a row come to no
    harm: for each n, whether the call went through."""
    went = []
    while len(went) < most and not (len(went) >= 12 and all(went[-12:])):
        with failing(len(went) + 1):
            try:
                op(len(went) + 1)
                went.append(True)
            except hs.HysetError as e:
                assert e.status == E_NOMEM, str(e)
                went.append(False)
    assert len(went) < most
    return went


def _sorted(p):
    p = np.asarray(p, np.int64).reshape(-1, 2)
    return p[np.lexsort((p[:, 1], p[:, 0]))]


@pytest.mark.parametrize("tech", ["bitmap", "fgss"])
@pytest.mark.parametrize("form", ["partition", "block"])
def test_handler_pairs_that_outgrow_their_buffer(ctx, keep, tech, form):
    """600 equal sets, 179,700 pairs, from a buffer of 65,536."""
    n = 600
    tokens = np.tile(np.arange(3, 23, dtype=np.uint32), n)
    sizes = np.full(n, 20, np.uint32)
    hc = hs.from_arrays(tokens, sizes, 100 if form == "partition" else n, 0.8)
    coll = keep(ctx.upload(tokens, sizes))
    want = np.array([(i, j) for i in range(n) for j in range(i)])

    def join(h):
        whole = hs.Partition(0, hc.blocks)
        h.join(*((whole, whole) if form == "partition" else (hc.blocks[0], hc.blocks[0])))

    def op(k):
        h = keep(BitmapHandler(ctx, hc, coll, 64, 100, False, 0.8) if tech == "bitmap"
                 else FgssHandler(ctx, hc, coll, 100, False, 0.8))
        out = hs.PairsHandler()
        h.set_output_handler(out)
        try:
            join(h)
        except hs.HysetError:
            h._lib.hyset_handler_clear_output(h.handle)
            join(h)  # the failure is behind it: the same handler, complete
            np.testing.assert_array_equal(_sorted(out.pairs), want)
            raise
        np.testing.assert_array_equal(_sorted(out.pairs), want)

    assert not all(outcomes(op, 60))


def test_block_index_that_was_not_finished(ctx, keep):
    """A failed build leaves no block's index behind, and no block id stands for "none"."""
    c = synth.generate(synth.C2, n_sets=4000, universe=2500, dup_frac=0.2, seed=9)
    hc = hs.from_arrays(c.tokens, c.sizes, 1000, 0.7)
    coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
    pairs = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.7))
    b = list(hc.blocks)

    def between(f, s):
        return {(p, q) for p, q in pairs if s.start_id <= p <= s.end_id and f.start_id <= q <= f.end_id}

    def op(k):
        h = keep(FgssHandler(ctx, hc, coll, 1000, False, 0.7))
        out = hs.PairsHandler()
        h.set_output_handler(out)
        h.join(b[0], b[2])
        try:
            h.join(b[3], b[3])  # longer sets: a larger index
        except hs.HysetError:
            h.join(b[0], b[1])
            assert oracle.as_set(out.pairs) == between(b[0], b[2]) | between(b[0], b[1])
            raise
        assert oracle.as_set(out.pairs) == between(b[0], b[2]) | between(b[3], b[3])

    assert not all(outcomes(op, 60))


def test_every_block_id_is_indexed(ctx, keep):
    c = synth.generate(synth.C2, n_sets=2000, universe=2500, dup_frac=0.2, seed=9)
    hc = hs.from_arrays(c.tokens, c.sizes, 2000, 0.7)
    coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
    last = dataclasses.replace(hc.blocks[0], id=0xFFFFFFFF)
    h = keep(FgssHandler(ctx, hc, coll, 2000, False, 0.7))
    out = hs.PairsHandler()
    h.set_output_handler(out)
    h.join(last, last)
    assert oracle.as_set(out.pairs) == oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.7))


def test_a_refused_allocation_is_reported_once(ctx, keep):
    """CUDA itself refuses a pair buffer of 256 TB; the next call starts clean."""
    c = synth.generate(synth.C2, n_sets=2000, universe=2500, dup_frac=0.2, seed=9)
    coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
    want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.7))
    for kw in (dict(technique="bitmap"), dict(technique="fgss", probe_major=True)):
        with pytest.raises(hs.HysetError) as e:
            ctx.self_join(coll, threshold=0.7, pair_capacity=1 << 45, **kw)
        assert e.value.status == E_NOMEM
        assert oracle.as_set(ctx.self_join(coll, threshold=0.7, **kw).pairs) == want
