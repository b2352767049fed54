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
from test_gpu_index_lists import _plant

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


def outcomes(op, most, ready=lambda: None):
    """op(ready()) with the n-th allocation of op failing, n from 1 until twelve
    in a row come to no harm: for each n, whether the call went through."""
    went = []
    while len(went) < most and not (len(went) >= 12 and all(went[-12:])):
        x = ready()
        with failing(len(went) + 1):
            try:
                op(x)
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

    def op(_):
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

    def op(_):
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


def _uniform(n, spread, size=30, seed=1):
    """n sets whose prefix tokens (four of 30 at Jaccard 0.8) spread evenly over
    `spread` tokens; near-copies among them."""
    rng = np.random.default_rng(seed)
    low = np.arange(4) * (spread // 4) + rng.integers(0, spread // 4, (n, 4))
    high = spread + np.arange(size - 4) * 64 + rng.integers(0, 64, (n, size - 4))
    rows = np.concatenate([low, high], axis=1).astype(np.uint32)
    rows[n // 2:n // 2 + n // 8] = rows[:n // 8]
    rows[n // 2:n // 2 + n // 8, 9] = spread + 5 * 64 + rng.integers(0, 64, n // 8)
    return rows.reshape(-1), np.full(n, size, np.uint32)


PREFIX = dict(threshold=0.8, technique="fgss", probe_major=True, bitmap=128, sort_pairs=True)  # midprefix of 30: 4


# (sets, universe, the record width in words after the first and after later builds; 0: lists)
@pytest.mark.parametrize("n,spread,first,later", [
    (2_000, 1 << 20, 32, 32),    # few sets over many tokens
    (40_000, 1 << 15, 64, 32),   # five entries to a token, none with 32
    (60_000, 1 << 14, 64, 64),   # fifteen, and some with more than 31
    (100_000, 1 << 14, 64, 64),  # twenty-four: lists first, then their records
    (200_000, 1 << 14, 0, 0),    # fifty: lists
])
def test_records_no_wider_than_the_lists_need(ctx, keep, n, spread, first, later):
    tokens, sizes = _uniform(n, spread)
    entries = np.concatenate([tokens[k::30] for k in range(4)])
    longest = np.bincount(entries).max()
    assert (later == 32) == (longest <= 31) and (later == 0) == (longest > 63)
    universe = int(tokens.max()) + 1
    coll = keep(ctx.upload(tokens, sizes))
    keep(ctx.upload(tokens, sizes))
    bytes_now = hs._lib.load().hyset_device_bytes
    other = keep(ctx.upload(tokens, sizes))
    ctx.self_join(other, **PREFIX)  # the context's own buffers
    before = bytes_now()
    got = ctx.self_join(coll, **PREFIX)
    lists = (universe + 1) * 4 + entries.size * 8  # list offsets, entries and their positions
    signatures = n * (16 + 32) + 8 + 32
    assert bytes_now() - before <= lists + signatures + universe * first * 4 + 64
    again = ctx.self_join(coll, **PREFIX)
    assert bytes_now() - before <= lists + signatures + universe * later * 4 + 64
    want = oracle.as_set(oracle.join(tokens, np.arange(n, dtype=np.uint32) * 30, sizes, 0.8))
    assert oracle.as_set(got.pairs) == want and oracle.as_set(again.pairs) == want and len(want) >= n // 8


def test_lists_that_outgrow_the_guessed_records(ctx, keep):
    c = _plant(synth.generate(synth.C2, n_sets=20000, seed=64), 90, seed=2)
    bytes_now = hs._lib.load().hyset_device_bytes
    ctx.self_join(keep(ctx.upload(c.tokens, c.sizes, c.starts)), **PREFIX)
    coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
    before = bytes_now()
    got = ctx.self_join(coll, **PREFIX)
    assert bytes_now() - before < (int(c.tokens.max()) + 1) * 128  # no record buffer is kept
    assert oracle.as_set(got.pairs) == oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.8))


@pytest.mark.parametrize("builds", [0, 1, 2])
def test_join_without_room_for_records(ctx, keep, builds):
    """A first build, and one after `builds` others; R-S joins have two indexes."""
    c = synth.generate(synth.C2, n_sets=12000, universe=9000, dup_frac=0.1, seed=31)
    s = synth.generate(synth.C2, n_sets=13000, universe=9000, dup_frac=0.1, seed=32)
    want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.8))
    want_rs = oracle.as_set(oracle.brute_rs((c.tokens, c.starts, c.sizes), (s.tokens, s.starts, s.sizes), 0.8))
    S = keep(ctx.upload(s.tokens, s.sizes, s.starts))
    ctx.rs_join(keep(ctx.upload(c.tokens, c.sizes, c.starts)), S, **PREFIX)
    for join, exp in ((lambda x: ctx.self_join(x, **PREFIX), want), (lambda x: ctx.rs_join(x, S, **PREFIX), want_rs)):
        def ready():
            coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
            for _ in range(builds):
                join(coll)
            return coll

        def op(coll):
            assert oracle.as_set(join(coll).pairs) == exp

        went = outcomes(op, 60, ready)
        if builds == 0:  # list offsets, entries, positions, signatures: records come after them
            assert not went[0] and sum(not w for w in went) <= (4 if exp is want else 7)


def test_host_join_without_room_for_records(ctx):
    c = synth.generate(synth.C2, n_sets=12000, universe=9000, dup_frac=0.1, seed=31)
    want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.8))

    def join():
        return ctx.self_join_host(c.tokens, c.sizes, c.starts, **PREFIX)

    for _ in range(3):
        join()

    def op(_):
        assert oracle.as_set(join().pairs) == want

    went = outcomes(op, 60)
    assert False in went and True in went[:len(went) - 1 - went[::-1].index(False)]  # records are not the last buffer


@pytest.mark.parametrize("tech,aggregate", [("fgss", False), ("fgss", True), ("bitmap", False)])
def test_partitions_without_room_for_their_index(ctx, keep, tech, aggregate):
    """Any one allocation may fail: the blocks are then joined pair by pair."""
    c = synth.generate(synth.C2, n_sets=20_000, universe=15_000, dup_frac=0.1, seed=33)
    want = oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, 0.8))
    hc = hs.from_arrays(c.tokens, c.sizes, 5_000, 0.8)
    coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
    whole = hs.Partition(0, hc.blocks)
    for n in range(1, 40):
        own = keep(hs.Context(0)) if n < 25 else ctx  # with and without a context's scratch from earlier calls
        mine = keep(own.upload(c.tokens, c.sizes, c.starts)) if own is not ctx else coll
        h = keep(BitmapHandler(own, hc, mine, 64, 5_000, aggregate, 0.8) if tech == "bitmap"
                 else FgssHandler(own, hc, mine, 5_000, aggregate, 0.8))
        out = hs.CountHandler() if aggregate else hs.PairsHandler()
        h.set_output_handler(out)
        with failing(n if own is not ctx else n - 24):
            h.join(whole, whole)
        assert out.get_count() == len(want)
        assert aggregate or oracle.as_set(out.pairs) == want


def test_batch_with_room_for_fewer_branches(ctx, keep):
    """Five joins: five scratches, the first of which is needed."""
    c = synth.generate(synth.C2, n_sets=3000, universe=2000, dup_frac=0.05, seed=77)
    coll = keep(ctx.upload(c.tokens, c.sizes, c.starts))
    taus = (0.6, 0.65, 0.7, 0.8, 0.9)
    joins = [(coll, None, dict(threshold=t, technique="fgss", probe_major=True, bitmap=64)) for t in taus]
    want = [oracle.as_set(oracle.join(c.tokens, c.starts, c.sizes, t)) for t in taus]
    bytes_now = hs._lib.load().hyset_device_bytes
    ctx.batch_join(joins)  # the bound tables, and the plan's whole size
    held = bytes_now()
    plain = keep(ctx.upload(c.tokens, c.sizes, c.starts))
    less, failed = 0, 0
    for n in range(1, 90):
        ctx.batch_join([(plain, None, dict(threshold=0.95))])  # another batch: the plan is made again
        with failing(n):
            try:
                got = ctx.batch_join(joins)
            except hs.HysetError as e:
                assert e.status == E_NOMEM
                failed += 1
                continue
        assert [oracle.as_set(r.pairs) for r in got] == want
        less = max(less, held - bytes_now())
    # each join's lists, positions, entries, signatures and pairs, eleven arrays of the
    # first scratch, and the plan's counts, counters, descriptors and units
    assert failed == 5 * 5 + 11 + 4
    assert less > 4 * 6 * 3000 * 4 // 2  # four scratches fewer, six arrays of the longest index's entries each
