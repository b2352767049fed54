"""Partition joins of the reference-shaped handlers run as one join of two id
ranges where that is the same result: every form of block list (whole, parts
that overlap, lie apart or are in the wrong order, gaps, repeats, ids against
their order) against the same block pairs joined one by one."""
import dataclasses

import numpy as np
import pytest

import hyset_gb300 as hs
from hyset_gb300 import similarity, synth
from hyset_gb300.handlers import BitmapHandler, FgssHandler

pytestmark = pytest.mark.gpu

N, BLOCK, TAU = 4900, 500, 0.6


def _forms(b):
    again = [dataclasses.replace(x, id=len(b) - x.id) for x in b]  # ids against the order of the ranges
    return {
        "whole": (b, b), "one": (b[3:4], b[3:4]), "later": (b[:4], b[4:]), "earlier": (b[5:], b[:5]),
        "overlap": (b[2:6], b[4:9]), "overlap_back": (b[4:9], b[2:6]), "gap": (b[:2] + b[4:6], b),
        "gap_probe": (b, b[1:3] + b[6:]), "reversed": (b[::-1], b), "repeat": (b[:3] + b[2:4], b[:5]),
        "twice": (b[:2], b[:2] + b[:2]), "ids_back": (again, b), "ids_back_both": (again, again), "none": ([], b),
        "last_odd": (b[-2:], b[-1:]),
    }


def _sorted(p):
    p = np.asarray(p, np.int64).reshape(-1, 2)
    return p[np.lexsort((p[:, 1], p[:, 0]))]


@pytest.mark.parametrize("tech", ["bitmap", "fgss"])
@pytest.mark.parametrize("name", ["whole", "one", "later", "earlier", "overlap", "overlap_back", "gap", "gap_probe",
                                  "reversed", "repeat", "twice", "ids_back", "ids_back_both", "none", "last_odd"])
def test_partition_forms(ctx, tech, name):
    c = synth.generate(synth.C2, n_sets=N, universe=3000, dup_frac=0.2, seed=17)
    hc = hs.from_arrays(c.tokens, c.sizes, BLOCK, TAU)
    first, second = _forms(list(hc.blocks))[name]
    coll = ctx.upload(c.tokens, c.sizes, c.starts)

    def handler(aggregate):
        if tech == "bitmap":
            return BitmapHandler(ctx, hc, coll, 128, BLOCK, aggregate, TAU)
        return FgssHandler(ctx, hc, coll, BLOCK, aggregate, TAU)

    out, one = hs.PairsHandler(), hs.PairsHandler()
    h = handler(False)
    h.set_output_handler(one)
    for f in first:
        for s in second:
            if s.id < f.id:
                continue
            if c.sizes[f.end_id] >= similarity.minsize("jaccard", int(c.sizes[s.start_id]), TAU):
                h.join(f, s)
    h.set_output_handler(out)
    for _ in range(2):  # the second join finds the lists' lengths known
        out._chunks = []
        h.join(hs.Partition(0, first), hs.Partition(0, second))
        np.testing.assert_array_equal(_sorted(out.pairs), _sorted(one.pairs))
    if name in ("whole", "overlap", "twice", "ids_back_both"):
        assert out.get_count() > 0
    count, h = hs.CountHandler(), handler(True)
    h.set_output_handler(count)
    h.join(hs.Partition(0, first), hs.Partition(0, second))
    assert count.get_count() == one.get_count()
