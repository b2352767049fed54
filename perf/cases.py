"""The calls whose speed this project follows: what a program that joins set
collections on a GPU has it do, through the public entry points of the
package, over the sizes of the benchmark's configurations and below.

Inputs are seeded synthetic collections (hyset_gb300.synth) in the shapes of
the benchmark: `plain` (uniform sizes 5..50), `short` (lognormal sizes, mean
about 30) and `long` (lognormal sizes, mean about 110, up to 2,000 tokens).
Every join's pairs come back in order and in an array with room to spare,
zeros after the last, so two runs (and other inputs) can be compared.
"""
import math

import numpy as np
import torch

import hyset_gb300 as hs
from hyset_gb300 import handlers, similarity, synth

# name: (preset of hyset_gb300.synth, overrides, mean set size)
SHAPES = {
    "plain": (synth.C1, dict(dup_frac=0.05, dup_edit_lo=0.0, dup_edit_hi=0.2), 27.5),
    "short": (synth.C2, {}, 29.3),
    "long": (synth.C3, {}, 112.0),
}


def listed():
    return [
        # the smallest configuration of the benchmark: the call's latency
        dict(name="self-10k", kind="self", shape="plain", n=10_000, universe=5_000, sim="jaccard", tau=0.8),
        # the 200,000-set configuration at the ends of its threshold sweep
        dict(name="self-200k-05", kind="self", shape="short", n=200_000, universe=100_000, sim="jaccard", tau=0.5),
        dict(name="self-200k-09", kind="self", shape="short", n=200_000, universe=100_000, sim="jaccard", tau=0.9),
        # its signature (bitmap) filter, asked for by name, at the reference's default width
        dict(name="bitmap-200k", kind="bitmap", shape="short", n=200_000, universe=100_000, sim="jaccard", tau=0.7,
             bits=64),
        # the headline: a million long sets, resident, and from pinned host arrays
        dict(name="self-1m", kind="self", shape="long", n=1_000_000, universe=1_000_000, sim="jaccard", tau=0.8),
        dict(name="host-1m", kind="host", shape="long", n=1_000_000, universe=1_000_000, sim="jaccard", tau=0.8),
        # long sets under cosine (prefixes twice as long as Jaccard's)
        dict(name="cosine-300k", kind="self", shape="long", n=300_000, universe=300_000, sim="cosine", tau=0.8),
        # two collections of uneven sizes, odd counts
        dict(name="rs-dice", kind="rs", shape="long", n=61_003, n2=147_001, universe=250_007, sim="dice", tau=0.75),
        # many small joins of mixed sizes, similarities and thresholds in one call, the same batch repeatedly
        dict(name="batch-24", kind="batch", joins=24, n_max=30_000),
        # a program written for the reference's handlers: 10,000-set blocks, partition against partition
        dict(name="handler-200k", kind="handler", shape="short", n=200_000, universe=100_000, sim="jaccard", tau=0.8,
             block=10_000),
        # candidate lists from another filter, already on the device
        dict(name="verify-4m", kind="verify", shape="long", n=200_000, universe=300_000, sim="jaccard", tau=0.8,
             probes=131_072, per=32),
        # the whole of a driver's work: text from host memory to pairs
        dict(name="text-200k", kind="text", shape="long", n=200_000, universe=200_000, sim="jaccard", tau=0.8),
    ]


def _between(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["self", "self", "self", "bitmap", "host", "rs", "batch", "handler", "verify", "text"])
    if kind == "batch":
        return dict(kind=kind, joins=rng.randint(2, 24), n_max=_between(rng, 2_000, 30_000))
    shape = rng.choice(["plain", "short", "long"])
    top = {"self": 1_000_000, "host": 1_000_000, "bitmap": 150_000, "rs": 150_000, "handler": 200_000,
           "verify": 200_000, "text": 200_000}[kind]
    low = 500 if kind == "self" else 5_000
    n = _between(rng, low, min(top, 300_000) if shape != "long" else top)
    case = dict(kind=kind, shape=shape, n=n, universe=max(4_096, int(n * rng.uniform(0.4, 1.2))),
                sim=rng.choice(["jaccard", "cosine", "dice"]), tau=round(rng.uniform(0.75, 0.95), 3))
    if shape == "short" and kind == "self" and case["sim"] == "jaccard":
        case["tau"] = round(rng.uniform(0.5, 0.95), 3)
    if kind == "bitmap":
        case["bits"] = rng.choice([64, 128, 256])
    if kind == "rs":
        case["n2"] = _between(rng, low, 150_000)
    if kind == "handler":
        case["block"] = rng.choice([5_000, 10_000, 20_000])
        case["sim"] = "jaccard"
    if kind == "verify":
        case["probes"] = max(64, n // rng.randint(2, 8))
        case["per"] = rng.choice([7, 16, 32, 50])
        case["sim"] = "jaccard"
    return case


def _generate(shape, n, universe, seed, **over):
    spec, changes, _ = SHAPES[shape]
    return synth.generate(spec, **dict(changes, n_sets=n, universe=universe, seed=1 + seed, **over))


def _split(c, side):
    """The sets of c with side[i], and the others, as two collections in the same order."""
    parts = []
    for mask in (side, ~side):
        ids = np.nonzero(mask)[0]
        sizes = c.sizes[ids].astype(np.int64)
        starts = np.concatenate([[0], np.cumsum(sizes)])[:-1] if ids.size else np.zeros(0, np.int64)
        src = np.repeat(c.starts[ids].astype(np.int64) - starts, sizes) + np.arange(int(sizes.sum()))
        parts.append((c.tokens[src], c.sizes[ids], starts.astype(np.uint32)))
    return parts


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    t[:] = a
    return t


def _candidates(ctx, coll, c, case, seed):
    """Sorted probes and `per` candidates of each from its length window, as a
    CPU filter hands them over; pairs at a lower threshold are among them."""
    rng = np.random.default_rng(seed)
    found = ctx.self_join(coll, threshold=case["tau"] - 0.1, technique="fgss", probe_major=True, bitmap=256,
                          sort_pairs=True).pairs.astype(np.int64)
    probes = np.sort(rng.choice(np.arange(1, c.n), size=min(c.n - 1, case["probes"]), replace=False))
    sizes = c.sizes.astype(np.int64)
    least = np.array([similarity.minsize("jaccard", l, case["tau"]) for l in range(int(sizes.max()) + 1)])
    lo = np.searchsorted(sizes, least[sizes[probes]], side="left")
    keep = lo < probes
    probes, lo = probes[keep], lo[keep]
    cands = lo[:, None] + (rng.random((probes.size, case["per"])) * (probes - lo)[:, None]).astype(np.int64)
    at = np.searchsorted(probes, found[:, 0])
    hit = (at < probes.size) & (probes[np.minimum(at, probes.size - 1)] == found[:, 0])
    cands[at[hit], 0] = found[hit, 1]
    offsets = np.arange(1, probes.size + 1) * case["per"]
    return [torch.from_numpy(a.astype(np.int32)).cuda() for a in (probes, offsets, cands.reshape(-1))]


def prepare(case, seed):
    kind = case["kind"]
    room, arrays = (16 * case["n_max"], case["joins"]) if kind == "batch" else (4 * case["n"] + 4096, 1)
    one = np.zeros(room, np.int64) if kind in ("handler", "verify") else None
    s = dict(case=case, ctx=hs.Context(0), used=[0] * arrays,
             out=[np.zeros((room, 2), np.int32) if one is None else one for _ in range(arrays)])
    ctx = s["ctx"]
    if kind == "batch":
        rng = np.random.default_rng(seed)
        s["joins"] = []
        for j in range(case["joins"]):
            nr, ns = (int(math.exp(rng.uniform(math.log(1_000), math.log(case["n_max"])))) for _ in range(2))
            mean = math.exp(rng.uniform(math.log(12), math.log(120)))
            c = synth.generate(synth.C2, n_sets=nr + ns, universe=int(rng.uniform(2e4, 2e5)),
                               zipf_s=float(rng.uniform(0.7, 1.3)), size_a=math.log(mean) - 0.125, size_b=0.5,
                               size_min=5, size_max=int(mean * 6), dup_frac=0.05, dup_edit_lo=0.02, dup_edit_hi=0.12,
                               seed=int(rng.integers(1, 2**31)))
            r, t = (ctx.upload(*p) for p in _split(c, rng.random(c.n) < nr / (nr + ns)))
            s["joins"].append((r, t, dict(threshold=float(rng.uniform(0.6, 0.95)),
                                          sim=("jaccard", "cosine", "dice")[j % 3], sort_pairs=True)))
        return s
    c = _generate(case["shape"], case["n"] + case.get("n2", 0), case["universe"], seed)
    if kind == "host":
        s["host"] = [_pinned(a) for a in (c.tokens, c.sizes, c.starts)]
    elif kind == "text":
        s["text"] = synth.format_text(c.tokens, c.starts, c.sizes)
    elif kind == "rs":
        side = np.random.default_rng(seed).random(c.n) < case["n"] / c.n
        s["coll"], s["probe"] = (ctx.upload(*p) for p in _split(c, side))
    else:
        s["coll"] = ctx.upload(c.tokens, c.sizes, c.starts)
    if kind == "handler":
        s["blocks"] = hs.Partition(0, hs.from_arrays(c.tokens, c.sizes, case["block"], case["tau"]).blocks)
        s["handler"] = handlers.FgssHandler(ctx, None, s["coll"], case["block"], False, case["tau"])
    if kind == "verify":
        s["lists"] = _candidates(ctx, s["coll"], c, case, seed)
    return s


def _in_order(pairs):
    """Pairs of a call that has no option to sort them, as one number each."""
    return np.sort((pairs[:, 0].astype(np.int64) << 32) | pairs[:, 1])


def _whole(pairs, s, k=0):
    """The number of pairs, and the pairs in the state's k-th array, which has room for many to a set."""
    out, used = s["out"][k], min(len(pairs), len(s["out"][k]))
    out[:used] = pairs[:used]
    out[used:s["used"][k]] = 0
    s["used"][k] = used
    return len(pairs), out


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "batch":
        return [_whole(r.pairs, s, k) for k, r in enumerate(ctx.batch_join(s["joins"]))]
    opts = dict(threshold=case["tau"], sim=case["sim"], sort_pairs=True)
    if kind == "self":
        pairs = ctx.self_join(s["coll"], **opts).pairs
    elif kind == "bitmap":
        pairs = ctx.self_join(s["coll"], technique="bitmap", bitmap=case["bits"], **opts).pairs
    elif kind == "host":
        pairs = ctx.self_join_host(*s["host"], **opts).pairs
    elif kind == "rs":
        pairs = ctx.rs_join(s["coll"], s["probe"], **opts).pairs
    elif kind == "handler":
        out = hs.PairsHandler()
        s["handler"].set_output_handler(out)
        s["handler"].join(s["blocks"], s["blocks"])
        pairs = _in_order(out.pairs)
    elif kind == "verify":
        probes, offsets, cands = s["lists"]
        pairs = _in_order(ctx.verify_device(s["coll"], probes.data_ptr(), offsets.data_ptr(), cands.data_ptr(),
                                            probes.numel(), threshold=case["tau"]).pairs)
    else:
        coll = ctx.parse(s["text"])
        pairs = ctx.self_join(coll, **opts).pairs
        coll.free()
    return _whole(pairs, s)


def work(case):
    """Every token, size and start read once (or every byte of text, every
    candidate), the pairs written."""
    kind = case["kind"]
    if kind == "batch":
        sets = case["joins"] * 2 * (case["n_max"] - 1_000) / math.log(case["n_max"] / 1_000)
        return {"bytes": sets * (4 * 47 + 8 + 8 * 0.03), "flops": 0}
    mean = SHAPES[case["shape"]][2]
    n = case["n"] + case.get("n2", 0)
    out = 8 * 0.04 * n
    if kind == "text":
        return {"bytes": n * mean * 6.9 + out, "flops": 0}
    lists = case["probes"] * (8 + 4 * case["per"]) if kind == "verify" else 0
    return {"bytes": n * (4 * mean + 8) + lists + out, "flops": 0}


def exact(case, seed):
    """Whole numbers throughout."""
    return None
