"""Timed cases of the tree: the calls a program makes through the Python API, each with its inputs.

A case is a plain dict. `prepare` makes what a program holds before the call (a tree with its keys,
a batch plan, inputs and result buffers on the GPU), `run` is one pass of the calls. A pass can be
repeated on the same state: what it inserts it erases again or finds present the next time, and
version copies are reclaimed as a long-running program does, so the pool does not grow. Every
output is a whole number that any correct implementation gives exactly: found values, range counts
and pairs, at stated snapshots.

Kinds of case:
  find        point lookups in a standing index, at the newest state or at an older snapshot
  range       range queries into fixed slots of twice the expected length
  build       an index built from scratch, probed once and dropped (a hash-join style use)
  update      snapshot, a bulk update, and both states read back
  churn       insert new keys into a plain tree, look up, erase them again, look up
  concurrent  the two concurrent calls: inserts beside range queries, finds beside erases
  batches     mixed batches (10 % erase, 20 % insert, 50 % find, 20 % range), one snapshot a batch

Key sets are distinct uniform uint32 keys in random order, lookups hit about half the time, and
sizes follow the benchmark's workloads (2^20 plain, 2^25 versioned, 40M keys) down to single calls.
Serving traces are not among them: they are paced by wall-clock arrivals, and the batch runs that
they issue are the `batches` cases.
"""
import math

import numpy as np
import torch

import mvgpubtree_b200 as mv

NODE = 128       # bytes of a tree node
FILL = 10        # keys per leaf of a loaded tree
U32 = 1 << 32
MODES = {"persistent": mv.BATCH_PERSISTENT, "graph": mv.BATCH_GRAPH, "per_launch": mv.BATCH_PER_LAUNCH}


def listed():
    return [
        # A request's worth of lookups in a small dictionary: launch latency.
        {"name": "find_small", "kind": "find", "tree": "plain", "keys": 65536, "n": 1000, "tile": 8, "updates": 0},
        # Bulk lookups in a plain tree of as many keys (the reference's find benchmark).
        {"name": "find_1M", "kind": "find", "tree": "plain", "keys": 1 << 20, "n": 1 << 20, "tile": 8, "updates": 0},
        # The largest scan of lookups: every key at a snapshot that later updates left behind.
        {"name": "find_snapshot_32M", "kind": "find", "tree": "versioned", "keys": 1 << 25, "n": 1 << 25, "tile": 8,
         "updates": 1 << 22},
        # Lookups that are few against a large index, so neighbours share little.
        {"name": "find_sparse_40M", "kind": "find", "tree": "versioned", "keys": 40_000_000, "n": 200_003, "tile": 16,
         "updates": 0},
        # Scattered range queries on the large index.
        {"name": "range_sparse_40M", "kind": "range", "tree": "versioned", "keys": 40_000_000, "n": 250_007,
         "length": 32, "tile": 8},
        # Range queries dense enough to overlap: an analytical pass over the index.
        {"name": "range_dense_10M", "kind": "range", "tree": "versioned", "keys": 10_000_000, "n": 2_000_003,
         "length": 32, "tile": 16},
        # An index built from unordered pairs and probed: load throughput.
        {"name": "build_32M", "kind": "build", "tree": "versioned", "keys": 1 << 25, "sorted": False, "probes": 1 << 22,
         "tile": 8},
        # A bulk update under a snapshot, both states read back (the versioning benchmark).
        {"name": "update_32M", "kind": "update", "keys": 1 << 25, "n": 1 << 22, "tile": 8},
        # Keys that come and go in a plain tree of ordinary size.
        {"name": "churn_1M", "kind": "churn", "keys": 1 << 20, "n": 300_007, "tile": 8},
        # Writers beside snapshot readers in one call (the concurrent benchmark, half writes).
        {"name": "concurrent_10M", "kind": "concurrent", "keys": 10_000_000, "inserts": 500_009, "ranges": 500_000,
         "length": 32, "tile": 8},
        # A few requests' worth of mixed operations: the latency of a serving step.
        {"name": "batches_small", "kind": "batches", "keys": 1 << 20, "batches": 8, "median": 256, "mode": "graph",
         "tile": 8, "blocks": -1},
        # The headline step: 256 mixed batches on 40M keys in one launch that reclaims as it runs.
        {"name": "batches_40M", "kind": "batches", "keys": 40_000_000, "batches": 256, "median": 16384,
         "mode": "persistent", "tile": 16, "blocks": 6},
    ]


def draw(rng):
    def span(lo, hi):  # spread over the logarithm
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    tile = rng.choice((8, 16))
    kind = rng.choice(("find", "find", "range", "range", "build", "update", "churn", "concurrent", "batches", "batches"))
    if kind == "find":
        keys = span(1 << 12, 40_000_000)
        tree = rng.choice(("plain", "versioned"))
        return {"kind": kind, "tree": tree, "keys": keys, "n": span(1, 1 << 25), "tile": tile,
                "updates": keys // rng.randint(4, 16) if tree == "versioned" and rng.random() < 0.5 else 0}
    if kind == "range":
        length = span(1, 128)
        return {"kind": kind, "tree": rng.choice(("plain", "versioned")), "keys": span(1 << 14, 40_000_000),
                "n": span(1, min(2_000_003, (1 << 26) // length)), "length": length, "tile": tile}
    if kind == "build":
        keys = span(1 << 10, 1 << 25)
        return {"kind": kind, "tree": rng.choice(("plain", "versioned")), "keys": keys, "sorted": rng.random() < 0.3,
                "probes": span(1, min(keys, 1 << 22)), "tile": tile}
    if kind == "update":
        keys = span(1 << 14, 1 << 25)
        return {"kind": kind, "keys": keys, "n": span(1, keys // 8), "tile": tile}
    if kind == "churn":
        keys = span(1 << 14, 1 << 22)
        return {"kind": kind, "keys": keys, "n": span(1, keys // 2), "tile": tile}
    if kind == "concurrent":
        keys = span(1 << 16, 10_000_000)
        return {"kind": kind, "keys": keys, "inserts": span(1, min(500_009, keys // 4)),
                "ranges": span(1, min(500_000, keys // 4)), "length": span(1, 64), "tile": tile}
    mode = rng.choice(("persistent", "persistent", "graph", "per_launch", "noalloc"))
    c = {"kind": kind, "keys": 0, "batches": span(4, 32 if mode == "per_launch" else 256), "median": span(32, 16384),
         "mode": mode, "tile": tile, "blocks": rng.choice((-1, 6)) if mode in ("persistent", "graph") else -1}
    most = {"per_launch": 500_000, "noalloc": mv.NOALLOC_MAX_OPS}.get(mode, 10_000_000)
    while _batch_sizes(c).sum() > most and c["median"] > 16:
        c["median"] = c["median"] * 2 // 3
    c["keys"] = span(max(1 << 16, int(_batch_sizes(c).sum())), 40_000_000)
    return c


# ---- inputs ----
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _ints(g, lo, hi, n):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=torch.int64)


def _u32(x):
    return x.to(torch.int32)  # the low 32 bits


def _values(keys, salt):
    return _u32(((keys * 0x9E3779B1 + salt * 0x85EBCA6B) ^ (keys >> 7)) & 0xFFFFFFFE)


def _key_set(g, count):
    """Distinct keys in ascending order, at least 2 apart: key + 1 is never among them."""
    mean = max(3, int(0.98 * U32 / count))
    return torch.cumsum(_ints(g, 2, 2 * mean - 2, count), 0)


def _shuffled(g, x, n=None):
    p = torch.randperm(x.numel(), generator=g, device="cuda")
    return x[p if n is None else p[:n]]


def _lookups(g, keys, n):
    """Half of them present."""
    return keys[_ints(g, 0, keys.numel(), n)] + _ints(g, 0, 2, n)


def _bounds(g, keys, n, length):
    lo = _ints(g, 0, int(0.98 * U32), n)
    return lo, torch.clamp(lo + length * int(0.98 * U32 / keys.numel()), max=U32 - 2)


def _zeros(n, dtype=torch.int32):
    return torch.zeros(n, dtype=dtype, device="cuda")


def _tree(case, pool_nodes, reclaim=False):
    cls = mv.gpu_blink_tree if case.get("tree", "versioned") == "plain" else mv.gpu_versioned_btree
    return cls(pool_bytes=NODE * (int(pool_nodes) + (1 << 17)), tile_width=case["tile"], reclaim=reclaim)


def _loaded(case, g, pool_nodes=0, reclaim=False, extra=None):
    """A tree of case["keys"] keys (and `extra`) inserted in random order, and its sorted keys."""
    keys = _key_set(g, case["keys"])
    tree = _tree(case, 0.2 * case["keys"] + pool_nodes, reclaim)
    load = _shuffled(g, keys if extra is None else torch.cat([keys, extra(keys)]))
    tree.insert(_u32(load), _values(load, 1))
    return tree, keys


def _batch_sizes(case):
    """Lognormal batch sizes (sigma 1.5), none over 40 % of the run; a function of the case alone."""
    r = np.random.RandomState(case["batches"] * 7919 + case["median"])
    sizes = np.exp(math.log(case["median"]) + 1.5 * r.standard_normal(case["batches"]))
    sizes = np.clip(np.round(sizes), max(1, case["median"] // 16), 256 * case["median"]).astype(np.int64)
    for _ in range(8):
        sizes = np.minimum(sizes, max(1, int(0.4 * sizes.sum())))
    return sizes


def _prepare_batches(case, seed, g):
    sizes = _batch_sizes(case)
    n = int(sizes.sum())
    kind = torch.rand(n, generator=g, device="cuda")
    erase, insert = kind < 0.1, (kind >= 0.1) & (kind < 0.3)
    find, rng = (kind >= 0.3) & (kind < 0.8), kind >= 0.8
    n_erase, n_insert = int(erase.sum()), int(insert.sum())
    n_new = min(n_erase, n_insert)
    # Every erase removes a key that an insert half a run earlier (or late in the run before) made,
    # so each pass finds the tree as the one before left it; the other inserts are updates.
    made = {}

    def late(keys):
        made["new"] = _shuffled(g, keys, n_new) + 1
        return made["new"][n_new // 2:]

    copies = n // 3
    tree, keys = _loaded(case, g, 3 * copies + 2 * n_new, True, late)
    new = made["new"]
    key, arg, cap = _zeros(n, torch.int64), _zeros(n, torch.int64), _zeros(n, torch.int64)
    order = torch.arange(n_erase, device="cuda")
    key[erase] = new[(order + n_new // 2) % max(n_new, 1)] if n_new else keys[:n_erase] + 1
    fresh = torch.zeros(n_insert, dtype=torch.bool, device="cuda")
    fresh[torch.sort(torch.randperm(n_insert, generator=g, device="cuda")[:n_new]).values] = True
    put = _shuffled(g, keys, n_insert)
    put[fresh] = new
    key[insert] = put
    arg[insert] = _values(put, 2).to(torch.int64)
    key[find] = _lookups(g, keys, int(find.sum()))
    n_rng = int(rng.sum())
    length = torch.clamp(torch.floor(torch.log(torch.rand(n_rng, generator=g, device="cuda")) / math.log1p(-1 / 32)) + 1,
                         1, 1024).to(torch.int64)
    key[rng], arg[rng] = _bounds(g, keys, n_rng, length)
    cap[rng] = 2 * length
    ops = _zeros(n)
    ops[insert], ops[erase], ops[rng] = 1, 2, 3
    # The slots of all range queries, in a buffer whose size follows from the case alone: a fifth of
    # the operations with 64 pairs each on average, and room for the spread.
    room = 14 * n + (1 << 16)
    cap[rng] = torch.where(torch.cumsum(cap[rng], 0) <= room, cap[rng], 0)
    ends = torch.cumsum(cap, 0)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    s = {"case": case, "tree": tree, "off": off, "type": ops, "key": _u32(key), "arg": _u32(arg), "out_off": ends - cap,
         "cap": _u32(cap), "result": _zeros(n), "pairs": _zeros(2 * room)}
    if case["mode"] == "noalloc":
        s["off_dev"] = torch.from_numpy(off.astype(np.int64)).cuda()
    else:
        s["plan"] = tree.batch_plan(n, case["batches"])
        if case["mode"] != "per_launch":
            s["plan"].set_launch(0, case["blocks"])
            s["plan"].set_reclaim(True)
    return s


def prepare(case, seed):
    g = _gen(seed * 1000003 + 17)
    kind, n = case["kind"], case.get("n", 0)
    if kind == "find":
        tree, keys = _loaded(case, g, 2 * case["updates"])
        at = mv.LATEST
        if case["updates"]:
            at = tree.take_snapshot()
            upd = _shuffled(g, keys, case["updates"])
            tree.insert(_u32(upd), _values(upd, 3))
        s = {"tree": tree, "at": at, "q": _u32(_lookups(g, keys, n)), "out": _zeros(n)}
    elif kind == "range":
        tree, keys = _loaded(case, g)
        lo, hi = _bounds(g, keys, n, case["length"])
        slot = 2 * case["length"]
        s = {"tree": tree, "lo": _u32(lo), "hi": _u32(hi), "slot": slot, "counts": _zeros(n), "pairs": _zeros(2 * n * slot)}
    elif kind == "build":
        keys = _key_set(g, case["keys"])
        load = keys if case["sorted"] else _shuffled(g, keys)
        s = {"keys": _u32(load), "values": _values(load, 1), "q": _u32(_lookups(g, keys, case["probes"])),
             "out": _zeros(case["probes"])}
    elif kind == "update":
        tree, keys = _loaded(case, g, 4 * n, True)
        upd = _shuffled(g, keys, n)
        s = {"tree": tree, "keys": _u32(upd), "values": _values(upd, 3), "old": _zeros(n), "new": _zeros(n)}
    elif kind == "churn":
        tree, keys = _loaded(dict(case, tree="plain"), g, 2 * n)
        new = _shuffled(g, keys, n) + 1
        s = {"tree": tree, "keys": _u32(new), "values": _values(new, 3), "q": _u32(_lookups(g, keys, n)), "with": _zeros(n),
             "without": _zeros(n)}
    elif kind == "concurrent":
        ins, rq = case["inserts"], case["ranges"]
        tree, keys = _loaded(case, g, 8 * ins, True)
        new = _shuffled(g, keys, ins) + 1
        lo, hi = _bounds(g, keys, rq, case["length"])
        slot = 2 * case["length"]
        s = {"tree": tree, "keys": _u32(new), "values": _values(new, 3), "lo": _u32(lo), "hi": _u32(hi), "slot": slot,
             "counts": _zeros(rq), "pairs": _zeros(2 * rq * slot), "q": _u32(_lookups(g, keys, rq)), "found": _zeros(rq)}
    else:
        s = _prepare_batches(case, seed, g)
    s["case"] = case
    if "tree" in s:
        s["tree"].check_errors()
    return s


# ---- one pass ----
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "find":
        s["tree"].find(s["q"], s["out"], timestamp=s["at"])
        return s["out"]
    if kind == "range":
        s["tree"].range_query(s["lo"], s["hi"], s["pairs"], s["counts"], s["slot"])
        return {"counts": s["counts"], "pairs": s["pairs"]}
    if kind == "build":
        tree = _tree(case, 0.2 * case["keys"])
        if case["sorted"]:
            tree.bulk_build(s["keys"], s["values"])
        else:
            tree.insert(s["keys"], s["values"])
        tree.find(s["q"], s["out"])
        tree.close()
        return s["out"]
    tree = s["tree"]
    if kind == "update":
        before = tree.take_snapshot()
        tree.insert(s["keys"], s["values"])
        tree.find(s["keys"], s["old"], timestamp=before)
        tree.find(s["keys"], s["new"])
        tree.reclaim()
        return {"old": s["old"], "new": s["new"]}
    if kind == "churn":
        tree.insert(s["keys"], s["values"])
        tree.find(s["q"], s["with"])
        tree.erase(s["keys"])
        tree.find(s["q"], s["without"])
        return {"with": s["with"], "without": s["without"]}
    if kind == "concurrent":
        tree.concurrent_insert_range(s["keys"], s["values"], case["inserts"], s["lo"], s["hi"], case["ranges"], s["pairs"],
                                     s["slot"], s["counts"])
        tree.concurrent_find_erase(s["q"], s["found"], case["ranges"], s["keys"], case["inserts"])
        tree.reclaim()
        return {"counts": s["counts"], "pairs": s["pairs"], "found": s["found"]}
    args = (s["type"], s["key"], s["arg"], s["out_off"], s["cap"], s["result"], s["pairs"])
    if case["mode"] == "noalloc":
        tree.batch_run_noalloc(s["off_dev"], s["result"].numel(), *args)
        tree.reclaim()
    else:
        s["plan"].run(s["off"], *args, mode=MODES[case["mode"]])
        if case["mode"] == "per_launch":
            tree.reclaim()
    return {"result": s["result"], "pairs": s["pairs"]}


# ---- what a pass cannot do without ----
def _nodes(keys, visits):
    """Distinct nodes (leaves and their share of interior nodes) that `visits` random visits touch."""
    leaves = max(1.0, keys / FILL)
    return 1.1 * leaves * -math.expm1(-visits / leaves)


def work(case):
    kind, keys, n = case["kind"], case.get("keys", 0), case.get("n", 0)
    if kind == "find":  # keys in, values out, the nodes on the way
        size = 8 * n + NODE * _nodes(keys, n)
    elif kind == "range":  # bounds in, counts and pairs out
        size = n * (12 + 8 * case["length"]) + NODE * _nodes(keys, n * (1 + case["length"] / FILL))
    elif kind == "build":  # pairs in, nodes out, then the probes
        size = 8 * keys + 1.1 * NODE * keys / FILL + 8 * case["probes"] + NODE * _nodes(keys, case["probes"])
    elif kind == "update":  # a node read, its old version and its new state written; two lookups
        size = 8 * n + 3 * NODE * _nodes(keys, n) + 2 * (8 * n + 2 * NODE * _nodes(keys, n))
    elif kind == "churn":
        size = 12 * n + 4 * NODE * _nodes(keys, n) + 16 * n + 2 * NODE * _nodes(keys, n)
    elif kind == "concurrent":
        ins, rq = case["inserts"], case["ranges"]
        size = (12 * ins + 6 * NODE * _nodes(keys, ins) + rq * (12 + 8 * case["length"]) + 8 * rq +
                NODE * (_nodes(keys, rq * (1 + case["length"] / FILL)) + _nodes(keys, rq)))
    else:  # type, key, arg, offset, capacity in, result and pairs out; nodes touched once a batch
        sizes = _batch_sizes(case)
        ops = float(sizes.sum())
        size = 28 * ops + 0.2 * ops * 8 * 32
        size += NODE * sum(3 * _nodes(keys, 0.3 * b) + _nodes(keys, 0.5 * b) + _nodes(keys, 0.2 * b * 4.2) for b in sizes)
    return {"bytes": float(size), "flops": 0.0}


def tolerance(case):
    return "exact"
