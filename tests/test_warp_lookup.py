"""Lookups by whole warps (mvbt::find_warp, k_find_warp): every lane holds a key, nodes are staged in
shared memory. Checked against the oracle on trees whose snapshots, erased keys and split nodes give
every kind of step, in a sorted run (with path memory) and in the caller's order, with full and
partial groups of keys."""
import numpy as np
import pytest

ABSENT = np.array([0, 1, 2**31, 0xFFFFFFFE, 0xFFFFFFFF], np.uint32)


def _history(seed, n0):
    """Initial keys, updates, erases and late inserts with their values, and lookups of all of them."""
    import workload as wl
    keys = wl.distinct_keys(seed, 0, n0)
    late = wl.distinct_keys(seed, n0, n0 // 2)
    upd, gone = wl.shuffle(seed + 1, keys)[: n0 // 3], wl.shuffle(seed + 2, keys)[: n0 // 4]
    q = wl.shuffle(seed + 3, np.concatenate([keys, late, wl.distinct_keys(seed, wl.MISS_INDEX_BASE, n0 // 2), ABSENT]))
    v = lambda k, s: wl.values_for(k, seed + s)
    return [("insert", keys, v(keys, 0)), ("insert", upd, v(upd, 1)), ("erase", gone, None), ("insert", late, v(late, 2))], q


@pytest.mark.parametrize("versioned", [False, True])
@pytest.mark.parametrize("lanes,sorted_run,bits", [(32, False, 0), (8, False, 0), (5, False, 0), (32, True, 32), (32, True, 8)])
def test_emulated_warp_lookups_match_oracle(versioned, lanes, sorted_run, bits):
    from emu import EmuTree
    import oracle
    ops, q = _history(71, 900)
    t, m = EmuTree(versioned, capacity=1 << 14, tiles=4, W=8), oracle.MVMap(versioned)
    snaps = [0xFFFFFFFF]
    for kind, k, v in ops:
        for x in (t, m):
            x.insert(k, v) if kind == "insert" else x.erase(k)
        if versioned:
            snaps.append(t.snapshot())
            assert snaps[-1] == m.take_snapshot()
    for ts in snaps:
        for n in (1, 31, 33, q.size):
            got = t.find_warp(q[:n], ts=ts, warps=3, lanes=lanes, sorted_run=sorted_run, bits=bits)
            assert np.array_equal(got, m.find(q[:n], ts) if versioned else m.find(q[:n]))
    assert t.errors == 0


def _queries(seed, q, n):
    """Bounds around present and absent keys: empty, inverted, one key wide, over many leaves, to the end."""
    lo = np.resize(q, n).astype(np.uint64)
    width = np.resize(np.array([0, 1, 2, 1 << 20, 1 << 24, 1 << 27, 1 << 29], np.uint64), n)
    hi = np.minimum(lo + width, 0xFFFFFFFF)
    hi[::17] = lo[::17] // 2
    return lo.astype(np.uint32), hi.astype(np.uint32)


def _same_ranges(got, want, cap):
    (gp, gc), (wp, wc) = got, want
    assert np.array_equal(gc, wc)
    mask = np.arange(cap)[None, :] < np.minimum(wc, cap)[:, None]
    assert np.array_equal(gp[mask], wp[mask])
    assert np.all(gp[~mask] == 0xFFFFFFFF)  # nothing past the count


@pytest.mark.parametrize("versioned,live,sorted_run", [(False, False, False), (False, False, True), (True, False, True),
                                                       (True, False, False), (True, True, False)])
def test_emulated_warp_ranges_match_oracle(versioned, live, sorted_run):
    from emu import EmuTree
    import oracle
    ops, q = _history(73, 700)
    lo, hi = _queries(5, q, 150)
    t, m = EmuTree(versioned, capacity=1 << 14, tiles=4, W=8), oracle.MVMap(versioned)
    snaps = [] if live else [0xFFFFFFFF]
    for kind, k, v in ops:
        for x in (t, m):
            x.insert(k, v) if kind == "insert" else x.erase(k)
        if versioned:
            snaps.append(t.snapshot())
            assert snaps[-1] == m.take_snapshot()
    for ts in snaps:
        for n, cap in ((1, 4), (33, 20), (lo.size, 64)):
            want = m.range_query(lo[:n], hi[:n], cap, ts) if versioned else m.range_query(lo[:n], hi[:n], cap)
            _same_ranges(t.range_warp(lo[:n], hi[:n], cap, ts=ts, warps=3, live=live, sorted_run=sorted_run), want, cap)
    assert t.errors == 0


@pytest.mark.parametrize("versioned,lanes,w", [(False, 5, 8), (False, 32, 16), (True, 4, 16), (True, 7, 8), (True, 32, 8)])
def test_emulated_units_beside_writers_match_oracle(versioned, lanes, w):
    """The two concurrent calls by six warps: reads at the call's snapshot beside writers of the same few leaves, which
    readers find locked, changed since they were staged, or newer than their snapshot."""
    from emu import EmuTree
    import oracle
    import workload as wl
    t, m = EmuTree(versioned, capacity=1 << 14, tiles=6 * 32 // w, W=w), oracle.MVMap(versioned)
    keys = np.arange(1, 161, dtype=np.uint32) * 100
    t.write_warp(np.ones(keys.size), keys, keys)
    m.insert(keys, keys)
    for r in range(6):
        new = wl.shuffle(r, np.concatenate([keys + 1 + r, keys[::2]]))
        lo = wl.shuffle(r + 50, np.resize(keys, 400))
        hi = lo + 700
        pairs, counts = t.insert_range(new, new + r, lo, hi, 64, lanes=lanes)
        if versioned:
            want, wc = m.range_query(lo, hi, 64, m.take_snapshot())
            mask = np.arange(64)[None, :] < np.minimum(wc, 64)[:, None]
            assert np.array_equal(counts, wc) and np.array_equal(pairs[mask], want[mask])
        m.insert(new, new + r)
        gone, q = wl.shuffle(r + 9, new)[::3], wl.shuffle(r + 90, np.concatenate([new, keys]))
        got = t.find_erase(q, gone, lanes=lanes)
        was = m.find(q, m.take_snapshot()) if versioned else m.find(q)
        assert np.all((got == was) | ((not versioned) & np.isin(q, gone) & (got == 0xFFFFFFFF)))
        m.erase(gone)
        assert t.errors == 0, t.stats()
        assert np.array_equal(t.find_warp(q), m.find(q))
    rep = t.validate()
    assert rep["violations"] == 0 and rep["locked_nodes"] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("versioned,frontend", [(False, 0), (True, 1), (True, 2)])
def test_gpu_ranges_of_warps_match_oracle(versioned, frontend):
    import torch
    import mvgpubtree_b200 as mv
    import oracle
    ops, q = _history(74, 20_000)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()
    cls = mv.gpu_versioned_btree if versioned else mv.gpu_blink_tree
    t, m = cls(pool_bytes=1 << 28, frontend=frontend), oracle.MVMap(versioned)
    snaps = [mv.LATEST]
    for kind, k, v in ops:
        t.insert(dev(k), dev(v)) if kind == "insert" else t.erase(dev(k))
        m.insert(k, v) if kind == "insert" else m.erase(k)
        if versioned:
            snaps.append(t.take_snapshot())
            assert snaps[-1] == m.take_snapshot()
    lo, hi = _queries(6, q, 8193)
    for ts in snaps[:1] + snaps[2:3]:
        for cap in (1, 13, 40):
            want = m.range_query(lo, hi, cap, ts) if versioned else m.range_query(lo, hi, cap)
            for n in (8191, 8192, 8193):
                pairs = torch.full((n * cap * 2,), -1, dtype=torch.int32, device="cuda")
                counts = torch.zeros(n, dtype=torch.int32, device="cuda")
                t.range_query(dev(lo[:n]), dev(hi[:n]), pairs, counts, cap, timestamp=ts)
                got = pairs.cpu().numpy().view(np.uint32).reshape(n, cap, 2), counts.cpu().numpy().view(np.uint32)
                _same_ranges(got, (want[0][:n], want[1][:n]), cap)
    assert t.check_errors() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("versioned,block", [(False, 256), (True, 256), (True, 32), (True, 96)])
def test_gpu_lookup_sizes_around_the_rules_match_oracle(versioned, block):
    """Call sizes on both sides of the tile / warp and the unsorted / sorted rules, odd ones among them."""
    import torch
    import mvgpubtree_b200 as mv
    import oracle
    ops, q = _history(72, 40_000)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()
    cls = mv.gpu_versioned_btree if versioned else mv.gpu_blink_tree
    t, m = cls(pool_bytes=1 << 28, block_size=block), oracle.MVMap(versioned)
    snaps = [mv.LATEST]
    for kind, k, v in ops:
        t.insert(dev(k), dev(v)) if kind == "insert" else t.erase(dev(k))
        m.insert(k, v) if kind == "insert" else m.erase(k)
        if versioned:
            snaps.append(t.take_snapshot())
            assert snaps[-1] == m.take_snapshot()
    many = np.resize(q, (1 << 20) + 33)
    for ts in snaps[:1] + snaps[2:3]:
        want = m.find(q, ts) if versioned else m.find(q)
        for n in (1, 8191, 8192, 8193, (1 << 20) - 1, 1 << 20, (1 << 20) + 33):
            out = torch.zeros(n, dtype=torch.int32, device="cuda")
            t.find(dev(many[:n]), out, timestamp=ts)
            assert np.array_equal(out.cpu().numpy().view(np.uint32), np.resize(want, n))
    assert t.check_errors() == 0
