"""Inserts and erases by whole warps (mvbt::write_warp): one op per lane, the leaves of a warp locked, copied
and written back together, full leaves split by the tile path. Checked against the oracle: dense runs
that split a leaf several times, updates, erases of present and absent keys, several warps writing at
once, snapshots in between, reclamation."""
import numpy as np
import pytest


@pytest.mark.parametrize("w,versioned,reclaim,chunk,sorted_run", [
    (8, False, False, 64, False), (16, False, False, 64, True), (8, True, True, 64, False), (16, True, True, 32, True),
    (8, True, False, 8, True)])
def test_emulated_warp_writes_match_oracle(w, versioned, reclaim, chunk, sorted_run):
    from emu import EmuTree
    import oracle
    import workload as wl
    seed = 83
    t = EmuTree(versioned, capacity=1 << 14, tiles=4, W=w, chunk=chunk, reclaim=reclaim)
    m = oracle.MVMap(versioned)
    keys = wl.distinct_keys(seed, 0, 600)
    dense = np.arange(keys[0], keys[0] + 130, dtype=np.uint32)  # more than one group in one leaf
    every = np.unique(np.concatenate([keys, dense, np.array([0, 1, 0xFFFFFFFE], np.uint32)]))
    rng = np.random.default_rng(seed)
    for r in range(4):
        op = rng.permutation(every)[: every.size * (3 if r else 4) // 4]
        kind = np.where(rng.random(op.size) < (0.35 if r else 0.0), 2, 1).astype(np.uint32)
        vals = wl.values_for(op, seed + r)
        if sorted_run:  # repeated keys: only the last op of each counts
            op, kind, vals = np.concatenate([op[:40], op]), np.concatenate([np.full(40, 1, np.uint32), kind]), np.concatenate([vals[:40] ^ 1, vals])
        t.write_warp(kind, op, vals, warps=3, sorted_run=sorted_run)
        last = {int(k): i for i, k in enumerate(op)}
        idx = np.array(sorted(last.values()))
        ok, kk, vv = op[idx], kind[idx], vals[idx]
        m.insert(ok[kk == 1], vv[kk == 1])
        m.erase(ok[kk == 2])
        assert t.errors == 0, t.stats()
        assert np.array_equal(t.find(every), m.find(every))
        if versioned:
            s = t.snapshot()
            assert s == m.take_snapshot()
            if r:
                assert np.array_equal(t.find(every, s - 1), m.find(every, s - 1))
            if reclaim and r == 2:
                t.reclaim(s)
    rep = t.validate()
    assert rep["violations"] == 0 and rep["locked_nodes"] == 0
    assert t.stats()["splits"] > 20


def test_warp_writes_wait_for_a_lock_by_the_clock():
    """A leaf that stays locked for long, but not past the wait limit, delays the warp's writes and loses none,
    however often they look at it meanwhile; one that stays locked past the limit (4 s in the emulator) is given
    up as a wait, not as a broken structure."""
    import threading
    from emu import EmuTree
    keys = np.arange(1, 9, dtype=np.uint32)
    t = EmuTree(False, capacity=1 << 10, chunk=64)
    t.hold_first_leaf(True)
    t.L.emu_slow_clock(64)
    timer = threading.Timer(8, t.hold_first_leaf, (False,))
    timer.start()
    try:
        t.write_warp(np.ones(8), keys, keys, warps=1)
    finally:
        t.L.emu_slow_clock(1)
        timer.join()
    assert t.errors == 0, t.stats()
    assert np.array_equal(t.find(keys), keys)
    t.hold_first_leaf(True)
    t.write_warp(np.ones(8), keys, keys + 1, warps=1)
    assert t.errors == 2, t.stats()
    t.hold_first_leaf(False)
    assert np.array_equal(t.find(keys), keys)


@pytest.mark.parametrize("w,versioned,every,warps", [(8, False, 1, 1), (8, True, 1, 3), (16, True, 2, 3), (8, True, 6, 1),
                                                     (8, False, 9, 3), (16, True, 20, 2)])
def test_sorted_inserts_of_new_keys_split_like_the_oracle(w, versioned, every, warps):
    """Runs of new keys in key order, so dense that a group of 32 splits one or two leaves, or so sparse that each of
    its keys may split another (fewer slots than splits), over several rounds: parents fill up and split too."""
    from emu import EmuTree
    import oracle
    t = EmuTree(versioned, capacity=1 << 14, tiles=4, W=w, chunk=64)
    m = oracle.MVMap(versioned)
    base = np.arange(1, 701, dtype=np.uint32) * 3000
    snaps = []
    for r in range(4):
        new = base[::every] + r
        t.write_warp(np.ones(new.size), new, new ^ r, warps=warps, sorted_run=True) if r else t.write_warp(np.ones(base.size), base, base)
        m.insert(new, new ^ r) if r else m.insert(base, base)
        if versioned:
            snaps.append(t.snapshot())
            assert snaps[-1] == m.take_snapshot()
        assert t.errors == 0, t.stats()
    q = np.concatenate([base + r for r in range(5)])
    for s in snaps or [0xFFFFFFFF]:
        assert np.array_equal(t.find_warp(q, s), m.find(q, s) if versioned else m.find(q)), s
        rep = t.validate(s)
        assert rep["violations"] == 0 and rep["locked_nodes"] == 0


def test_splits_without_a_node_give_up_their_key_alone():
    """The pool runs out among the splits of a sorted run: the status says so, and the tree stays whole."""
    from emu import EmuTree
    t = EmuTree(False, capacity=256, chunk=32)
    base = np.arange(1, 601, dtype=np.uint32) * 3000
    t.write_warp(np.ones(base.size), base, base)
    assert t.errors == 0
    new = np.concatenate([base + d for d in range(1, 6)])
    t.write_warp(np.ones(new.size), new, new, warps=2, sorted_run=True)
    assert t.errors == 1, t.stats()
    assert np.array_equal(t.find_warp(base), base)
    got = t.find_warp(np.sort(new))
    assert np.all((got == np.sort(new)) | (got == 0xFFFFFFFF)) and np.count_nonzero(got != 0xFFFFFFFF) > 100
    # A split that takes the last node while its parent has to split too stays without a separator, as on the tile
    # path: readers come to its right half by the link. The validator counts that once for a level below the top
    # (two at this size) and any other fault for each node it meets.
    rep = t.validate()
    assert rep["violations"] <= 2 and rep["locked_nodes"] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("versioned,tile,every", [(False, 8, 1), (True, 16, 1), (True, 8, 3), (False, 16, 11)])
def test_gpu_sorted_inserts_of_new_keys_match_oracle(versioned, tile, every):
    import torch
    import mvgpubtree_b200 as mv
    import oracle
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.uint32).view(np.int32)).cuda()
    cls = mv.gpu_versioned_btree if versioned else mv.gpu_blink_tree
    t, m = cls(pool_bytes=1 << 28, tile_width=tile, frontend=2), oracle.MVMap(versioned)
    rng = np.random.default_rng(every)
    base = rng.permutation(np.arange(1, 120_001, dtype=np.uint32)) * 30_000
    snaps = []
    for r in range(5):
        new = base[::every] + r if r else base
        t.insert(dev(new), dev(new ^ r))
        m.insert(new, new ^ r)
        if versioned:
            snaps.append(t.take_snapshot())
            assert snaps[-1] == m.take_snapshot()
    q = np.concatenate([base + r for r in range(6)])
    out = torch.zeros(q.size, dtype=torch.int32, device="cuda")
    for s in snaps[::2] or [mv.LATEST]:
        t.find(dev(q), out, timestamp=s)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), m.find(q, s) if versioned else m.find(q))
    assert t.check_errors() == 0
    rep = t.validate_tree_structure()
    assert rep["violations"] == 0 and rep["locked_nodes"] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("versioned", [False, True])
@pytest.mark.parametrize("frontend", [0, 1])
def test_gpu_writes_queueing_on_one_leaf_all_run(versioned, frontend):
    """A million erases in a tree of one leaf, and 100 000 inserts of one key: thousands of warps wait for one lock."""
    import torch
    import mvgpubtree_b200 as mv
    cls = mv.gpu_versioned_btree if versioned else mv.gpu_blink_tree
    t = cls(pool_bytes=1 << 26, frontend=frontend)
    t.erase(torch.arange(1, 1_000_001, dtype=torch.int32, device="cuda"))
    assert t.check_errors() == 0
    base = torch.arange(1, 300_000, dtype=torch.int32, device="cuda")
    t.insert(base * 5000, base)
    one = torch.full((100_000,), 777, dtype=torch.int32, device="cuda")
    t.insert(one, one)
    assert t.check_errors() == 0
    out = torch.zeros(1, dtype=torch.int32, device="cuda")
    t.find(one[:1], out)
    assert int(out) == 777
