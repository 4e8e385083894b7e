"""CPU tier: the persistent batch worker (mvbt::batched_worker) on lists and launch shapes where its claims, waits
and reclamation can go wrong, run by the emulator against the oracle."""
import numpy as np
import pytest


def _list(ops):
    """workload.Batches of ops: per batch a list of (type, key, value or upper bound, range capacity)."""
    import workload as wl
    flat = [o for b in ops for o in b]
    off = np.cumsum([0] + [len(b) for b in ops]).astype(np.uint64)
    col = lambda j, t: np.ascontiguousarray(np.array([o[j] for o in flat] or [0]).astype(t))
    cap = col(3, np.uint32)
    ends = np.cumsum(cap.astype(np.uint64))
    return wl.Batches(off, col(0, np.uint32), col(1, np.uint32), col(2, np.uint32), ends - cap, cap, int(ends[-1]))


def _insert(k, v): return (1, k, v, 0)
def _find(k): return (0, k, 0, 0)


def _same_as_oracle(t, m, b, **how):
    got, pairs = t.run_batches(b, **how)
    want, want_pairs = m.run_batches(b)
    assert t.errors == 0, t.stats()
    n = b.num_ops
    assert np.array_equal(got[:n], want[:n]) and np.array_equal(pairs[: want_pairs.size], want_pairs)


@pytest.mark.parametrize("warps,lead", [(1, 2), (2, 2), (3, 3), (4, 2), (8, 2)])
def test_reads_claimed_far_ahead_leave_warps_for_the_writes(warps, lead):
    """The first `lead` batches hold no write, so every warp takes reads first: one claim of them reaches over many
    batches, and each warp's claims need writes that no warp has taken yet."""
    from emu import EmuTree
    import oracle
    t, m = EmuTree(True, capacity=1 << 13, tiles=4 * warps, W=8), oracle.MVMap(True)
    ops = [[_find(10 * b)] if b < lead else [_insert(10 * b + 10, b + 1), _find(10 * b)] for b in range(200)]
    _same_as_oracle(t, m, _list(ops), together=True)


def _updates(keys, batches, per, reads=0, read_only=0):
    """`batches` batches of `per` updates of `keys` and `reads` lookups, then `read_only` ones that hold as many
    lookups as there were updates, and one more each."""
    rng = np.random.default_rng(5)
    out = [[_insert(int(k), b + 1) for k in rng.permutation(keys)[:per]] + [_find(int(k)) for k in rng.choice(keys, reads)]
           for b in range(batches)]
    return _list(out + [[_find(int(k)) for k in rng.choice(keys, batches * per // max(read_only, 1) + 1)] for _ in range(read_only)])


def test_chunks_of_idle_sms_go_back_before_the_ring_comes_round():
    """SMs that take a chunk from the free ring and then run nothing: a later run on fewer warps pushes more than a
    lap of the ring past the unread rest of their chunks."""
    from emu import EmuTree
    import oracle
    t, m = EmuTree(True, capacity=1 << 12, tiles=32, W=8, reclaim=True), oracle.MVMap(True)
    keys = np.arange(10, 12010, 10, dtype=np.uint32)
    t.insert(keys, keys)
    m.insert(keys, keys)
    for _ in range(3):  # 8 warps, an SM each: their chunks come from the ring
        _same_as_oracle(t, m, _updates(keys, 12, 150, 5), reclaim=True)
    assert t.stats()["reused"] > 0
    t.tiles = 4  # one warp
    before = t.stats()["reclaimed"]
    _same_as_oracle(t, m, _updates(keys, 110, 150), reclaim=True)
    assert t.stats()["reclaimed"] - before > 8192  # more than the ring holds


def test_reclamation_keeps_pace_in_batches_that_only_write():
    """Write-only batches in a list that reads more than it writes elsewhere: their copies are reclaimed while they
    run, so a pool far smaller than the copies of the whole list suffices."""
    from emu import EmuTree
    import oracle
    t, m = EmuTree(True, capacity=1 << 12, tiles=8, W=8, reclaim=True), oracle.MVMap(True)
    keys = np.arange(10, 12010, 10, dtype=np.uint32)
    t.insert(keys, keys)
    m.insert(keys, keys)
    b = _updates(keys, 60, 150, read_only=10)
    assert np.count_nonzero(b.type == 1) < np.count_nonzero(b.type == 0)
    _same_as_oracle(t, m, b, reclaim=True)
    assert t.stats()["cow"] > 4096  # more copies than the pool has nodes


def test_an_empty_list_of_batches_runs_nothing():
    from emu import EmuTree
    import oracle
    t, m = EmuTree(True, capacity=1 << 10), oracle.MVMap(True)
    _same_as_oracle(t, m, _list([]))
    assert t.snapshot() == 0
