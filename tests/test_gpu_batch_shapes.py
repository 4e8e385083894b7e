"""GPU tier: batch lists at the edges of the run's kernels (no write, no read, empty batches, more batches
than a block has threads, one warp in all), bulk loads at the edges of their tiles with repeated keys, and
trees made and dropped again, whose blocks and host words are reused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int64 if a.dtype.itemsize == 8 else np.int32)).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint32)


def _keep(b, keep):
    """The batches of b with the ops of `keep` (a mask) only: some become empty, or lose all writes or reads."""
    import copy
    c = copy.copy(b)
    sizes = [int(keep[int(s):int(e)].sum()) for s, e in zip(b.batch_off[:-1], b.batch_off[1:])]
    c.batch_off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    for f in ("type", "key", "arg", "out_off", "range_cap"):
        setattr(c, f, np.ascontiguousarray(getattr(b, f)[keep]))
    return c


@pytest.mark.parametrize("mode", [0, 2, "noalloc"])
@pytest.mark.parametrize("case", ["mixed", "no_writes", "no_reads", "late_writes", "empty_batches"])
@pytest.mark.parametrize("nb,one_warp", [(3, False), (700, False), (40, True)])
def test_batch_lists_at_the_edges_match_oracle(mode, case, nb, one_warp):
    import torch
    import mvgpubtree_b200 as mv
    import oracle
    import workload as wl
    n0 = 3000
    init = wl.distinct_keys(9, 0, n0)
    t = mv.gpu_versioned_btree(pool_bytes=1 << 28, block_size=32 if one_warp else 256, max_blocks=1 if one_warp else 0)
    m = oracle.MVMap(True)
    t.insert(_dev(init), _dev(wl.values_for(init, 0)))
    m.insert(init, wl.values_for(init, 0))
    gen = wl.MixGenerator(9, n0, stride=wl.stride_for(n0), fixed_batch=9)
    plan = None if mode == "noalloc" else t.batch_plan(1 << 14, 800)
    for _ in range(2):
        b = gen.generate(nb)
        batch = np.repeat(np.arange(nb), np.diff(b.batch_off.astype(np.int64)))
        write = (b.type == 1) | (b.type == 2)
        keep = {"mixed": np.ones(b.num_ops, bool), "no_writes": ~write, "no_reads": write,
                "late_writes": ~write | (batch >= nb // 2), "empty_batches": batch % 3 == 1}[case]
        c = _keep(b, keep)
        n = int(c.batch_off[-1])
        result = torch.zeros(n, dtype=torch.int32, device="cuda")
        pairs = torch.full((max(1, int(b.range_pairs)) * 2,), -1, dtype=torch.int32, device="cuda")
        ops = [_dev(x) for x in (c.type, c.key, c.arg, c.out_off, c.range_cap)]
        if mode == "noalloc":
            t.batch_run_noalloc(_dev(c.batch_off), n, *ops, result, pairs)
        else:
            plan.run(c.batch_off, *ops, result, pairs, mode=mode)
        t.check_errors()
        want, want_pairs = m.run_batches(c)
        assert np.array_equal(_host(result), want)
        assert np.array_equal(_host(pairs), want_pairs)
    assert t.take_snapshot() == m.take_snapshot()


@pytest.mark.parametrize("mode", [0, "noalloc"])
@pytest.mark.parametrize("block", [64, 96, 128, 256])
def test_late_writes_in_one_block_match_oracle(mode, block):
    """2, 3, 4 and 8 warps in all and a list whose first batches only read: the first claims of the warps are
    reads that reach over many batches, and wait for writes that are not claimed yet."""
    import torch
    import mvgpubtree_b200 as mv
    import oracle
    import workload as wl
    n0, nb = 3000, 200
    init = wl.distinct_keys(9, 0, n0)
    t = mv.gpu_versioned_btree(pool_bytes=1 << 28, block_size=block, max_blocks=1)
    m = oracle.MVMap(True)
    t.insert(_dev(init), _dev(wl.values_for(init, 0)))
    m.insert(init, wl.values_for(init, 0))
    gen = wl.MixGenerator(9, n0, stride=wl.stride_for(n0), fixed_batch=4)
    b = gen.generate(nb)
    batch = np.repeat(np.arange(nb), np.diff(b.batch_off.astype(np.int64)))
    c = _keep(b, ~((b.type == 1) | (b.type == 2)) | (batch >= 3))
    n = int(c.batch_off[-1])
    result = torch.zeros(n, dtype=torch.int32, device="cuda")
    pairs = torch.full((max(1, int(b.range_pairs)) * 2,), -1, dtype=torch.int32, device="cuda")
    ops = [_dev(x) for x in (c.type, c.key, c.arg, c.out_off, c.range_cap)]
    if mode == "noalloc":
        t.batch_run_noalloc(_dev(c.batch_off), n, *ops, result, pairs)
    else:
        t.batch_plan(n, nb).run(c.batch_off, *ops, result, pairs, mode=mode)
    assert t.check_errors() == 0
    want, want_pairs = m.run_batches(c)
    assert np.array_equal(_host(result), want)
    assert np.array_equal(_host(pairs), want_pairs)


@pytest.mark.parametrize("n", [4096, 4097, 10239, 10240, 10241])
def test_loads_at_tile_edges_keep_the_last_of_each_key(n):
    import torch
    import mvgpubtree_b200 as mv
    rng = np.random.default_rng(n)
    keys = rng.choice(np.concatenate([rng.integers(1, 2**32 - 2, n // 2, np.uint32), np.array([0, 0xFFFFFFFF], np.uint32)]), n)
    keys[:700] = keys[0]  # one key over many positions of a tile
    vals = rng.integers(0, 2**32 - 1, n, np.uint32)
    last = {int(k): int(v) for k, v in zip(keys, vals) if k != 0xFFFFFFFF}
    for cls in (mv.gpu_blink_tree, mv.gpu_versioned_btree):
        t = cls(pool_bytes=1 << 26)
        t.insert(_dev(keys), _dev(vals))
        q = np.array(sorted(last) + [7, 0xFFFFFFFF], np.uint32)
        out = torch.zeros(q.size, dtype=torch.int32, device="cuda")
        t.find(_dev(q), out)
        assert np.array_equal(_host(out), np.array([last.get(int(k), 0xFFFFFFFF) for k in q], np.uint32))
        assert t.validate_tree_structure()["violations"] == 0
        t.close()


def test_trees_made_and_dropped_reuse_their_memory():
    import torch
    import mvgpubtree_b200 as mv
    keys = _dev(np.arange(10, 6010, dtype=np.uint32))
    out = torch.zeros(6000, dtype=torch.int32, device="cuda")
    trees = []
    for r in range(150):  # more at once than a page of host words holds
        t = (mv.gpu_versioned_btree if r % 2 else mv.gpu_blink_tree)(pool_bytes=(1 + r % 3) << 24)
        t.find(keys, out)
        assert int((out != -1).sum()) == 0  # a reused block starts as an empty tree
        t.insert(keys, keys)
        if r % 2:
            assert t.take_snapshot() == 0
        trees.append(t)
        if r % 4 == 3:
            trees.pop(len(trees) // 2).close()
    for t in trees:
        t.find(keys, out)
        assert torch.equal(out, keys) and t.check_errors() == 0
        t.close()


@pytest.mark.parametrize("shape", [{}, {"max_blocks": 1}, {"block_size": 32, "max_blocks": 2}, {"tile_width": 16}])
def test_unsorted_inserts_into_a_growing_tree_run_in_launches(shape):
    """Sizes on both sides of the launches' lines, down to a grid of one block: every key is there afterwards."""
    import torch
    import mvgpubtree_b200 as mv
    few = "max_blocks" in shape
    t = mv.gpu_blink_tree(pool_bytes=1 << 28, frontend=mv.FRONTEND_UNSORTED, **shape)
    keys = torch.randperm(1 << 21, device="cuda").to(torch.int32) * 1000 + 1
    done = 0
    for n in (1, 8191, 8192, 8193, 30_000) if few else (1, 8192, 100_003, 400_000, 1_200_000):
        t.insert(keys[done:done + n], keys[done:done + n] ^ 5)
        done += n
        out = torch.zeros(done, dtype=torch.int32, device="cuda")
        t.find(keys[:done].contiguous(), out)
        assert torch.equal(out, keys[:done] ^ 5)
    assert t.check_errors() == 0
    assert t.validate_tree_structure()["violations"] == 0
