"""GPU tier: what the library keeps of dropped trees and of the sort's scratch is given back on request, and before
any of its own allocations fails; captured reads hold no scratch that they did not need before."""
import pytest

pytestmark = pytest.mark.gpu
GIB = 1 << 30


def _drop_trees():
    """Two trees of 1.5 GiB, made and dropped: their blocks stay with the library."""
    import mvgpubtree_b200 as mv
    trees = [mv.gpu_blink_tree(pool_bytes=GIB + GIB // 2) for _ in range(2)]
    for t in trees:
        t.close()


def _free():
    import gc
    import torch
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # of the tests before
    return torch.cuda.mem_get_info()[0]


def test_release_memory_gives_back_what_dropped_trees_left():
    import torch
    import mvgpubtree_b200 as mv
    torch.zeros(1, device="cuda")
    mv.release_memory()
    before = _free()
    _drop_trees()
    keys = torch.arange(1, 1 << 22, dtype=torch.int32, device="cuda")
    t = mv.gpu_blink_tree(pool_bytes=1 << 28)
    t.insert(keys, keys)
    t.close()
    del keys
    assert before - _free() >= 3 * GIB
    mv.release_memory()
    assert before - _free() < GIB // 4


@pytest.mark.parametrize("what", ["rings", "plan", "sort"])
def test_own_allocations_take_what_dropped_trees_left(what):
    """With all but 1 GiB of the device in use and 3 GiB kept of dropped trees, 2 GiB more are there."""
    import torch
    import mvgpubtree_b200 as mv
    torch.zeros(1, device="cuda")
    mv.release_memory()
    n = 100_000_000
    keys = torch.randint(1, 2**31 - 2, (n,), dtype=torch.int32, device="cuda") if what == "sort" else None
    out = torch.zeros_like(keys) if what == "sort" else None
    t = mv.gpu_versioned_btree(pool_bytes=1 << 28, frontend=mv.FRONTEND_SORTED)
    _drop_trees()
    fill = torch.empty(max(0, _free() - GIB), dtype=torch.uint8, device="cuda")  # reserved, not written
    try:
        if what == "rings":  # 2 rings of 1 GiB or more, beside a node block from the pool
            big = mv.gpu_versioned_btree(pool_bytes=7 << 27, reclaim=True, chunk_nodes=1 << 20)
            big.close()
        elif what == "plan":
            t.batch_plan(500_000_000, 4).close()
        else:
            t.find(keys, out)
            assert int((out != -1).sum()) == 0 and t.check_errors() == 0
    finally:
        del fill
        torch.cuda.empty_cache()
        t.close()
        mv.release_memory()


@pytest.mark.parametrize("ranges", [False, True])
def test_captured_reads_that_are_sparse_in_the_tree_are_one_kernel(ranges):
    """A captured read of 2^20 keys that the front-end would sort otherwise: one kernel node, no allocation, and
    the replay answers for what the buffers hold then."""
    import torch
    from cuda.bindings import runtime as rt
    import mvgpubtree_b200 as mv
    n, keys = 1 << 20, torch.arange(1, (1 << 22) + 1, dtype=torch.int32, device="cuda") * 400
    t = mv.gpu_blink_tree(pool_bytes=1 << 28)
    for r in range(34):  # keys put into the tree so far: more than 128 for each of the call
        t.insert(keys, keys + r)
    q = torch.zeros(n, dtype=torch.int32, device="cuda")
    hi, out, pairs = torch.zeros_like(q), torch.zeros_like(q), torch.zeros(4 * n, dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()

    def ok(r):
        assert int(r[0]) == 0, r
        return r[1:] if len(r) > 2 else (r[1] if len(r) > 1 else None)

    ok(rt.cudaStreamBeginCapture(s.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
    if ranges:
        t.range_query(q, hi, pairs, out, 2, stream=s)
    else:
        t.find(q, out, stream=s)
    graph = ok(rt.cudaStreamEndCapture(s.cuda_stream))
    assert ok(rt.cudaGraphGetNodes(graph, 0))[1] == 1
    execs = [ok(rt.cudaGraphInstantiate(graph, 0)) for _ in range(2)]  # both at a time
    q.copy_(keys[torch.randperm(keys.numel(), device="cuda")[:n]])
    hi.copy_(q + 1)
    torch.cuda.synchronize()
    for e in execs:
        out.fill_(7)
        pairs.zero_()
        ok(rt.cudaGraphLaunch(e, s.cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(pairs[1::4] if ranges else out, q + 33) and (not ranges or torch.equal(out, torch.ones_like(q)))
    assert t.check_errors() == 0
