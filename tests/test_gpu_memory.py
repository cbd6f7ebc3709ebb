"""Calls on a device whose memory is short: a stream-ordered pool of a limited
size stands in for it (the library allocates from the device's current pool)."""
import contextlib

import numpy as np
import pytest

from curtree_b200 import datasets as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def crt():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    torch.cuda.init()
    import curtree_b200 as C
    C._lib.load()
    return C


@contextlib.contextmanager
def pool_of(nbytes):
    """The device's current pool holds at most nbytes (rounded up by the driver)
    inside the block."""
    import torch
    from cuda.bindings import runtime as rt

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r
        return r[1] if len(r) > 1 else None
    torch.zeros(1, device="cuda")
    p = rt.cudaMemPoolProps()
    p.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
    p.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
    p.location.id = 0
    p.maxSize = nbytes
    old = ok(rt.cudaDeviceGetMemPool(0))
    pool = ok(rt.cudaMemPoolCreate(p))
    ok(rt.cudaDeviceSetMemPool(0, pool))
    try:
        yield
    finally:
        torch.cuda.synchronize()
        ok(rt.cudaDeviceSetMemPool(0, old))
        ok(rt.cudaMemPoolDestroy(pool))


def windows(nq, side, seed):
    rng = np.random.default_rng(seed)
    return D._boxes(rng.random(nq), rng.random(nq), np.full(nq, side), np.full(nq, side))


def same_pairs(crt, rt, d, b, fanout, q):
    pairs = crt.bfs_frontier(rt, d, crt.BBox.from_host(q))
    got = O.canonical_pairs(*pairs.to_host())
    pairs.free()
    sb, t = O.build(b, fanout)
    want = O.canonical_pairs(*O.tree_query_pairs(t, sb, q))
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    return len(want[0])


@pytest.mark.parametrize("nq", [30_000, 60_000])
def test_drop_in_batch_after_a_query_of_many_pairs(crt, nq):
    """The size of a batch's output is first guessed from the last query's pairs
    per window: after one window with millions of them, many windows with few."""
    b = D.uniform_boxes(2_000_003, seed=1)
    d = crt.BBox.from_host(b)
    rt = crt.RTree(16)
    crt.build_rtree(d, rt)
    pairs = crt.bfs_frontier(rt, d, crt.BBox.from_host(windows(1, 3.0, 1)))
    assert pairs.sz == b.n
    pairs.free()
    q = windows(nq, 1e-4, 2)
    assert same_pairs(crt, rt, d, b, 16, q) < 40 * nq


@pytest.mark.parametrize("nq", [20_000, 40_000])
def test_drop_in_batch_whose_first_size_does_not_fit(crt, nq):
    """Guessed at 2^28 slots where 1 GiB may be allocated, then few pairs, and
    more pairs than the fallback's size."""
    b = D.uniform_boxes(500_003, seed=3)
    d = crt.BBox.from_host(b)
    rt = crt.RTree(16)
    crt.build_rtree(d, rt)
    for side in (1e-4, 5e-3):
        pairs = crt.bfs_frontier(rt, d, crt.BBox.from_host(windows(1, 3.0, 1)))
        pairs.free()
        with pool_of(1 << 30):
            same_pairs(crt, rt, d, b, 16, windows(nq, side, 4))


def test_build_whose_record_blocks_do_not_fit(crt):
    """A set large enough for records in blocks where only the tiles' own slots
    fit: 48 bytes a box and the sort's zeroed block, against 134 MB more."""
    import torch
    from cuda.bindings import runtime as rt
    n = (1 << 23) + 4321
    b = D.uniform_boxes(n, seed=6)
    src, out = crt.BBox.from_host(b), None
    with pool_of(470 << 20):
        err, _ = rt.cudaMallocAsync(48 * n + (134 << 20), 0)
        assert err == rt.cudaError_t.cudaErrorMemoryAllocation
        rt.cudaGetLastError()
        out, tree = crt.build_into(src, 10)
        torch.cuda.synchronize()
    sb, t = O.build(b, 10)
    got, nodes = out.to_host(), tree.to_host()
    assert np.array_equal(got.id, sb.id)
    for f in ("xmin", "ymin", "xmax", "ymax"):
        assert np.array_equal(getattr(got, f), getattr(sb, f)) and np.array_equal(getattr(nodes, f), getattr(t, f))
    assert np.array_equal(nodes.pos, t.pos) and np.array_equal(nodes.len, t.len)
