"""The persistent form's window classes (small, large, huge): every class and
mix of classes gives exactly the oracle's pairs, at the batch sizes, fanouts
and tree depths where the kernels' shapes change."""
import numpy as np
import pytest

from curtree_b200 import datasets as D
from curtree_b200.datasets import HostBoxes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def crt():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import curtree_b200 as C
    C._lib.load()
    return C


def windows(rng, nq, sides):
    cx, cy, s = rng.random(nq), rng.random(nq), rng.choice(sides, nq)
    return D._boxes(cx, cy, s, s * rng.choice([0.3, 1.0, 2.0], nq))


def check(crt, b, q, fanout, rt=None, **opts):
    d = crt.BBox.from_host(b)
    rt = crt.RTree(fanout)
    crt.build_rtree(d, rt)
    sb, t = O.build(b, fanout)
    want = O.canonical_pairs(*O.tree_query_pairs(t, sb, q))
    fid, tid = crt.query(rt, d, crt.BBox.from_host(q), **opts)
    got = O.canonical_pairs(fid.cpu().numpy(), tid.cpu().numpy())
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (fanout, opts)
    return len(want[0])


SMALL, LARGE, HUGE = (0.0, 1e-4, 2e-3), (3e-2, 8e-2), (0.35, 0.8, 3.0)


@pytest.mark.parametrize("fanout", [2, 3, 7, 10, 16, 17, 31, 32, 33, 48])
@pytest.mark.parametrize("sides", [SMALL, LARGE, HUGE, SMALL + LARGE + HUGE],
                         ids=["small", "large", "huge", "mixed"])
def test_classes_and_fanouts(crt, fanout, sides):
    """One class alone and all together, around a batch of 32 windows."""
    rng = np.random.default_rng(fanout)
    b = D.clustered_boxes(40_003, seed=fanout)
    for nq in (2, 31, 33, 700):
        check(crt, b, windows(rng, nq, sides), fanout, warps_per_cta=rng.choice([8, 16, 32]))


@pytest.mark.parametrize("n", [1, 2, 9, 10, 11, 100, 101, 1001])
def test_shallow_trees(crt, n):
    """Trees of no node, of a root over boxes, and of two and three levels."""
    rng = np.random.default_rng(n)
    b = D.uniform_boxes(n, seed=n, max_side=0.2)
    assert check(crt, b, windows(rng, 300, SMALL + LARGE + HUGE), 10) > 0


def test_frontiers_that_do_not_fit(crt):
    """Dense duplicates and windows spread so that a batch's frontier stops at
    every level (equal keys: input order), and identical windows (no sort
    pass runs)."""
    rng = np.random.default_rng(5)
    b = D.uniform_boxes(60_000, seed=5, max_side=2e-2)
    check(crt, b, windows(rng, 2000, (1e-3, 5e-3)), 16)
    one = windows(rng, 1, (4e-3,))
    same = HostBoxes(*(np.repeat(getattr(one, f), 500) for f in ("xmin", "ymin", "xmax", "ymax")),
                     np.arange(500, dtype=np.int32))
    check(crt, b, same, 8)
    dup = b.take(np.repeat(np.arange(300), 50))
    dup.id = np.arange(dup.n, dtype=np.int32)
    check(crt, dup, windows(rng, 1000, SMALL + HUGE), 10)


def test_special_windows_and_boxes(crt):
    """NaN, infinite and inverted windows; a box set with a NaN and an
    inverted box, where every window takes the general way."""
    rng = np.random.default_rng(6)
    b = D.uniform_boxes(30_000, seed=6)
    q = windows(rng, 400, SMALL + LARGE + HUGE)
    q.xmin[::7] = np.nan
    q.ymax[3::11] = np.inf
    q.xmin[5::13], q.xmax[5::13] = q.xmax[5::13].copy(), q.xmin[5::13].copy()
    q.ymin[6::17] = -np.inf
    check(crt, b, q, 10)
    b.xmin[123] = np.nan
    b.ymin[4567], b.ymax[4567] = b.ymax[4567] + 1, b.ymin[4567]
    check(crt, b, q, 10)


def test_overflow_of_classed_windows(crt):
    """A buffer below the pair count: the exact count is reported, nothing
    past the buffer is written, and the retry at that size succeeds."""
    import torch
    rng = np.random.default_rng(7)
    b = D.uniform_boxes(50_000, seed=7)
    q = windows(rng, 3000, SMALL + LARGE + HUGE[:1])
    d, rt = crt.build_into(crt.BBox.from_host(b), 16)
    dq = crt.BBox.from_host(q)
    want = crt.query_stats(rt, d, dq)["hits"]
    guard = 4096
    buf = torch.full((2, want // 2 + guard), -7, dtype=torch.int32, device="cuda")
    res = crt.new_result_block()
    crt.query_into(rt, d, dq, buf[0][:want // 2], buf[1][:want // 2], res)
    r = crt.read_result(res)
    assert r["overflow"] == 1 and r["required"] == want and r["count"] == 0 and r["error"] == 0
    assert bool((buf[:, want // 2:] == -7).all())
    fid, tid = crt.query(rt, d, dq, capacity=want // 2)
    sb, t = O.build(b, 16)
    ref = O.canonical_pairs(*O.tree_query_pairs(t, sb, q))
    got = O.canonical_pairs(fid.cpu().numpy(), tid.cpu().numpy())
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("opts", [dict(sort_windows=0), dict(no_contain=1), dict(warps_per_window=4),
                                  dict(stage_levels=0, chunk=64)], ids=str)
def test_options_beside_classes(crt, opts):
    """Options that turn the classes off or run beside them."""
    rng = np.random.default_rng(8)
    b = D.uniform_boxes(40_000, seed=8)
    check(crt, b, windows(rng, 1500, SMALL + LARGE + HUGE), 10, **opts)


@pytest.mark.parametrize("fanout", [2, 10, 16, 40])
@pytest.mark.parametrize("odd", [False, True])
def test_small_drop_in_batches(crt, fanout, odd):
    """Batches around the line where several warps share a window (148 * 32 / 8
    windows), on boxes that are all ordinary and on a set that is not, a
    batch of many pairs after one of few (the output is sized from the last)."""
    rng = np.random.default_rng(fanout)
    b = D.clustered_boxes(50_021, seed=fanout)
    if odd:
        b.xmax[77] = np.nan
        b.xmin[99], b.xmax[99] = b.xmax[99] + 3, b.xmin[99]
    d = crt.BBox.from_host(b)
    rt = crt.RTree(fanout)
    crt.build_rtree(d, rt)
    sb, t = O.build(b, fanout)
    for nq, sides in ((5000, SMALL), (1, HUGE), (592, SMALL + LARGE + HUGE), (593, SMALL + LARGE),
                      (40, LARGE), (16, SMALL)):
        q = windows(rng, nq, sides)
        pairs = crt.bfs_frontier(rt, d, crt.BBox.from_host(q))
        got = O.canonical_pairs(*pairs.to_host())
        want = O.canonical_pairs(*O.tree_query_pairs(t, sb, q))
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (nq, fanout)
        pairs.free()


@pytest.mark.parametrize("nq", [1, 7, 8, 8191, 8192, 8193, 65_536, 65_537])
def test_plain_offsets_at_scan_edges(crt, nq):
    """Plain offsets around the one-CTA scan's tile and its limit."""
    rng = np.random.default_rng(nq)
    b = D.uniform_boxes(5_003, seed=3)
    q = windows(rng, nq, (0.0, 1e-3, 2e-2))
    d, rt = crt.build_into(crt.BBox.from_host(b), 10)
    fid, tid, offs = crt.query(rt, d, crt.BBox.from_host(q), mode=crt.CRT_QUERY_PLAIN)
    sb, t = O.build(b, 10)
    counts = O.tree_query_stats(t, sb, q).counts
    assert np.array_equal(offs.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
    assert np.array_equal(tid.cpu().numpy(), np.repeat(np.arange(nq), counts))


@pytest.mark.parametrize("n,fanout,warps", [((1 << 25) + 5, 2, 32), (800_003, 870, 16), (3_100_003, 1740, 8)])
def test_stacks_that_leave_no_room_for_the_range_queues(crt, n, fanout, warps):
    """Trees whose stacks leave the warps no room for their queues of contained
    runs, as a query and a plan: the plain form's pairs."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(9)
    r = lambda n: torch.rand(n, generator=g, device="cuda") * 2 ** 15
    nq = 2000

    def boxes(n, side):
        x, y, w = r(n), r(n), r(n) * side
        return crt.BBox(x, y, x + w, y + w, torch.arange(n, dtype=torch.int32, device="cuda"))
    d, rt = crt.build_into(boxes(n, 1e-4), fanout)
    q = boxes(nq, 3e-2)

    def digest(fid, tid, n=None):
        out = crt.PairDigest(nq)
        out.add(fid, tid, n=n)
        return out
    fid, tid, _ = crt.query(rt, d, q, mode=crt.CRT_QUERY_PLAIN)
    want = digest(fid, tid)
    got = [digest(*crt.query(rt, d, q, warps_per_cta=warps))]
    cap = crt.query_capacity(int(fid.numel()))
    fid, tid = (torch.empty(cap, dtype=torch.int32, device="cuda") for _ in range(2))
    res = crt.new_result_block()
    plan = crt.Plan(rt, d, q, fid, tid, res, warps_per_cta=warps)
    plan.launch()
    got.append(digest(fid, tid, crt.read_result(res)["count"]))
    for other in got:
        assert torch.equal(want.counts, other.counts) and torch.equal(want.hashes, other.hashes)


def test_plain_queries_of_two_stack_sizes_on_two_threads(crt):
    """Two host threads query trees whose stacks take 214 KB and 7 KB of shared
    memory: neither makes the other's launches fail."""
    import threading

    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    r = lambda n: torch.rand(n, generator=g, device="cuda") * 2 ** 15
    x, y = r(3_200_000), r(3_200_000)
    boxes = crt.BBox(x, y, x + 5, y + 5, torch.arange(x.numel(), dtype=torch.int32, device="cuda"))
    qx, qy = r(64), r(64)
    q = crt.BBox(qx, qy, qx + 50, qy + 50, torch.arange(64, dtype=torch.int32, device="cuda"))
    trees = [crt.build_into(boxes, fanout) for fanout in (1700, 16)]
    want = [crt.query_stats(rt, d, q)["hits"] for d, rt in trees]
    bad = []

    def run(k):
        d, rt = trees[k]
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                fid, tid = (torch.empty(1 << 18, dtype=torch.int32, device="cuda") for _ in range(2))
                res = crt.new_result_block()
                for _ in range(3000):
                    crt.query_into(rt, d, q, fid, tid, res, None, crt.CRT_QUERY_PLAIN)
                if crt.read_result(res)["count"] != want[k]:
                    bad.append((k, "count differs"))
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


@pytest.mark.parametrize("nq", [31, 1023, 1024, 1025, 32_767, 32_768, 32_769, 33_793])
def test_plain_offsets_at_look_back_edges(crt, nq):
    """Plain offsets around one tile of 1024 counts and around the 32 tiles that
    a look-back reads at a time, with windows of no box, few and many."""
    rng = np.random.default_rng(nq)
    b = D.uniform_boxes(5_003, seed=3)
    q = windows(rng, nq, (0.0, 1e-3, 2e-2))
    d, rt = crt.build_into(crt.BBox.from_host(b), 10)
    fid, tid, offs = crt.query(rt, d, crt.BBox.from_host(q), mode=crt.CRT_QUERY_PLAIN)
    sb, t = O.build(b, 10)
    counts = O.tree_query_stats(t, sb, q).counts
    assert np.array_equal(offs.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
    assert np.array_equal(tid.cpu().numpy(), np.repeat(np.arange(nq), counts))
