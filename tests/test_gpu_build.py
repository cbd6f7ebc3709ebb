"""Bulk-load parity on the GPU: node arrays and the sorted box set of the CUDA
build, through the C ABI, are bit-identical to the oracle's and to the
reference's own GPU build (golden fixtures)."""
import glob
import os

import numpy as np
import pytest

from curtree_b200 import datasets as D
from curtree_b200.datasets import HostBoxes
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _bits_equal(a, b):
    a = np.asarray(a, np.float32)
    b = np.asarray(b, np.float32)
    if a.shape != b.shape:
        return False
    both_nan = np.isnan(a) & np.isnan(b)
    return bool(np.all((a.view(np.uint32) == b.view(np.uint32)) | both_nan))


@pytest.fixture(scope="module")
def crt():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import curtree_b200 as C
    C._lib.load()
    return C


def gpu_build(crt, b: HostBoxes, f: int):
    d = crt.BBox.from_host(b)
    rt = crt.RTree(f)
    rsz = crt.build_rtree(d, rt)
    return d, rt, rsz


def assert_tree_equal(crt, b, f, d, rt, rsz):
    sb, t = O.build(b, f)
    assert rsz == t.sz
    got = d.to_host()
    assert np.array_equal(got.id, sb.id), "sorted order differs"
    for k in ("xmin", "ymin", "xmax", "ymax"):
        assert _bits_equal(getattr(got, k), getattr(sb, k)), "permuted " + k
    if rsz:
        h = rt.to_host()
        for k in ("xmin", "ymin", "xmax", "ymax"):
            assert _bits_equal(getattr(h, k), getattr(t, k)), "node " + k
        assert np.array_equal(h.pos, t.pos)
        assert np.array_equal(h.len, t.len)


@pytest.mark.parametrize("f", [2, 3, 8, 10, 16, 32, 33, 100])
def test_build_matches_oracle_fanouts(crt, f):
    b = D.uniform_boxes(50_003, seed=30 + f)
    d, rt, rsz = gpu_build(crt, b, f)
    assert_tree_equal(crt, b, f, d, rt, rsz)
    rt.free()


@pytest.mark.parametrize("n", [1, 2, 7, 10, 11, 101, 8191, 8192, 8193, 100_000])
def test_build_small_and_tile_edges(crt, n):
    b = D.uniform_boxes(n, seed=n)
    d, rt, rsz = gpu_build(crt, b, 10)
    assert_tree_equal(crt, b, 10, d, rt, rsz)
    rt.free()


def test_build_uniform_1m(crt):
    b = D.uniform_boxes(1_000_000, seed=1)
    d, rt, rsz = gpu_build(crt, b, 10)
    assert rsz == 111_111
    assert_tree_equal(crt, b, 10, d, rt, rsz)


def test_build_clustered_with_duplicates_and_points(crt):
    b = D.clustered_boxes(3_000_000, seed=2, chunk=1_000_000)
    d, rt, rsz = gpu_build(crt, b, 10)
    assert_tree_equal(crt, b, 10, d, rt, rsz)


def test_build_raw_unit_data_is_identity(crt):
    b = D.uniform_boxes(20_000, seed=3, scale=False)
    d, rt, rsz = gpu_build(crt, b, 10)
    assert np.array_equal(d.to_host().id, np.arange(b.n))
    assert_tree_equal(crt, b, 10, d, rt, rsz)


def test_build_signed_keys_and_saturation(crt):
    rng = np.random.default_rng(12)
    n = 40_000
    cx = rng.uniform(-5000, 80000, n)
    cy = rng.uniform(-5000, 80000, n)
    w = rng.uniform(0, 30, n)
    b = HostBoxes(*(np.asarray(a, np.float32) for a in (cx - w, cy - w, cx + w, cy + w)),
                  np.arange(n, dtype=np.int32))
    d, rt, rsz = gpu_build(crt, b, 10)
    assert_tree_equal(crt, b, 10, d, rt, rsz)


def test_build_nan_and_signed_zero(crt):
    b = D.uniform_boxes(10_000, seed=13)
    b.xmin[10:20] = np.nan
    b.ymax[30:33] = np.nan
    b.xmin[40:60] = -0.0
    b.xmax[40:60] = 0.0
    d, rt, rsz = gpu_build(crt, b, 10)
    assert_tree_equal(crt, b, 10, d, rt, rsz)


def test_build_into_matches_in_place(crt):
    b = D.uniform_boxes(77_777, seed=14)
    d_in = crt.BBox.from_host(b)
    out, rt2 = crt.build_into(d_in, 16)
    # input untouched
    assert np.array_equal(d_in.to_host().id, b.id)
    d, rt, rsz = gpu_build(crt, b, 16)
    assert_tree_equal(crt, b, 16, out, rt2, rt2.sz)
    assert rt2.sz == rsz


def test_build_rejects_bad_arguments(crt):
    b = D.uniform_boxes(10, seed=1)
    d = crt.BBox.from_host(b)
    with pytest.raises(crt.CrtError):
        crt.build_rtree(d, crt.RTree(1))


GOLDEN = sorted(glob.glob(os.path.join(os.path.dirname(__file__), "golden", "*.npz")))


@pytest.mark.parametrize("path", GOLDEN, ids=[os.path.basename(p) for p in GOLDEN])
def test_build_matches_reference_golden(crt, path):
    z = np.load(path)
    b = HostBoxes(z["box_xmin"], z["box_ymin"], z["box_xmax"], z["box_ymax"], z["box_id"])
    f = int(z["fanout"])
    d, rt, rsz = gpu_build(crt, b, f)
    assert np.array_equal(d.to_host().id, z["sorted_id"])
    assert rsz == len(z["node_pos"])
    h = rt.to_host()
    for k in ("xmin", "ymin", "xmax", "ymax"):
        assert _bits_equal(getattr(h, k), z["node_" + k]), k
    assert np.array_equal(h.pos, z["node_pos"]) and np.array_equal(h.len, z["node_len"])
    rt.free()


@pytest.mark.parametrize("fanout", [2, 3, 7, 10, 16, 45, 46, 100, 300, 2100])
def test_levels_at_cta_and_tail_edges(crt, fanout):
    """Node arrays at sizes where a level launch's shape changes: one box past
    whole subtrees of a CTA, one CTA and several, levels of one node, and the
    last CTA's part of the tree (at most 16384 children)."""
    per = max(1, min(256, 2048 // fanout))
    sub = 1
    while sub * fanout <= per:
        sub *= fanout
    cta = per // sub * sub * fanout  # boxes of one leaf-level CTA
    for n in sorted({2, fanout, fanout + 1, cta - 1, cta, cta + 1, 3 * cta + 1, fanout * fanout + 1,
                     16384 * fanout + 1 if fanout < 20 else 2 * cta}):
        b = D.uniform_boxes(n, seed=n % 1000)
        d, rt = crt.build_into(crt.BBox.from_host(b), fanout)
        sb, t = O.build(b, fanout)
        h = rt.to_host()
        assert rt.sz == t.sz, (n, fanout)
        for f in ("xmin", "ymin", "xmax", "ymax"):
            assert np.array_equal(getattr(h, f).view(np.uint32), getattr(t, f).view(np.uint32)), (n, fanout, f)
        assert np.array_equal(h.pos, t.pos) and np.array_equal(h.len, t.len), (n, fanout)
        assert np.array_equal(d.to_host().id, sb.id)


@pytest.mark.parametrize("kind,n", [("uniform", (1 << 23) - 1), ("uniform", 1 << 23),
                                    ("clustered", (1 << 23) + 4097), ("one_corner", 8_400_001)])
def test_build_where_records_move_to_blocks(crt, kind, n):
    """Around the size from which a top byte's records fill blocks of their own:
    every top byte in use, few of them, and one that fills block after block."""
    if kind == "clustered":
        b = D.clustered_boxes(n, seed=5, chunk=n)
    else:
        b = D.uniform_boxes(n, seed=6)
        if kind == "one_corner":  # all but one box in one top byte
            s = np.float32(1 / 1024)
            cols = [(a * s).astype(np.float32) for a in (b.xmin, b.ymin, b.xmax, b.ymax)]
            for a, full in zip(cols, (b.xmin, b.ymin, b.xmax, b.ymax)):
                a[n // 2] = full.max()
            b = HostBoxes(*cols, b.id)
    d, rt, rsz = gpu_build(crt, b, 10)
    assert_tree_equal(crt, b, 10, d, rt, rsz)
    rt.free()


def test_builds_of_two_sizes_on_two_threads(crt):
    """Two host threads build sets whose sort passes ask for different amounts
    of shared memory: neither makes the other's launches fail."""
    import threading

    import torch
    sets = [D.uniform_boxes(500_000, seed=7), D.uniform_boxes(1_500_000, seed=8)]
    want = [O.build(b, 10)[0].id for b in sets]
    bad = []

    def run(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                d_in = crt.BBox.from_host(sets[k])
                for _ in range(40):
                    out, _ = crt.build_into(d_in, 10)
                    got = out.id.cpu().numpy()
                if not np.array_equal(got, want[k]):
                    bad.append((k, "order differs"))
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


@pytest.mark.parametrize("fanout", [3, 33, 48, 64, 100, 255, 300, 592, 1000, 2048, 5000])
def test_top_levels_of_large_fanouts(crt, fanout):
    """Parents whose children several threads of the last CTA share (2 to 256 of
    them), at child counts around the shares, among them NaN and signed zeros."""
    for children in sorted({2, 3, 31, 33, 65, 127, 129, 256, 257, 500, fanout + 1, 4 * fanout + 3}):
        if children * fanout > 3_000_000:
            continue
        n = (children - 1) * fanout + 1 + fanout // 3
        b = D.uniform_boxes(n, seed=children)
        for a, k in ((b.xmin, 5), (b.ymin, 7), (b.xmax, 11), (b.ymax, 13)):
            a[k::97] = np.float32(0.0)
            a[k + 1::89] = np.float32(-0.0)
            a[3 * k::1009] = np.nan
        d, rt, rsz = gpu_build(crt, b, fanout)
        assert_tree_equal(crt, b, fanout, d, rt, rsz)
        rt.free()
