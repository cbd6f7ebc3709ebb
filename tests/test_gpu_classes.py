"""The class of a window follows the density where it lies, not only the root's:
boxes of one density and one far from all others, and, for the pairs, sets whose
keys tell nothing (all alike, not in order, outside the key range)."""
import ctypes

import numpy as np
import pytest

from curtree_b200 import _lib
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


def class_counts(rt, d, q):
    fn = _lib.load()._ZN3crt19window_class_countsERK13crt_rtree_f32RK12crt_bbox_f32S5_PlP11CUstream_st
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p] * 5
    out = (ctypes.c_int64 * 3)()
    db, qb = d.c(), q.c()
    assert fn(ctypes.byref(rt.s), ctypes.byref(db), ctypes.byref(qb), out, None) == 0
    return list(out)


@pytest.mark.parametrize("n,fanout", [(1_000_000, 10), (1_300_021, 16), (900_000, 32)])
@pytest.mark.parametrize("far", [False, True])
def test_class_by_local_density(crt, n, fanout, far):
    """Windows inside uniform boxes, at 20 (small), 1000 (large) and 25000 boxes
    (huge), also where one box a thousand domains away makes the root's density
    a millionth.  A sample is n / 8192 boxes, some 120 to 160: an estimate is off
    by less than two of them, and by 10% of the samples' spacing."""
    rng = np.random.default_rng(n)
    b = D.uniform_boxes(n, seed=7, max_side=1e-6)
    if far:
        for a in (b.xmin, b.ymin, b.xmax, b.ymax):
            a[n // 2] = 3e7
    d, rt = crt.build_into(crt.BBox.from_host(b), fanout)
    nq = 500
    for hits, want in ((20, 2), (1000, 1), (25_000, 0)):
        s = np.full(nq, (hits / n) ** 0.5)
        q = D._boxes(0.2 + 0.6 * rng.random(nq), 0.2 + 0.6 * rng.random(nq), s, s)
        assert class_counts(rt, d, crt.BBox.from_host(q))[want] == nq, (hits, far)


def unit_square(b):
    return HostBoxes(*(a / np.float32(2 ** 15) for a in (b.xmin, b.ymin, b.xmax, b.ymax)), b.id)


def spread(b):
    """Coordinates from -2^17 to 2^17: keys of 0 and keys that repeat."""
    return HostBoxes(*((a - np.float32(2 ** 14)) * np.float32(8) for a in (b.xmin, b.ymin, b.xmax, b.ymax)), b.id)


@pytest.mark.parametrize("fanout", [2, 10, 16, 32])
@pytest.mark.parametrize("place", ["far", "unit", "spread", "mirrored"])
def test_pairs_where_the_keys_tell_nothing(crt, place, fanout):
    """Clustered boxes at the least count with an estimate and above it, windows
    of every class on them: the oracle's pairs."""
    rng = np.random.default_rng(fanout)
    for n in (8191, 8192, 30_011):
        b = D.clustered_boxes(n, seed=n)
        nq = 800
        pick = rng.integers(0, n, nq)
        cx, cy = ((lo[pick] / 2 + hi[pick] / 2) / 2 ** 15 for lo, hi in ((b.xmin, b.xmax), (b.ymin, b.ymax)))
        s = rng.choice([0.0, 1e-4, 2e-3, 3e-2, 0.3], nq)
        q = D._boxes(cx, cy, s, s * rng.choice([0.02, 1.0], nq))
        if place == "far":
            for a in (b.xmin, b.ymin, b.xmax, b.ymax):
                a[5] = 3e7
        elif place != "mirrored":
            b, q = ({"unit": unit_square, "spread": spread}[place](v) for v in (b, q))
        sb, t = O.build(b, fanout)
        d, rt = crt.build_into(crt.BBox.from_host(b), fanout)
        if place == "mirrored":  # the tree and its boxes, x for -x: every x key is 0 now
            q.xmin, q.xmax = -q.xmax, -q.xmin
            for lo, hi in ((sb.xmin, sb.xmax), (t.xmin, t.xmax), (d.xmin, d.xmax), rt._tensors[0:3:2]):
                old = -lo
                lo[:] = -hi
                hi[:] = old
        want = O.canonical_pairs(*O.tree_query_pairs(t, sb, q))
        for w in (8, 32):
            fid, tid = crt.query(rt, d, crt.BBox.from_host(q), warps_per_cta=w)
            got = O.canonical_pairs(fid.cpu().numpy(), tid.cpu().numpy())
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (n, w)
