"""Pair lists on the GPU at the sizes where the kernels' shapes change: the
digest's steps of 256 pairs and spans of 4096, against the oracle's digest."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def crt():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import curtree_b200 as C
    C._lib.load()
    return C


def run_windows(rng, n, nq, mean):
    """n window indices in runs of mean length `mean`, neighbouring runs
    sometimes of the same window, some windows outside [0, nq)."""
    lens = rng.geometric(1.0 / mean, 2 * n // mean + 64)
    w = np.repeat(rng.integers(-2, nq + 2, lens.size), lens)
    while w.size < n:
        w = np.concatenate([w, w])
    return w[:n].astype(np.int32)


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("mean", [1, 3, 9, 300, 5000])
def test_digest_at_step_and_span_edges(crt, mean, shift):
    """Sizes around a lane's eight pairs, a step and a span, columns on and
    off a 16-byte boundary, runs that end inside a lane, between lanes and
    between steps."""
    import torch
    rng = np.random.default_rng(mean * 10 + shift)
    nq = 37
    for n in (1, 7, 8, 9, 255, 256, 257, 511, 4095, 4096, 4097, 12_301):
        tid = run_windows(rng, n, nq, mean)
        fid = rng.integers(-2**31, 2**31, n).astype(np.int32)
        pad = np.zeros(shift, np.int32)
        put = lambda a: torch.from_numpy(np.concatenate([pad, a])).cuda()[shift:]
        dg = crt.PairDigest(nq)
        dg.add(put(fid), put(tid))
        ok = (tid >= 0) & (tid < nq)
        want_c, want_h = O.pair_hashes(fid[ok], tid[ok], nq)
        got_c, got_h, bad = dg.to_host()
        assert bad == int((~ok).sum()), (n, mean)
        assert np.array_equal(got_c, want_c) and np.array_equal(got_h, want_h), (n, mean)


@pytest.mark.parametrize("nf,nt", [(2**32, 2**32), (1, 300), (300, 1), (1, 1), (70_000, 9)])
def test_canonical_order_at_tile_edges(crt, nf, nt):
    """Sizes around the one-CTA sort's limit and the passes' tile shapes; columns whose digits are all, partly or never
    uniform (0 to 8 active passes: results in the caller's arrays whatever
    their number); signed order; arrays off a 16-byte boundary."""
    import torch
    rng = np.random.default_rng(nf % 1000 + nt % 7)
    sizes = [2, 31, 64, 65, 4096, 4097, 8191, 8192, 8193, 9217, 65_536, 65_537, 69_633, 131_071, 400_000, 400_001]
    if nf == 2**32:
        sizes += [786_433, 1_000_003, 1_212_417]
    for n in sizes:
        lo = lambda k: -2**31 if k == 2**32 else -(k // 2)
        fid = rng.integers(lo(nf), lo(nf) + nf, n).astype(np.int32)
        tid = rng.integers(lo(nt), lo(nt) + nt, n).astype(np.int32)
        pad = np.zeros(1, np.int32)
        f, t = (torch.from_numpy(np.concatenate([pad, a])).cuda()[1:] for a in (fid, tid))
        crt.canonicalize(f, t)
        order = np.lexsort((fid, tid))
        assert np.array_equal(t.cpu().numpy(), tid[order]), (n, nf, nt)
        assert np.array_equal(f.cpu().numpy(), fid[order]), (n, nf, nt)
