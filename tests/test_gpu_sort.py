"""The radix sort's passes on a plan that does not fit the keys they read (a
caller's columns that change during a call) and after a reported error: no pass
may write outside its columns."""
import ctypes

import numpy as np
import pytest

from curtree_b200 import _lib

pytestmark = pytest.mark.gpu

# SortCtrl and SortCols of csrc/sort.cuh
ERROR, ACTIVE, N_ACTIVE, BUCKETS = 32, 36, 40, 96 + 4 * 8 * 256


class SortCols(ctypes.Structure):
    _fields_ = [("key", ctypes.c_void_p * 3), ("val", ctypes.c_void_p * 3), ("flip", ctypes.c_uint32),
                ("home", ctypes.c_bool), ("make_values", ctypes.c_bool), ("drop_keys", ctypes.c_bool)]


@pytest.fixture(scope="module")
def passes():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    torch.cuda.init()
    L = _lib.load()
    size = L._ZN3crt15sort_zero_bytesEli
    size.restype, size.argtypes = ctypes.c_size_t, [ctypes.c_int64, ctypes.c_int]
    run = L._ZN3crt11sort_passesERKNS_8SortColsEliPvP11CUstream_st
    run.restype = None
    run.argtypes = [ctypes.POINTER(SortCols), ctypes.c_int64, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]

    def go(keys, plan_keys, digits, error=0):
        """Sorts `keys` (values: positions) by the plan of `plan_keys`; the
        three buffers with room for every index such a plan can give."""
        n = keys.size
        zero = np.zeros(size(n, digits), np.uint8)
        active = 0
        for d in range(digits):
            h = np.bincount((plan_keys >> np.uint32(8 * d)) & np.uint32(255), minlength=256)
            zero[BUCKETS + 1024 * d:][:1024] = (np.cumsum(h) - h).astype(np.int32).view(np.uint8)
            active |= (1 << d) if h.max() < n else 0
        zero[ERROR:ERROR + 4] = np.int32([error]).view(np.uint8)
        zero[ACTIVE:ACTIVE + 4] = np.int32([active]).view(np.uint8)
        zero[N_ACTIVE:N_ACTIVE + 4] = np.int32([bin(active).count("1")]).view(np.uint8)
        ctrl = torch.from_numpy(zero).cuda()
        buf = torch.full((2, 2, 3 * n), -7, dtype=torch.int32, device="cuda")
        buf[0, 0, :n] = torch.from_numpy(keys.view(np.int32)).cuda()
        buf[1, 0, :n] = torch.arange(n, dtype=torch.int32, device="cuda")
        c = SortCols()
        for b in range(2):
            c.key[b], c.val[b] = buf[0, b].data_ptr(), buf[1, b].data_ptr()
        torch.cuda.synchronize()
        run(ctypes.byref(c), n, digits, ctrl.data_ptr(), None)
        torch.cuda.synchronize()
        return buf.cpu().numpy()
    return go


SIZES = [20_011, 100_003, 500_009]  # one per tile shape


@pytest.mark.parametrize("n", SIZES)
def test_plan_of_the_keys(passes, n):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    out = passes(keys, keys, 4)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(out[0, 0, :n].view(np.uint32), keys[order])
    assert np.array_equal(out[1, 0, :n], order)
    assert (out[:, :, n:] == -7).all()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("digits", [1, 4])
def test_plan_of_other_keys(passes, n, digits):
    """All planned keys but one in the lowest bin, all sorted keys in the
    highest: every index a pass makes is n - 1 or more."""
    rng = np.random.default_rng(n)
    plan = np.zeros(n, np.uint32)
    plan[-1] = 0xFFFFFFFF
    keys = np.full(n, 0xFFFFFFFF, np.uint32) - rng.integers(0, 2, n, dtype=np.uint32)
    out = passes(keys, plan, digits)
    assert (out[:, :, n:] == -7).all()


@pytest.mark.parametrize("n", SIZES)
def test_pass_after_an_error(passes, n):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 32, n, dtype=np.uint32)
    out = passes(keys, keys, 4, error=_lib.CRT_ERR_DEVICE_TIMEOUT)
    assert np.array_equal(out[0, 0, :n].view(np.uint32), keys)
    assert (out[:, 1] == -7).all() and (out[:, :, n:] == -7).all()


@pytest.mark.parametrize("traversal,order,want", [(0, 0, 0), (0, _lib.CRT_ERR_DEVICE_TIMEOUT, _lib.CRT_ERR_DEVICE_TIMEOUT),
                                                  (_lib.CRT_ERR_NOT_SUPPORTED, _lib.CRT_ERR_DEVICE_TIMEOUT,
                                                   _lib.CRT_ERR_NOT_SUPPORTED)])
def test_error_of_a_window_order_is_reported(passes, traversal, order, want):
    """A persistent query whose window sort gave up says so in its result."""
    assert _lib.load()._ZN3crt20persist_result_errorEiiP11CUstream_st(traversal, order, None) == want
