"""SEARCHSORTED and UNIQUE at the sizes where their kernels change their course: the samples in shared
memory and what lies between them, the tiles of the compaction and the chain over them."""
import ctypes

import numpy as np
import pytest
import torch

import cupynumeric_b200 as num
from cupynumeric_b200 import _lib
from tests.helpers import to_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 8192, 8193, 12_289, 300_001])
def test_searchsorted_around_the_sample_count(cuda_device, n):
    rng = np.random.default_rng(n)
    for top in (3 * n, 5):   # mostly distinct keys; long runs of equal ones
        a = np.sort(rng.integers(0, top, n)).astype(np.int64)
        v = np.concatenate([a[:700], a[-700:], rng.integers(-2, top + 2, 3001)])
        for side in ("left", "right"):
            want = np.searchsorted(a, v, side=side)
            assert np.array_equal(num.searchsorted(a, v, side=side).to_numpy(), want)
            # the same positions from two tiles, combined
            cut, left, d_v = n // 3, int(side == "left"), to_device(v)
            pos = torch.full((v.size,), n if left else 0, dtype=torch.int64, device="cuda")
            for lo, hi in ((0, cut), (cut, n)):
                d_a = to_device(a[lo:hi])
                _lib.check(_lib.lib().b2s_searchsorted(_lib.DTYPE_CODE[a.dtype], d_a.data_ptr() if hi > lo else None, hi - lo, lo,
                                                       d_v.data_ptr(), v.size, left, pos.data_ptr(),
                                                       torch.cuda.current_stream().cuda_stream), "b2s_searchsorted")
            assert np.array_equal(pos.cpu().numpy(), want)


@pytest.mark.parametrize("dtype", [np.uint8, np.float16, np.int32, np.float64])
def test_unique_around_the_tile_size(cuda_device, dtype):
    rng = np.random.default_rng(3)
    for n in (1, 2, 4095, 4096, 4097, 8192, 8193, 70_001, 1_000_003):
        for top in (1, 2, 100, 10 * n):
            a = rng.integers(0, top, n).astype(dtype)   # (float16: infinities among them)
            assert np.array_equal(num.unique(a).to_numpy(), np.unique(a)), (n, top)


def test_unique_reports_the_count_of_every_head(cuda_device):
    n = 4096 * 40 + 17
    a = torch.arange(n, dtype=torch.int64, device="cuda")
    out, count, need = torch.empty_like(a), ctypes.c_size_t(), ctypes.c_size_t()
    lib = _lib.lib()
    _lib.check(lib.b2s_unique_workspace_bytes(n, ctypes.byref(need)), "ws")
    ws = torch.full((need.value,), 255, dtype=torch.uint8, device="cuda")   # whatever was there before
    _lib.check(lib.b2s_unique_sorted(_lib.DTYPE_CODE[np.dtype(np.int64)], a.data_ptr(), n, out.data_ptr(), ctypes.byref(count),
                                     ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "unique")
    assert count.value == n and torch.equal(out, a)


def test_unique_reports_a_wait_that_runs_out(cuda_device):
    """The library's own self-test: the first tile is processed by nobody, so the chain over the tiles gives
    up after a few thousand polls.  The workspace serves a correct call afterwards."""
    lib, stream = _lib.lib(), torch.cuda.current_stream().cuda_stream
    ws = torch.empty(2 << 20, dtype=torch.uint8, device="cuda")
    assert lib.b2s_selftest_unique_timeout(ws.data_ptr(), ws.numel(), stream) == 5   # B2S_ERR_TIMEOUT
    a = torch.arange(4096 * 40, dtype=torch.int32, device="cuda") // 3
    out, count = torch.empty_like(a), ctypes.c_size_t()
    _lib.check(lib.b2s_unique_sorted(_lib.DTYPE_CODE[np.dtype(np.int32)], a.data_ptr(), a.numel(), out.data_ptr(),
                                     ctypes.byref(count), ws.data_ptr(), ws.numel(), stream), "unique")
    assert torch.equal(out[:count.value], torch.unique(a))


@pytest.mark.parametrize("dtype", [np.uint8, np.float32, np.int64])
@pytest.mark.parametrize("n", [1, 4095, 4097, 12_289, 300_001])
def test_searchsorted_of_many_values(cuda_device, n, dtype):
    """Beyond one round of values per block the upper levels are searched in samples."""
    rng = np.random.default_rng(n)
    for m in (148 * 2048, 148 * 2048 + 1, (1 << 19) + 301):
        a = np.sort(rng.integers(0, 200, n).astype(dtype) if dtype == np.uint8 else rng.integers(0, 2 * n, n).astype(dtype))
        v = np.concatenate([a[:500], a[-500:], rng.integers(0, 250, m).astype(dtype)])[:m]
        d_a, d_v = to_device(a), to_device(v)
        for side in ("left", "right"):
            want = np.searchsorted(a, v, side=side)
            assert np.array_equal(num.searchsorted(a, v, side=side).to_numpy(), want), (m, side)
            left = int(side == "left")
            pos = torch.full((m,), n if left else 0, dtype=torch.int64, device="cuda")
            _lib.check(_lib.lib().b2s_searchsorted(_lib.DTYPE_CODE[a.dtype], d_a.data_ptr(), n, 0, d_v.data_ptr(), m, left,
                                                   pos.data_ptr(), torch.cuda.current_stream().cuda_stream), "b2s_searchsorted")
            assert np.array_equal(pos.cpu().numpy(), want), (m, side)


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.float32, torch.int64])
def test_unique_of_long_arrays(cuda_device, dtype):
    """From 2^22 keys on the tiles are twice as long."""
    for n in ((1 << 22) - 1, 1 << 22, (1 << 22) + 1, (1 << 22) + 8192, (1 << 22) + 8193):
        for top in (3, 100 if dtype == torch.uint8 else 30_000):
            a = torch.randint(0, top, (n,), device="cuda").to(dtype)
            assert torch.equal(num.unique(num.array(a)).torch(), torch.unique(a)), (n, top)
