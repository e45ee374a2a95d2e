"""1-D sorts at the lengths where the radix pass changes its tiles (csrc/b2s_launch.cuh), and where a tile
ends, against the oracle."""
import ctypes

import numpy as np
import pytest

from cupynumeric_b200 import _lib
from oracle import np_task_sort
from tests.helpers import assert_bit_equal, cabi_local_sort, random_keys

SMALL_TILE, SMALL_MAX, MEDIUM_MAX = 2048, 240 * 2048, 1 << 21


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.float16, np.int32, np.float32, np.int64, np.float64])
@pytest.mark.parametrize("n", [8193, 5 * SMALL_TILE, 5 * SMALL_TILE + 1, SMALL_MAX, SMALL_MAX + 1, MEDIUM_MAX, MEDIUM_MAX + 1])
def test_lengths_around_the_size_classes(cuda_device, dtype, n):
    rng = np.random.default_rng(n)
    for flavour in ("full", "small"):
        a = random_keys(rng, dtype, n, flavour)
        idx = np_task_sort(a, n, True, 3)
        out, _ = cabi_local_sort(a, n, False, inplace=flavour == "small")
        assert_bit_equal(out, a[idx - 3], f"sort {dtype} {n}")
        _, got = cabi_local_sort(a, n, True, index_offset=3)
        assert np.array_equal(got, idx), f"argsort {dtype} {n}"


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float32, np.float64])
@pytest.mark.parametrize("argsort", [0, 1])
def test_a_workspace_serves_every_shorter_sort(dtype, argsort):
    """Chunked sorts take their workspace once, for the longest chunk."""
    lib, need, last = _lib.lib(), ctypes.c_size_t(), 0
    sizes = sorted({8193, SMALL_MAX - 1, SMALL_MAX, SMALL_MAX + 1, 700_001, MEDIUM_MAX, MEDIUM_MAX + 1, 1 << 22, 1 << 24}
                   | {MEDIUM_MAX + 5120 * k for k in range(0, 40, 7)})
    for n in sizes:
        _lib.check(lib.b2s_workspace_bytes(_lib.DTYPE_CODE[np.dtype(dtype)], n, n, argsort, ctypes.byref(need)), "ws")
        assert need.value >= last, n
        last = need.value


# the longest 1-D sorts that the fixed scratch took when every length had one tile shape, by (bytes, argsort)
@pytest.mark.parametrize("dtype,argsort,tile", [(np.uint8, 0, 5120), (np.float16, 0, 5120), (np.int32, 0, 5120), (np.int64, 0, 7168),
                                                (np.uint8, 1, 8192), (np.float16, 1, 8192), (np.float32, 1, 8192), (np.uint64, 1, 5120)])
def test_the_fixed_scratch_takes_what_it_took(dtype, argsort, tile):
    kb, limit = np.dtype(dtype).itemsize, 32 << 20
    up = lambda v: (v + 255) // 256 * 256   # noqa: E731

    def single_shape(n):   # control block, look-back rows, two key and two position temporaries
        return up(ctrl) + up(kb * -(-n // tile) * 1024) + 2 * up(n * kb) + (2 * up(4 * n) if argsort else 0)

    lib, need = _lib.lib(), ctypes.c_size_t()
    code = _lib.DTYPE_CODE[np.dtype(dtype)]
    _lib.check(lib.b2s_workspace_bytes(code, 16, 16, argsort, ctypes.byref(need)), "ws")
    ctrl = need.value
    lo, hi = 8193, limit
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (mid, hi) if single_shape(mid) <= limit else (lo, mid)
    _lib.check(lib.b2s_workspace_bytes(code, lo, lo, argsort, ctypes.byref(need)), "ws")
    assert need.value <= limit, (lo, need.value)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1000, 100_003, 1 << 20])
def test_a_captured_sort_replays_on_new_keys(cuda_device, n):
    import torch

    lib, need = _lib.lib(), ctypes.c_size_t()
    code = _lib.DTYPE_CODE[np.dtype(np.float32)]
    _lib.check(lib.b2s_workspace_bytes(code, n, n, 1, ctypes.byref(need)), "ws")
    ws = torch.empty(max(need.value, 256), dtype=torch.uint8, device="cuda")
    keys, idx = torch.empty(n, device="cuda"), torch.empty(n, dtype=torch.int64, device="cuda")

    def argsort():
        _lib.check(lib.b2s_local_sort(code, keys.data_ptr(), None, idx.data_ptr(), n, n, 0, 1, 1, ws.data_ptr(), ws.numel(),
                                      torch.cuda.current_stream().cuda_stream), "b2s_local_sort")

    keys.normal_()
    argsort()   # (the first launch of a kernel sets its shared-memory size: not inside a capture)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        argsort()
        argsort()
    for _ in range(3):
        keys.normal_()
        graph.replay()
        want = torch.sort(keys, stable=True).indices
        assert torch.equal(idx, want)
    del graph


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1, 2])
def test_a_wait_that_runs_out_in_each_form_of_the_pass(cuda_device, which):
    """The library's own self-test in the passes of short arrays (dependent launches, a look-back window of 16),
    of long rows and of long arrays (a window of 4): the status is reported, and the workspace serves correct
    sorts of every form afterwards."""
    import torch

    lib, stream, code = _lib.lib(), torch.cuda.current_stream().cuda_stream, _lib.DTYPE_CODE[np.dtype(np.uint32)]
    ws = torch.empty(16 << 20, dtype=torch.uint8, device="cuda")
    assert lib.b2s_selftest_wait_timeout_in(which, ws.data_ptr(), 2 << 20, stream) == 0
    assert lib.b2s_check_status(ws.data_ptr(), stream) == 5          # B2S_ERR_TIMEOUT
    keys = torch.randint(0, 1 << 31, (600_000,), device="cuda").to(torch.int32)
    out = torch.empty_like(keys)
    for n, seg in ((100_000, 100_000), (600_000, 20_000), (600_000, 600_000)):
        _lib.check(lib.b2s_local_sort(code, keys.data_ptr(), out.data_ptr(), None, n, seg, 0, int(n == seg), 1, ws.data_ptr(),
                                      ws.numel(), stream), "b2s_local_sort")
        assert lib.b2s_check_status(ws.data_ptr(), stream) == 0
        assert torch.equal(out[:n].reshape(-1, seg), torch.sort(keys[:n].reshape(-1, seg), dim=1).values)
