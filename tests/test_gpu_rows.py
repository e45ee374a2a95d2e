"""Row sorts through the C ABI at the lengths where the on-chip kernels change their shape."""
import numpy as np
import pytest

from tests.helpers import assert_bit_equal, cabi_local_sort, random_keys
from oracle import complex_lex_argsort, np_task_sort

pytestmark = pytest.mark.gpu

# below, at and above every group size of the warp kernel (elements per thread times threads per row)
SHORT = [2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 64, 65, 100, 127, 128, 129, 200, 256, 257, 511, 512, 513]


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float16, np.int32, np.float32, np.uint64, np.float64])
@pytest.mark.parametrize("flavour", ["full", "small"])
def test_short_rows(cuda_device, dtype, flavour):
    rng = np.random.default_rng(7)
    for seg in SHORT:
        for nseg in (2, 67):   # a last warp with rows to spare
            a = random_keys(rng, dtype, nseg * seg, flavour)
            idx = np_task_sort(a, seg, True, 5, False)
            rows = np.arange(nseg).repeat(seg) * seg
            want = a[rows + idx - 5]   # the stable order's keys: the input's bits, signed zeros and NaNs included
            out, _ = cabi_local_sort(a, seg, False, ndim_is_1=False)
            assert_bit_equal(out, want, f"sort {dtype} {nseg}x{seg}")
            out, _ = cabi_local_sort(a, seg, False, ndim_is_1=False, inplace=True)
            assert_bit_equal(out, want, f"in place {dtype} {nseg}x{seg}")
            out, got = cabi_local_sort(a, seg, True, index_offset=5, ndim_is_1=False, want_keys_too=True)
            assert np.array_equal(got, idx), f"argsort {dtype} {nseg}x{seg}"
            assert_bit_equal(out, want, f"keys beside the indices {dtype} {nseg}x{seg}")


def test_short_complex_rows(cuda_device):
    rng = np.random.default_rng(8)
    for seg in SHORT:
        a = (rng.integers(-3, 4, 37 * seg) + 1j * rng.integers(-3, 4, 37 * seg)).astype(np.complex64)
        idx = complex_lex_argsort(a, seg)
        out, _ = cabi_local_sort(a, seg, False, ndim_is_1=False)
        assert_bit_equal(out, a[np.arange(37).repeat(seg) * seg + idx], f"sort 37x{seg}")
        _, got = cabi_local_sort(a, seg, True, ndim_is_1=False)
        assert np.array_equal(got, idx), f"argsort 37x{seg}"


def _long_rows(rng, dtype, nseg, seg, how):
    """Rows by how their keys spread: evenly, by a bell curve with special values, with one far outlier,
    over a handful of values, or in a narrow cluster far from zero."""
    dt, n = np.dtype(dtype), nseg * seg
    if how == "full":
        return random_keys(rng, dt, n, "full")
    if how == "few":
        return random_keys(rng, dt, n, "small")
    x = rng.standard_normal(n)
    if how == "outlier":
        x[::seg] = 1e6
    if dt.kind == "f":
        a = (x + (1e5 if how == "cluster" else 0.0)).astype(dt)
        if how == "bell":
            for v in (np.nan, -np.nan, np.inf, -np.inf, -0.0, 0.0):
                a[rng.integers(0, n, n // 300)] = v
        return a
    a = np.round(x * 50_000).astype(np.int64)
    return (a + (1 << 30) if how == "cluster" else np.abs(a)).astype(dt)


@pytest.mark.parametrize("dtype", [np.int32, np.uint32, np.float32, np.int64, np.float64])
@pytest.mark.parametrize("how", ["full", "bell", "outlier", "few", "cluster"])
def test_rows_of_one_block(cuda_device, dtype, how):
    rng = np.random.default_rng(9)
    for seg in (513, 1000, 1024, 1025, 2047, 2048, 2049, 4096, 4097, 8191, 8192):
        a = _long_rows(rng, dtype, 5, seg, how)
        if a.dtype.kind == "f":
            a[seg:2 * seg] = np.nan if how == "few" else 2.5   # a row of one value
        idx = np_task_sort(a, seg, True, 0, False)
        want = a[np.arange(5).repeat(seg) * seg + idx]
        out, _ = cabi_local_sort(a, seg, False, ndim_is_1=False)
        assert_bit_equal(out, want, f"sort {dtype} {how} 5x{seg}")
        out, got = cabi_local_sort(a, seg, True, ndim_is_1=False, want_keys_too=True, inplace=True)
        assert np.array_equal(got, idx), f"argsort {dtype} {how} 5x{seg}"
        assert_bit_equal(out, want, f"keys beside the indices {dtype} {how} 5x{seg}")


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float16, np.int32, np.float32, np.int64, np.float64])
@pytest.mark.parametrize("how", ["full", "bell", "outlier", "few", "cluster"])
def test_rows_of_one_warp(cuda_device, dtype, how):
    rng = np.random.default_rng(11)
    for seg in (65, 100, 128, 129, 256, 300, 512):
        a = _long_rows(rng, dtype, 9, seg, how)
        if a.dtype.kind == "f":
            a[seg:2 * seg] = np.nan if how == "few" else 2.5   # a row of one value
        idx = np_task_sort(a, seg, True, 0, False)
        want = a[np.arange(9).repeat(seg) * seg + idx]
        out, _ = cabi_local_sort(a, seg, False, ndim_is_1=False)
        assert_bit_equal(out, want, f"sort {dtype} {how} 9x{seg}")
        out, got = cabi_local_sort(a, seg, True, ndim_is_1=False, want_keys_too=True, inplace=True)
        assert np.array_equal(got, idx), f"argsort {dtype} {how} 9x{seg}"
        assert_bit_equal(out, want, f"keys beside the indices {dtype} {how} 9x{seg}")


def test_complex_rows_of_one_block(cuda_device):
    rng = np.random.default_rng(10)
    for seg in (600, 2000, 4097):
        a = (np.round(rng.standard_normal(5 * seg), 2) + 1j * rng.standard_normal(5 * seg)).astype(np.complex64)
        idx = complex_lex_argsort(a, seg)
        out, _ = cabi_local_sort(a, seg, False, ndim_is_1=False)
        assert_bit_equal(out, a[np.arange(5).repeat(seg) * seg + idx], f"sort 5x{seg}")


def _crowded_rows(dtype, seg, how, rng):
    """Rows for which counting by buckets is of no use: one value, three values, already in order (an outlier
    at the end takes most buckets), blocks of sixteen in order, and rows of all four kinds side by side."""
    kinds = ["one", "three", "in order", "blocks"] if how == "mixed" else [how] * 7
    rows = []
    for k in (kinds * 2)[:7]:
        if k == "one":
            x = np.full(seg, 5.0)
        elif k == "three":
            x = rng.integers(0, 3, seg).astype(float)
        else:
            x = np.sort(rng.integers(0, 60, seg)).astype(float)
            if k == "blocks":
                for i in range(0, seg, 16):
                    rng.shuffle(x[i:i + 16])
            x[-1] = 1e9 if np.dtype(dtype).itemsize > 2 else 100.0
        rows.append(x)
    a = np.concatenate(rows)
    return (a + 1j * np.tile(a[:seg], 7)).astype(dtype) if np.dtype(dtype).kind == "c" else a.astype(dtype)


@pytest.mark.parametrize("dtype", [np.uint8, np.float16, np.int32, np.float32, np.int64, np.float64, np.complex64])
@pytest.mark.parametrize("how", ["one", "three", "in order", "blocks", "mixed"])
def test_rows_whose_keys_crowd(cuda_device, dtype, how):
    rng = np.random.default_rng(12)
    for seg in (65, 128, 129, 200, 257, 512, 513, 1024, 2000, 4096, 4097, 8192):
        a = _crowded_rows(dtype, seg, how, rng)
        idx = complex_lex_argsort(a, seg) if a.dtype.kind == "c" else np_task_sort(a, seg, True, 0, False)
        out, _ = cabi_local_sort(a, seg, False, ndim_is_1=False)
        assert_bit_equal(out, a[np.arange(7).repeat(seg) * seg + idx], f"sort {dtype} {how} 7x{seg}")
        _, got = cabi_local_sort(a, seg, True, ndim_is_1=False)
        assert np.array_equal(got, idx), f"argsort {dtype} {how} 7x{seg}"
