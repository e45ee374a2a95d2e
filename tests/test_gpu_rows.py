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
