"""Sorts along another axis than the last, at shapes around the transposed copy's tiles."""
import numpy as np
import pytest
import torch

import cupynumeric_b200 as num
from tests.helpers import assert_bit_equal, random_keys

pytestmark = pytest.mark.gpu

SHAPES = [((32, 32), 0), ((31, 200), 0), ((33, 64), 0), ((64, 65), 0), ((257, 1003), 0), ((3, 65, 129), 1), ((3, 65, 40), 0),
          ((2, 5, 100, 33), 2), ((1000, 33), -2)]


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.float32, np.int64, np.complex64, np.complex128])
def test_sort_along_other_axes(cuda_device, dtype):
    rng = np.random.default_rng(1)
    for shape, axis in SHAPES:
        n = int(np.prod(shape))
        if np.dtype(dtype).kind == "c":
            a = (rng.integers(-9, 9, n) + 1j * rng.integers(-9, 9, n)).astype(dtype).reshape(shape)
        else:
            a = random_keys(rng, dtype, n, "small").reshape(shape)
            a = np.where(a == a, a + dtype(0), dtype(1))   # (no NaNs, one zero: numpy's own order is the oracle)
        assert_bit_equal(num.sort(a, axis=axis).to_numpy(), np.sort(a, axis=axis, kind="stable"), f"{shape} {axis}")
        assert np.array_equal(num.argsort(a, axis=axis, kind="stable").to_numpy(), np.argsort(a, axis=axis, kind="stable"))


def test_sort_columns_of_a_strided_view(cuda_device):
    t = torch.arange(100 * 120, device="cuda", dtype=torch.int32).flip(0).reshape(100, 120)
    view = t[::2, 5:85]
    got = num.sort(num.array(view), axis=0).torch()
    assert torch.equal(got, torch.sort(view, dim=0).values)


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.float32, torch.int64])
def test_transposed_matrices(cuda_device, dtype):
    from cupynumeric_b200 import _lib

    for shape in ((1, 64, 64), (3, 65, 129), (5, 33, 40), (7, 1, 200), (2, 200, 1)):
        a = torch.randint(0, 100, shape, device="cuda").to(dtype)
        out = torch.empty(shape[0], shape[2], shape[1], dtype=dtype, device="cuda")
        _lib.check(_lib.lib().b2s_transpose(a.element_size(), a.data_ptr(), out.data_ptr(), *shape,
                                            torch.cuda.current_stream().cuda_stream), "b2s_transpose")
        assert torch.equal(out, a.transpose(1, 2)), shape


@pytest.mark.parametrize("shape,axis", [((5, 64, 128), 1), ((70, 200, 64), 1), ((2000, 32, 32), 1), ((40, 33, 65), 1), ((33, 70_001), 0)])
def test_sort_along_other_axes_on_either_side_of_the_rule(cuda_device, shape, axis):
    for dtype in (torch.uint8, torch.int16, torch.int32, torch.float64):
        a = torch.randint(0, 100, shape, device="cuda").to(dtype)
        assert torch.equal(num.sort(num.array(a), axis=axis).torch(), torch.sort(a, dim=axis).values), (shape, dtype)
