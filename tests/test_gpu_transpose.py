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
