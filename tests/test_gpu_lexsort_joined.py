"""Lexicographic sorts whose neighbouring keys share one 8-byte key (csrc/b2s_lexsort.cu), against np.lexsort."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

KEYS = [("float64", "int32", "int16"), ("int32", "int32"), ("float32", "uint16"), ("bool", "int8", "float16", "uint32", "int64"),
        ("int8",) * 9, ("uint16", "float32", "int16", "float64", "uint8", "int8"), ("int64", "int32", "uint64"), ("int32", "int64", "uint32", "float32")]


def _columns(names, n, seed):
    rng, out = np.random.default_rng(seed), []
    for name in names:
        d = np.dtype(name)
        if d.kind == "f":
            a = np.round(rng.standard_normal(n) * 3).astype(d)   # ties, zeros of both signs
            a[rng.integers(0, n, n // 40 + 1)] = np.nan
        elif d.kind == "b":
            a = rng.random(n) < 0.5
        else:
            info = np.iinfo(d)
            a = rng.integers(info.min, info.max, n, dtype=d, endpoint=True)
            a[rng.random(n) < 0.7] = rng.choice([info.min, 0, 1, info.max])
        out.append(a)
    return out


def _row_bytes(names, n):
    from cupynumeric_b200 import _lib

    need, codes = ctypes.c_size_t(), (ctypes.c_int * len(names))(*[_lib.DTYPE_CODE[np.dtype(d)] for d in names])
    _lib.check(_lib.lib().b2s_lexsort_workspace_bytes(len(names), codes, n, n, ctypes.byref(need)), "ws")
    return need.value / n


@pytest.mark.parametrize("names,joined", [
    # rows at which keys are joined; the others' workspace has no room for an 8-byte key
    (("int32", "int32"), [2_000_003, 4_000_037]),
    (("float32", "uint16"), [2_000_003, 4_000_037]),
    (("uint8", "uint8"), []),
    (("int16", "int16"), []),
    (("uint8",) * 8, [2_000_003, 3_000_017, 4_000_037, 16_000_057]),
], ids=lambda v: "-".join(v) if isinstance(v, tuple) else "")
def test_what_is_joined(names, joined):
    for n in (2_000_003, 3_000_017, 4_000_037, 16_000_057):
        assert (_row_bytes(names, n) > 50) == (n in joined), n


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8192, 8193, 100_003])
@pytest.mark.parametrize("names", KEYS, ids="-".join)
def test_joined_keys(names, n):
    import cupynumeric_b200 as num

    cols = _columns(names, n, n)
    assert np.array_equal(num.lexsort(cols).to_numpy(), np.lexsort(cols))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2_121_728, 2_121_729])
def test_around_the_length_where_joining_ends(n):
    import cupynumeric_b200 as num

    names = ("float64", "int32", "uint16", "int8")
    assert (_row_bytes(names[1:], n) > 50) == (n == 2_121_728)
    cols = _columns(names, n, 4)
    assert np.array_equal(num.lexsort(cols).to_numpy(), np.lexsort(cols))


@pytest.mark.gpu
def test_a_workspace_without_room_for_joined_keys():
    from cupynumeric_b200 import _lib

    n, names = 50_021, ("int16", "int32", "float16")
    cols = _columns(names, n, 3)
    tiles = [torch.from_numpy(c).cuda() for c in cols]
    lib, need, part = _lib.lib(), ctypes.c_size_t(), ctypes.c_size_t()
    codes = (ctypes.c_int * 3)(*[_lib.DTYPE_CODE[c.dtype] for c in cols])
    ptrs = (ctypes.c_void_p * 3)(*[t.data_ptr() for t in tiles])
    _lib.check(lib.b2s_lexsort_workspace_bytes(3, codes, n, n, ctypes.byref(need)), "ws")
    # what key by key takes: the widest key gathered, three orders, the largest sort
    _lib.check(lib.b2s_workspace_bytes(codes[1], n, n, 1, ctypes.byref(part)), "ws")
    up = lambda v: (v + 255) // 256 * 256   # noqa: E731
    least = up(4 * n) + 3 * up(8 * n) + up(part.value)
    assert least < need.value
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    out = torch.empty(n, dtype=torch.int64, device="cuda")
    for size, status in ((need.value, 0), (least, 0), (least - 256, 4)):
        out.zero_()
        assert lib.b2s_lexsort(3, codes, ptrs, out.data_ptr(), n, n, ws.data_ptr(), size, torch.cuda.current_stream().cuda_stream) == status
        if status == 0:
            assert np.array_equal(out.cpu().numpy(), np.lexsort(cols)), size
