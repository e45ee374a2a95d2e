"""Host-side dispatch of the SORT task: axis handling and task construction.

Mirrors the routing of ``cupynumeric/_thunk/_sort.py:37-136`` (same function names and
argument meaning) on top of device-resident tiles instead of Legate stores:

* ``sort_deferred``  0-D / ``axis=None`` / last-axis / other-axis routing   (ref ``:110-136``)
* ``sort_flattened`` ``axis=None`` on an N-D array: sort the C-order flattening (ref ``:37-47``)
* ``sort_swapped``   other axes: swap to last, dense copy, sort, swap back   (ref ``:50-76``)
* ``sort_task``      one point task per process on its tile                  (ref ``:79-107``)
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch
from numpy.exceptions import AxisError
from numpy.lib.array_utils import normalize_axis_index

from .. import _lib
from ..runtime import runtime
from .deferred import DeferredArray, create_deferred_thunk, to_numpy_dtype


# Segments of up to this many elements are sorted on chip (SEG_CAP in csrc/b2s_launch.cuh) by kernels
# that wait for nothing: there is no status to collect.
ON_CHIP = 8192


def local_sort_tile(tile: torch.Tensor, argsort: bool, stable: bool, index_offset: int = 0,
                    out: torch.Tensor | None = None) -> torch.Tensor:
    """Runs the point task body on one dense row-major tile: sorts along the last axis.

    This is the call the reference's ``SortImplBody<GPU>`` makes into ``local_sort``
    (``src/cupynumeric/sort/sort.cu:1881-1891``), here into ``b2s_local_sort``.
    """
    lib = _lib.lib()
    assert tile.is_cuda and tile.is_contiguous()
    code = _lib.DTYPE_CODE[to_numpy_dtype(tile.dtype)]
    volume = tile.numel()
    segment = tile.shape[-1] if tile.ndim else 1
    if out is None:
        out = torch.empty(tile.shape, dtype=torch.int64 if argsort else tile.dtype, device=tile.device)
    if volume == 0:
        return out
    need = ctypes.c_size_t(0)
    _lib.check(lib.b2s_workspace_bytes(code, volume, segment, int(argsort), ctypes.byref(need)),
               "b2s_workspace_bytes")
    device = torch.cuda.current_device()
    stream = torch.cuda.current_stream(device).cuda_stream
    own = runtime.scratch(need.value, device, stream)
    st = lib.b2s_local_sort(code, tile.data_ptr(), None if argsort else out.data_ptr(),
                            out.data_ptr() if argsort else None, volume, segment, int(index_offset),
                            int(tile.ndim == 1), int(stable), own.ptr, own.nbytes, stream)
    _lib.check(st, "b2s_local_sort")
    if segment > ON_CHIP and tile.dtype != torch.complex128:  # (its inner sorts keep their control blocks elsewhere)
        runtime.note_sort(own)
    return out


def sort_flattened(output: DeferredArray, input: DeferredArray, argsort: bool, stable: bool) -> None:
    flat = input.reshape((input.size,), order="C")
    result = create_deferred_thunk(flat.shape, dtype=output.dtype)
    sort_deferred(result, flat, argsort, stable=stable)
    output.base, output.global_lo, output.tiled_axis = result.base, result.global_lo, result.tiled_axis


def _transposes(size: int, batch: int, rows: int, cols: int) -> bool:
    """Whether the tiled transpose is the faster copy of ``batch`` matrices of elements of ``size`` bytes.

    Its tiles are 64 x 64 elements, and what they cost hardly depends on how full they are.  Measured against
    torch's strided copy at 2^22 elements: many small matrices break even where the tiles are 0.7, 0.6, 0.5 and
    0.6 full for 1, 2, 4 and 8 bytes (100000 x 32 x 32, a quarter full: uint8 448 against 181 us; 5000 x 64 x 100:
    float32 54 against 91).  One long matrix pays from half full on, since torch reads a sector per element there
    (float32 2^20 x 33: 74 against 632 us), but for bytes in short rows."""
    if size > 8 or min(rows, cols) < 32:
        return False
    fill = rows * cols / (-(-rows // 64) * -(-cols // 64) * 4096)
    long = batch == 1 and not (size == 1 and cols < 64)
    return fill >= (0.5 if long else {1: 0.7, 2: 0.6, 4: 0.5, 8: 0.6}[size])


def _transpose(moved: DeferredArray, input: DeferredArray, sort_axis: int) -> bool:
    """Fills ``moved`` with the dense copy of ``input`` whose last two axes are swapped, tile by tile
    through shared memory.  False (nothing done) where that is not the copy that is wanted: other axes, a
    strided or conjugated input, shapes that torch copies faster, more tiles than a grid holds."""
    t = input.base
    if sort_axis != input.ndim - 2 or not t.is_contiguous() or t.is_conj() or t.is_neg() or not t.is_cuda:
        return False
    rows, cols = t.shape[-2:]
    size = t.element_size()
    batch = t.numel() // max(rows * cols, 1)
    if not _transposes(size, batch, rows, cols) or t.numel() >= 1 << 40:
        return False
    swapped = input.swapaxes(sort_axis, input.ndim - 1)
    out = torch.empty(swapped.shape, dtype=t.dtype, device=t.device)
    _lib.check(_lib.lib().b2s_transpose(size, t.data_ptr(), out.data_ptr(), batch, rows, cols, runtime.stream_handle()),
               "b2s_transpose")
    moved.base = out
    moved.global_lo, moved.tiled_axis = swapped.global_lo, swapped.tiled_axis
    return True


def sort_swapped(output: DeferredArray, input: DeferredArray, argsort: bool, sort_axis: int,
                 stable: bool) -> None:
    sort_axis = normalize_axis_index(sort_axis, input.ndim)
    last = input.ndim - 1
    moved = create_deferred_thunk(input.swapaxes(sort_axis, last).shape, dtype=input.dtype)
    if not _transpose(moved, input, sort_axis):
        moved.copy(input.swapaxes(sort_axis, last), deep=True)
    if argsort:
        result = create_deferred_thunk(moved.shape, dtype=output.dtype)
        sort_deferred(result, moved, argsort, stable=stable)
        back = result.swapaxes(last, sort_axis)
    else:
        sort_deferred(moved, moved, argsort, stable=stable)
        back = moved.swapaxes(last, sort_axis)
    output.base, output.global_lo, output.tiled_axis = back.base, back.global_lo, back.tiled_axis


def sort_task(output: DeferredArray, input: DeferredArray, argsort: bool, stable: bool) -> None:
    """One point task per process on its tile; the tile's last axis is the sort axis.

    A 1-D array held by several processes gets an "unbound" output: each process ends up with
    however many elements fall between its splitters (ref ``:87,99-103``); N-D arrays are tiled
    by rows, so every segment is local and no exchange happens (the reference reaches the same
    state: ``need_distributed_sort == false``, ``src/cupynumeric/sort/sort.cu:1825``).
    """
    tile = input.base if input.base.is_contiguous() else input.base.contiguous()
    if runtime.num_procs > 1 and input.ndim > 1 and input.tiled_axis == input.ndim - 1:
        sort_split_axis(output, input, tile, argsort)
        return
    uses_unbound_output = runtime.num_procs > 1 and input.ndim == 1
    if uses_unbound_output:
        from .._dist import dist_sort_1d

        output.base, output.global_lo = dist_sort_1d(tile, argsort, input.global_lo)
        return
    # write straight into the output's memory when it is already there (in-place ndarray.sort)
    out = output.base if (not argsort and output.base is not None and output.base.is_contiguous()
                          and output.base.shape == tile.shape and output.base.dtype == tile.dtype) else None
    output.base = local_sort_tile(tile, argsort, stable,
                                  index_offset=input.global_lo if input.ndim == 1 else 0, out=out)
    output.global_lo, output.tiled_axis = input.global_lo, input.tiled_axis


def sort_split_axis(output: DeferredArray, input: DeferredArray, tile: torch.Tensor, argsort: bool) -> None:
    """N-D tile whose sort (last) axis is the one split over the processes: every row is a 1-D
    array spanning the ranks, and the output store is bound and aligned with the input, so every
    rank must end up with exactly its own extent of every sorted row (the reference:
    sample_sort_nccl_nd over all segments + rebalance_data,
    ``src/cupynumeric/sort/sort.cu:1759-1773,799-1261``).  With at least as many rows as ranks all
    rows go through one call (``b2s_dist_sort_nd``: rows dealt out, completed by one exchange,
    sorted, returned by another).  Fewer rows than ranks would leave ranks idle that way: each row
    then takes the distributed 1-D sort and is moved back into this rank's extent."""
    from .._dist import dist_sort_1d, dist_sort_nd, rebalance_1d

    extent = tile.shape[-1]
    rows = tile.reshape(-1, extent)
    if rows.shape[0] >= runtime.num_procs:
        out = dist_sort_nd(rows, argsort)
    else:
        out = torch.empty(rows.shape, dtype=torch.int64 if argsort else tile.dtype, device=tile.device)
        for i in range(rows.shape[0]):
            part, start = dist_sort_1d(rows[i], argsort, input.global_lo)
            rebalance_1d(part, start, out[i], input.global_lo)
    output.base = out.reshape(tile.shape)
    output.global_lo, output.tiled_axis = input.global_lo, input.tiled_axis


def sort_deferred(output: DeferredArray, input: DeferredArray, argsort: bool, axis: int | None = -1,
                  stable: bool = False) -> None:
    if input.ndim == 0:
        if axis is not None:
            raise AxisError(axis, input.ndim)
        output.base = input.base
        return
    if axis is None and input.ndim > 1:
        sort_flattened(output, input, argsort, stable)
        return
    computed_axis = 0 if axis is None else normalize_axis_index(axis, input.ndim)
    if computed_axis == input.ndim - 1:
        sort_task(output, input, argsort, stable)
    else:
        sort_swapped(output, input, argsort, computed_axis, stable)
