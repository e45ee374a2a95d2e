"""Process-level state of the host layer: which GPU this process drives, how many processes
take part (one per GPU), and the scratch memory handed to the kernels.

Plays the role the Legate runtime plays for the reference's SORT task: it owns device memory
(through torch's caching allocator, the stand-in for Legate's framebuffer pool,
``src/cupynumeric/mapper.cc:635-643``), the stream, and the communicator
(``cupynumeric/_thunk/_sort.py:87-92``).
"""
from __future__ import annotations

import threading
from collections import OrderedDict

import torch
import torch.distributed as dist

from . import _lib


class Runtime:
    KEPT = 8       # workspaces kept per process, least recently used first out
    STICKY = 64    # status words kept per process

    def __init__(self) -> None:
        # (device, stream, thread) -> the workspace and the status word at its head
        self._ws: OrderedDict[tuple[int, int, int], tuple[torch.Tensor, torch.Tensor]] = OrderedDict()
        self._sticky: dict[tuple[int, int], torch.Tensor] = {}   # (device, stream) -> status of its sorts so far
        self._failed: dict[int, int] = {}                        # device -> status read but not raised yet
        self._lock = threading.Lock()
        self._comm = None

    # --- topology -------------------------------------------------------------------------
    @property
    def num_procs(self) -> int:
        return dist.get_world_size() if dist.is_available() and dist.is_initialized() else 1

    @property
    def rank(self) -> int:
        return dist.get_rank() if dist.is_available() and dist.is_initialized() else 0

    @property
    def num_gpus(self) -> int:
        return self.num_procs if torch.cuda.is_available() else 0

    @property
    def device(self) -> torch.device:
        if not torch.cuda.is_available():
            raise RuntimeError("cupynumeric_b200 needs a CUDA device: the sort kernels have no CPU path")
        return torch.device("cuda", torch.cuda.current_device())

    def stream_handle(self) -> int:
        return torch.cuda.current_stream().cuda_stream

    # --- scratch memory -------------------------------------------------------------------
    def _scratch(self, nbytes: int) -> torch.Tensor:
        return torch.empty(nbytes, dtype=torch.uint8, device=self.device)

    def workspace(self, nbytes: int) -> torch.Tensor:
        """A 256-byte aligned device buffer of at least ``nbytes``, reused by the calls of one thread on
        one stream of one device.  These are ordered.  Sorts of two streams run at the same time, and two
        threads enqueue the kernels of their sorts in any order even on one stream; the kernels of a sort take
        their store addresses from its workspace, so such sorts never share one.  A buffer that goes returns to the
        allocator, which hands it out again on the stream it was made on."""
        key = (torch.cuda.current_device(), self.stream_handle(), threading.get_ident())
        with self._lock:
            cur = self._ws.get(key)
            if cur is not None and cur[0].numel() >= nbytes:
                self._ws.move_to_end(key)
                return cur[0]
            self._ws.pop(key, None)
            cur = None
            while len(self._ws) >= self.KEPT:
                self._ws.popitem(last=False)
            size = max(int(nbytes), 1 << 16)
            try:
                ws = self._scratch(size)
            except torch.cuda.OutOfMemoryError:
                self._ws.clear()   # what other streams and threads keep for their next call
                ws = self._scratch(size)
            assert ws.data_ptr() % 256 == 0
            self._ws[key] = (ws, ws[:4].view(torch.int32))
            return ws

    def release_workspace(self) -> None:
        with self._lock:
            self._ws.clear()

    # --- device-side status of the sorts enqueued so far ------------------------------------
    def note_sort(self, ws: torch.Tensor) -> None:
        """Folds the status word at the head of a workspace (0, or the code a kernel left when a
        bounded wait ran out) into a word per stream that survives the workspace's reuse.  Stream
        ordered, no synchronisation."""
        dev, stream = torch.cuda.current_device(), self.stream_handle()
        with self._lock:
            acc = self._sticky.get((dev, stream))
            if acc is None:
                if len(self._sticky) >= self.STICKY:
                    self._collect()
                acc = self._sticky[(dev, stream)] = torch.zeros(1, dtype=torch.int32, device=self.device)
            own = self._ws.get((dev, stream, threading.get_ident()))
        torch.maximum(acc, own[1] if own is not None and own[0] is ws else ws[:4].view(torch.int32), out=acc)

    def _collect(self) -> None:
        """Reads the status words of all streams and lets go of them."""
        for (dev, _), acc in self._sticky.items():
            torch.cuda.synchronize(dev)
            self._failed[dev] = max(self._failed.get(dev, 0), int(acc.item()))
        self._sticky.clear()

    def raise_pending(self) -> None:
        """Called where a result reaches the host: raises if any sort of this device since the last call reported
        a device-side failure (role of CUPYNUMERIC_CHECK_CUDA_STREAM in the reference's task
        bodies, ``src/cupynumeric/cuda_help.h:291-302``)."""
        if not torch.cuda.is_available():
            return
        dev = torch.cuda.current_device()
        with self._lock:
            words = [acc for (d, _), acc in self._sticky.items() if d == dev]
            status = self._failed.pop(dev, 0)
        for acc in words:
            own = int(acc.item())
            if own != 0:
                acc.zero_()
            status = max(status, own)
        if status != 0:
            raise _lib.B2SError(status, "a sort kernel")


runtime = Runtime()
