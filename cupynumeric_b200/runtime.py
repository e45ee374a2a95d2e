"""Process-level state of the host layer: which GPU this process drives, how many processes
take part (one per GPU), and the scratch memory handed to the kernels.

Plays the role the Legate runtime plays for the reference's SORT task: it owns device memory
(through torch's caching allocator, the stand-in for Legate's framebuffer pool,
``src/cupynumeric/mapper.cc:635-643``), the stream, and the communicator
(``cupynumeric/_thunk/_sort.py:87-92``).
"""
from __future__ import annotations

import threading

import torch
import torch.distributed as dist

from . import _lib


class Scratch:
    """What the calls of one thread on one stream sort with: a workspace, and the word that keeps the status of its sorts."""

    __slots__ = ("ws", "ptr", "nbytes", "status", "failed", "used")

    def __init__(self, ws: torch.Tensor, failed: torch.Tensor) -> None:
        self.ws, self.failed, self.used = ws, failed, 0
        self.ptr, self.nbytes, self.status = ws.data_ptr(), ws.numel(), ws[:4].view(torch.int32)


class Runtime:
    KEPT = 8       # workspaces kept per process, least recently used first out,
    KEPT_BYTES = 16 << 30   # and what the others may hold when one is made
    STICKY = 64    # status words kept per process

    def __init__(self) -> None:
        # by (device, stream, thread)
        self._kept: dict[tuple[int, int, int], Scratch] = {}
        self._sticky: dict[tuple[int, int, int], torch.Tensor] = {}   # status of the sorts so far
        self._failed: dict[int, int] = {}                             # device -> status read but not raised yet
        self._lock = threading.Lock()
        self._calls = 0
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
    def _bytes(self, nbytes: int) -> torch.Tensor:
        return torch.empty(nbytes, dtype=torch.uint8, device=self.device)

    def scratch(self, nbytes: int, device: int, stream: int) -> Scratch:
        """A workspace of at least ``nbytes``, 256-byte aligned, for a call on this stream, the current one of
        the current device.  It is reused by the calls of one thread on one stream: these are ordered.  Sorts of two streams
        run at the same time, and two threads enqueue the kernels of their sorts in any order even on one
        stream; the kernels of a sort take their store addresses from its workspace, so such sorts never share one.  A buffer
        that goes returns to the allocator, which hands it out again on the stream it was made on."""
        key = (device, stream, threading.get_ident())
        self._calls += 1
        own = self._kept.get(key)
        if own is None or own.nbytes < nbytes:
            own = self._renew(key, max(int(nbytes), 1 << 16))
        own.used = self._calls
        return own

    def _renew(self, key: tuple[int, int, int], nbytes: int) -> Scratch:
        with self._lock:
            self._kept.pop(key, None)
            while len(self._kept) >= self.KEPT or sum(k.nbytes for k in self._kept.values()) > self.KEPT_BYTES:
                del self._kept[min(self._kept, key=lambda k: self._kept[k].used)]
            try:
                ws = self._bytes(nbytes)
            except torch.cuda.OutOfMemoryError:
                self._kept.clear()   # what other streams and threads keep for their next call
                ws = self._bytes(nbytes)
            assert ws.data_ptr() % 256 == 0
            if key not in self._sticky:
                if len(self._sticky) >= self.STICKY:
                    self._collect()
                self._sticky[key] = torch.zeros(1, dtype=torch.int32, device=self.device)
            own = self._kept[key] = Scratch(ws, self._sticky[key])
            return own

    def workspace(self, nbytes: int) -> torch.Tensor:
        """The workspace of a call on the current stream."""
        return self.scratch(nbytes, torch.cuda.current_device(), self.stream_handle()).ws

    def release_workspace(self) -> None:
        with self._lock:
            self._kept.clear()

    # --- device-side status of the sorts enqueued so far ------------------------------------
    def note_sort(self, own: Scratch) -> None:
        """Folds the status word at the head of a workspace (0, or the code a kernel left when a
        bounded wait ran out) into a word that survives the workspace's reuse.  Stream
        ordered, no synchronisation."""
        torch.maximum(own.failed, own.status, out=own.failed)

    def _collect(self) -> None:
        """Reads the status words whose workspaces are gone and lets go of them."""
        for key in [k for k in self._sticky if k not in self._kept]:
            torch.cuda.synchronize(key[0])
            self._failed[key[0]] = max(self._failed.get(key[0], 0), int(self._sticky.pop(key).item()))

    def raise_pending(self) -> None:
        """Called where a result reaches the host: raises if any sort of this device since the last call reported
        a device-side failure (role of CUPYNUMERIC_CHECK_CUDA_STREAM in the reference's task
        bodies, ``src/cupynumeric/cuda_help.h:291-302``)."""
        if not torch.cuda.is_available():
            return
        dev = torch.cuda.current_device()
        with self._lock:
            words = [word for key, word in self._sticky.items() if key[0] == dev]
            status = self._failed.pop(dev, 0)
        for word in words:
            own = int(word.item())
            if own != 0:
                word.zero_()
            status = max(status, own)
        if status != 0:
            raise _lib.B2SError(status, "a sort kernel")


runtime = Runtime()
