"""Result arrays in pinned host memory.

The device copies straight into pinned memory; into ordinary memory the
runtime copies through a buffer of its own, one array at a time, while the
caller waits, and a large new array's pages fault in on the way. `empty` gives
numpy arrays on blocks of a pool: a block returns when its last array (or view
of it) is gone, so a program that drops each frame's image reuses one block.
The pool holds at most LIMIT bytes, in use or not; beyond that, and for small
arrays, `empty` is numpy's own. It gives its memory back when the last executor
and batch are disposed.

A new block costs its pages (host_memory.cu): a 1080p image into a new block
3.3 ms, into ordinary memory 4.0, into a block used before 1.5; of results below
a megabyte some pay 0.3 to 1 ms for a slab that others are cut from. So new
blocks are for programs whose results come back: a size has FRESH new blocks to
begin with, and earns one more with each result of that size that is dropped,
whichever memory it was in, at most FRESH more than it has. A program that keeps
its results gets ordinary memory after that: the pool's room is for those that
return.

A block is handed out again as soon as its arrays are gone, so whoever queues a
copy into one keeps the array until that copy is done.
"""
from __future__ import annotations

import ctypes as C
import operator
import threading
import weakref
from typing import Any, Dict, List, Optional

import numpy as np

from ._lib import McrtError, call

SMALL = 1 << 16
LIMIT = 256 << 20
FRESH = 2


class _Pool:
    def __init__(self) -> None:
        self._lock = threading.RLock()  # give() may run inside take(): a collection can free arrays there
        self._free: Dict[int, List[int]] = {}
        self._held = 0  # bytes of all blocks, in use or free
        self._blocks: Dict[int, int] = {}  # blocks of each size, in use or free
        self._fresh: Dict[int, int] = {}  # new blocks each size may still have
        self.users = 0  # executors and batches
        self._closed = False  # the last of them is gone

    def attach(self) -> None:
        """An executor or a batch begins to ask for results."""
        with self._lock:
            self.users += 1
            self._closed = False

    def detach(self) -> None:
        """It is disposed: with the last one the free blocks go back, and those in use as they are dropped."""
        with self._lock:
            self.users -= 1
            if self.users > 0:
                return
            self._closed = True
            gone = [(size, p) for size, free in self._free.items() for p in free]
            self._free.clear()
            self._fresh.clear()
            for size, _ in gone:
                self._held -= size
                self._blocks[size] -= 1
        for _, p in gone:
            call("mcrt_host_free", C.c_void_p(p))

    @staticmethod
    def block_size(nbytes: int) -> int:
        """The size class of nbytes: quarters of powers of two."""
        step = 1 << max(12, nbytes.bit_length() - 3)
        return -(-nbytes // step) * step

    def take(self, size: int, device: Optional[int] = None) -> int:
        """Address of a block of `size` bytes, or 0 when the limit leaves no room or too few were dropped.
        A new one is allocated from `device`; any device may copy into it."""
        with self._lock:
            blocks = self._free.get(size)
            if blocks:
                return blocks.pop()
            if self._fresh.setdefault(size, FRESH) <= 0:
                return 0
            drop = []
            for other in sorted(self._free, reverse=True):  # make room from other sizes' free blocks
                while self._held + size > LIMIT and self._free[other]:
                    drop.append(self._free[other].pop())
                    self._held -= other
                    self._blocks[other] -= 1
            if self._held + size > LIMIT:
                size = 0
            else:
                self._held += size
                self._fresh[size] -= 1
                self._blocks[size] = self._blocks.get(size, 0) + 1
        for p in drop:
            call("mcrt_host_free", C.c_void_p(p))
        if size == 0:
            return 0
        p = C.c_void_p()
        try:
            if device is None:
                call("mcrt_host_alloc", size, C.byref(p))
            else:
                call("mcrt_host_alloc_on", int(device), size, C.byref(p))
        except McrtError:
            with self._lock:
                self._held -= size
                self._blocks[size] -= 1
            return 0
        return int(p.value or 0)

    def give(self, address: int, size: int) -> None:
        with self._lock:
            if not self._closed:
                self._free.setdefault(size, []).append(address)
                self.dropped(size)
                return
            self._held -= size
            self._blocks[size] -= 1
        call("mcrt_host_free", C.c_void_p(address))

    def dropped(self, size: int) -> None:
        with self._lock:
            self._fresh[size] = min(self._fresh.get(size, FRESH) + 1, FRESH + self._blocks.get(size, 0))

    def empty(self, count: int, dtype: Any, device: Optional[int] = None) -> np.ndarray:
        count, dtype = operator.index(count), np.dtype(dtype)
        nbytes = count * dtype.itemsize
        if nbytes < SMALL:
            return np.empty(count, dtype)
        size = self.block_size(nbytes)
        if size > LIMIT:
            return np.empty(count, dtype)
        address = self.take(size, device)
        if not address:
            plain = np.empty(count, dtype)
            weakref.finalize(plain, self.dropped, size).atexit = False
            return plain
        block = (C.c_uint8 * size).from_address(address)
        # At interpreter exit the driver takes the memory back with the process.
        weakref.finalize(block, self.give, address, size).atexit = False
        return np.frombuffer(block, dtype, count)


_pool = _Pool()


def attach() -> None:
    """Before an executor's or a batch's first result; detach() once it is disposed."""
    _pool.attach()


def detach() -> None:
    _pool.detach()


def empty(count: int, dtype: Any, device: Optional[int] = None) -> np.ndarray:
    """An uninitialised one-dimensional array, in pinned memory where that is worth it, for results of `device`."""
    return _pool.empty(count, dtype, device)


def zeros(count: int, dtype: Any, device: Optional[int] = None) -> np.ndarray:
    a = _pool.empty(count, dtype, device)
    a.fill(0)
    return a
