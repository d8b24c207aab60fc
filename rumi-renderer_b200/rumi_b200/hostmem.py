"""Result arrays in page-locked memory.

A film copied to a fresh numpy array costs more in page faults and staging copies than the
frame's last kernels (3.7 MB: 0.5 ms).  ``empty`` hands out arrays over page-locked blocks that
go back to a pool when the last view of them is gone; the pool and what it has handed out are
bounded together, and beyond the bound (or without a device) the array is an ordinary one.

Making a block costs more than it saves once, so ``result``, which the frames use, makes one only
for a program that lets go of its results: each ordinary result that is gone pays for one block of
its size.  A program that keeps its films gets ordinary arrays: frames of 64x48 and 256x256 pixels
take 0.13 and 0.2 to 0.5 ms each (as fresh as the process's pages are), where a block made for each
film takes 0.51 and 0.99; 640x480 films take 0.44 to 1.9 ms, and 1.4 with blocks."""
from __future__ import annotations

import ctypes as C
import math
import os
import threading
import weakref

import numpy as np

from . import _capi

LIMIT = 256 << 20    # bytes of page-locked memory, handed out and pooled
SMALLEST = 1 << 16   # block sizes are powers of two from here


class _Pool:
    def __init__(self, limit: int = LIMIT):
        self.limit = limit
        self.total = 0
        self.free = {}
        self.gone = {}  # ordinary results of a block's size that are gone, not yet paid for a block
        # a finalizer can run inside any allocation of the thread that holds the lock
        self.lock = threading.RLock()

    def take(self, size: int):
        """Address of a block of `size` bytes (a power of two), or None."""
        with self.lock:
            blocks = self.free.get(size)
            if blocks:
                return blocks.pop()
            if self.total + size > self.limit:
                self._drop(self.total + size - self.limit)
            if self.total + size > self.limit:
                return None
            self.total += size
        p = C.c_void_p()
        if _capi.load().rumi_host_alloc(size, C.byref(p)) != 0:
            with self.lock:
                self.total -= size
            return None
        return p.value

    def _drop(self, need: int):
        """Gives pooled blocks of other sizes back, largest first."""
        for size in sorted(self.free, reverse=True):
            while need > 0 and self.free.get(size):
                _capi.load().rumi_host_free(C.c_void_p(self.free[size].pop()))
                self.total -= size
                need -= size

    def give(self, address: int, size: int):
        with self.lock:
            self.free.setdefault(size, []).append(address)
            if self.total > self.limit:
                self._drop(self.total - self.limit)

    def set_limit(self, limit: int):
        with self.lock:
            self.limit = limit
            self.gone.clear()
            self._drop(self.total - limit)

    def wanted(self, size: int) -> bool:
        """Whether the next result of this size takes a block."""
        with self.lock:
            if self.free.get(size):
                return True
            if self.gone.get(size, 0) == 0:
                return False
            self.gone[size] -= 1
            return True

    def let_go(self, size: int):
        with self.lock:
            self.gone[size] = self.gone.get(size, 0) + 1


_pool = _Pool()


def _after_fork():
    """In a forked child: another thread of the parent may have held the lock."""
    _pool.lock = threading.RLock()


os.register_at_fork(after_in_child=_after_fork)


def set_limit(limit: int):
    """Bounds the page-locked memory to `limit` bytes from now on (0: none, every array is an ordinary
    one).  Pooled blocks beyond the bound are given back at once, those in use when their last view is
    gone."""
    _pool.set_limit(int(limit))


def release():
    """Gives the pooled blocks back to the system; arrays in use keep theirs."""
    limit = _pool.limit
    _pool.set_limit(0)
    _pool.set_limit(limit)


def _block_size(need: int) -> int:
    return max(SMALLEST, 1 << (need - 1).bit_length())


def _in_block(shape, dtype, count: int, size: int) -> np.ndarray:
    address = _pool.take(size)
    if address is None:
        return np.empty(shape, dtype)
    block = (C.c_char * size).from_address(address)
    weakref.finalize(block, _pool.give, address, size).atexit = False
    return np.frombuffer(block, dtype, count).reshape(shape)


def empty(shape, dtype) -> np.ndarray:
    """An uninitialised C-contiguous array, page-locked when the pool has room."""
    dtype = np.dtype(dtype)
    count = math.prod(shape)
    need = count * dtype.itemsize
    if need == 0 or need > _pool.limit // 4:
        return np.empty(shape, dtype)
    return _in_block(shape, dtype, count, _block_size(need))


def result(shape, dtype) -> np.ndarray:
    """``empty`` where the program has let go of results of this size, else an ordinary array."""
    dtype = np.dtype(dtype)
    count = math.prod(shape)
    need = count * dtype.itemsize
    if need == 0 or need > _pool.limit // 4:
        return np.empty(shape, dtype)
    size = _block_size(need)
    if _pool.wanted(size):
        return _in_block(shape, dtype, count, size)
    array = np.empty(shape, dtype)  # its views refer to it
    weakref.finalize(array, _pool.let_go, size).atexit = False
    return array
