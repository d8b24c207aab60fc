"""The pool behind result arrays (rumi_b200.hostmem), over a fake allocator: blocks are reused only
when the last view is gone, and what is handed out and pooled stays within the bound."""
import ctypes as C
import gc
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "rumi-renderer_b200"))

from rumi_b200 import _capi, hostmem  # noqa: E402


class FakeLib:
    def __init__(self):
        self.live = {}

    def rumi_host_alloc(self, size, out):
        block = (C.c_char * size)()
        self.live[C.addressof(block)] = block
        out._obj.value = C.addressof(block)
        return 0

    def rumi_host_free(self, p):
        del self.live[p.value]
        return 0


@pytest.fixture
def lib(monkeypatch):
    fake = FakeLib()
    monkeypatch.setattr(_capi, "load", lambda *a: fake)
    monkeypatch.setattr(hostmem, "_pool", hostmem._Pool(1 << 20))
    return fake


def test_a_block_returns_with_its_last_view(lib):
    a = hostmem.empty((10, 10, 3), np.float32)
    a[:] = 3.0
    address, view = a.ctypes.data, a[2:, ::2]
    del a
    gc.collect()
    b = hostmem.empty((300,), np.float32)
    assert b.ctypes.data != address and (view == 3.0).all()
    del view
    gc.collect()
    c = hostmem.empty((5,), np.uint8)
    assert c.ctypes.data == address and c.flags.writeable and len(lib.live) == 2


@pytest.mark.parametrize("shape", [(0,), (1,), (16384,), (16385,), (40000,), (100000,)])
def test_memory_stays_within_the_bound(lib, shape):
    held = [hostmem.empty(shape, np.float32) for _ in range(40)]
    assert all(h.shape == shape and h.dtype == np.float32 for h in held)
    assert sum(C.sizeof(b) for b in lib.live.values()) <= 1 << 20
    held = None
    gc.collect()
    held = [hostmem.empty((1 << 16,), np.uint8) for _ in range(17)]  # other sizes make room
    assert sum(C.sizeof(b) for b in lib.live.values()) <= 1 << 20 and len(lib.live) == 16


def test_without_memory_to_lock_the_array_is_ordinary(lib):
    lib.rumi_host_alloc = lambda size, out: 3
    a = hostmem.empty((7, 5), np.float32)
    assert a.shape == (7, 5) and hostmem._pool.total == 0
