"""Results of frames (rumi_b200.hostmem.result), over a fake allocator: page-locked blocks are made for a
program that lets go of its results, and not for one that keeps them."""
import gc

import numpy as np
import pytest

from rumi_b200 import hostmem
from test_hostmem import lib  # noqa: F401


@pytest.mark.parametrize("shape", [(1,), (16, 16, 3), (150, 100, 3)])
def test_kept_results_are_ordinary(lib, shape):  # noqa: F811
    held = [hostmem.result(shape, np.float32) for _ in range(12)]
    assert len(lib.live) == 0 and len({h.ctypes.data for h in held}) == 12
    for k, h in enumerate(held):
        h[:] = k
    assert all((h == k).all() and h.shape == shape and h.flags.writeable for k, h in enumerate(held))


def test_dropped_results_move_to_blocks(lib):  # noqa: F811
    seen = []
    for _ in range(12):  # as a loop of frames: the last film lives until the next one is there
        film = hostmem.result((50, 40, 3), np.float32)
        seen.append(film.ctypes.data)
        gc.collect()
    assert len(lib.live) == 2 and set(seen[-6:]) <= set(lib.live)


def test_every_second_result_kept(lib):  # noqa: F811
    held = []
    for _ in range(20):
        held.append(hostmem.result((50, 40, 3), np.float32))
        hostmem.result((50, 40, 3), np.float32)
        gc.collect()
    # each block made was paid for by a result that is gone
    assert len(lib.live) <= 20 and len({h.ctypes.data for h in held}) == 20


def test_a_view_keeps_an_ordinary_result(lib):  # noqa: F811
    a = hostmem.result((10, 10), np.float32)
    a[:] = 5.0
    view = a[3:, ::2]
    del a
    gc.collect()
    assert hostmem._pool.gone == {} and (view == 5.0).all()
    del view
    gc.collect()
    assert sum(hostmem._pool.gone.values()) == 1


def test_blocks_are_given_back(lib):  # noqa: F811
    a, b = hostmem.empty((16384,), np.float32), hostmem.empty((16384,), np.float32)
    b[:] = 2.0
    del a
    gc.collect()
    assert len(lib.live) == 2
    hostmem.release()
    assert len(lib.live) == 1 and (b == 2.0).all()
    c = hostmem.empty((16384,), np.float32)  # the pool still works
    assert c.ctypes.data in lib.live
    hostmem.set_limit(0)
    assert len(lib.live) == 2 and hostmem.empty((16384,), np.float32).ctypes.data not in lib.live
    del b, c
    gc.collect()
    assert len(lib.live) == 0 and hostmem._pool.total == 0
    for _ in range(6):
        hostmem.result((16384,), np.float32)
    assert len(lib.live) == 0


@pytest.mark.gpu
def test_kept_films_lock_no_pages(monkeypatch):
    import rumi_b200
    from rumi_b200 import scenes
    monkeypatch.setattr(hostmem, "_pool", hostmem._Pool())
    gs = rumi_b200.GpuScene(scenes.cornell_pt(96, 80, 1, 2))
    try:
        films = [gs.render(seed=3)[0] for _ in range(6)]
        assert hostmem._pool.total == 0
        assert all(np.array_equal(films[0], f) for f in films)
        films = None
        for _ in range(6):
            film = gs.render(seed=3)[0]
        assert hostmem._pool.total > 0 and film.any()
    finally:
        gs.close()
