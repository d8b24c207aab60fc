"""Page-locked results in a process that forks: the child keeps its own copy of a film, whatever the
parent does with the block afterwards, and the parent's frames still land in its own."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ask(rd, wr, word):
    os.write(wr, word)
    return os.read(rd, 1)


@pytest.mark.parametrize("size", [(64, 48), (700, 500)])
def test_a_forked_child_has_its_own_film(size):
    import rumi_b200
    from rumi_b200 import hostmem, scenes
    gs = rumi_b200.GpuScene(scenes.cornell_pt(size[0], size[1], 1, 2))
    try:
        want = np.array(gs.render(seed=2)[0])
        film = hostmem.empty((size[1], size[0], 3), np.float32)
        address, film[:] = film.ctypes.data, 1.0
        down_r, down_w = os.pipe()
        up_r, up_w = os.pipe()
        pid = os.fork()
        if pid == 0:  # no CUDA call here
            try:
                for _ in range(2):
                    os.read(down_r, 1)
                    os.write(up_w, b"y" if (film == 1.0).all() else b"n")
                film[:] = 3.0
                os.read(down_r, 1)
            finally:
                os._exit(0)
        film[:] = 2.0
        first = _ask(up_r, down_w, b"a")
        kept = film[:1, :1]  # the block stays out; then it goes back and the next film takes it
        assert (kept == 2.0).all()
        del kept, film
        got = gs.render(seed=2)[0]
        second = _ask(up_r, down_w, b"b")
        os.write(down_w, b"c")
        os.waitpid(pid, 0)
        for fd in (down_r, down_w, up_r, up_w):
            os.close(fd)
        assert first == b"y" and second == b"y"
        assert np.array_equal(got, want)
        assert got.ctypes.data == address  # (else the recycled block was not looked at)
    finally:
        gs.close()
