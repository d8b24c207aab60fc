"""Memory that a call can do without (the order of a large wave's rays, the staging of small
queries): when it cannot be had, what is held stays, and the same is not asked for on every call."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def block(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ is missing")
    so = str(tmp_path_factory.mktemp("block") / "libblock.so")
    subprocess.run([gxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-o", so,
                    os.path.join(HERE, "host_build", "optional_block_host.cpp")], check=True)
    lib = C.CDLL(so)
    lib.block_reset.argtypes = lib.block_grow.argtypes = [C.c_size_t]
    lib.block_bytes.restype = C.c_size_t
    return lib


def test_a_refusal_leaves_the_block_and_is_remembered(block):
    block.block_reset(1000)
    assert block.block_grow(600) == 1 and block.block_bytes() == 600
    for _ in range(5):  # frames that would like more
        assert block.block_grow(1200) == 0 and block.block_grow(1500) == 0
    assert block.block_bytes() == 600 and block.block_asked() == 2 and block.block_released() == 0
    assert block.block_grow(500) == 1 and block.block_asked() == 2
    assert block.block_grow(900) == 1 and block.block_bytes() == 900 and block.block_released() == 1
    assert block.block_grow(1100) == 0 and block.block_asked() == 4  # less than what was refused: asked for once
    assert block.block_grow(1100) == 0 and block.block_asked() == 4


def test_memory_that_cannot_be_had_at_all(block):
    """A query's staging: refused once, then the query goes the other way without asking again."""
    block.block_reset(0)
    assert [block.block_grow(328448) for _ in range(4)] == [0] * 4
    assert block.block_asked() == 1 and block.block_bytes() == 0
