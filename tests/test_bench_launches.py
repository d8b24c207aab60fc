"""bench.py's count of the library's launches: where a wave's rays are ordered (pt.cu, sort_wave)."""
import importlib.util
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench_launches", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


@pytest.mark.parametrize("paths,triangles,mode,expect", [
    (1 << 22, 65546, 0, True),        # a 256x256, 64 spp frame of the inverse-rendering mesh
    (1 << 22, 256, 0, False),         # its 256-triangle form
    ((1 << 22) - 1, 65546, 0, False), (1 << 25, 1048586, 4, True), (1 << 25, 1048586, 1, False)])
def test_when_waves_are_ordered(bench, paths, triangles, mode, expect):
    assert bench.ordered(paths, triangles, mode) is expect
    assert bench.wave_launches(8, bench.ordered(paths, triangles, mode)) == (40 if expect else 26)


def test_the_line_is_the_librarys(bench):
    src = open(os.path.join(ROOT, "rumi-renderer_b200", "csrc", "pt.cu")).read()
    assert 1 << int(re.search(r"#define RUMI_SORT_PATHS \(1 << (\d+)\)", src).group(1)) == bench.ORDERED_PATHS
