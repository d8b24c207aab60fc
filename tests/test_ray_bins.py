"""The bins that order a large wave's rays, where the rays start close together: their counters lie
apart, so that the additions to them do not queue up at a few memory lines."""
import ctypes as C

import numpy as np
import pytest

from test_ray_order import host  # noqa: F401


@pytest.mark.parametrize("scale", [1.0, 40.0, 1e4])
def test_counters_of_one_place_lie_apart(host, scale):  # noqa: F811
    rng = np.random.Generator(np.random.PCG64(3))
    n = 20000
    od = np.zeros((n, 6), np.float32)
    od[:, :3] = rng.uniform(0.01, 0.02, (n, 3))
    d = rng.normal(size=(n, 3))
    od[:, 3:] = d / np.linalg.norm(d, axis=1, keepdims=True)
    bins = np.empty(n, np.int32)
    box = np.array([-scale] * 3 + [scale] * 3, np.float32)
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    total = host.rumi_host_sort_bins(n, p(box, C.c_float), p(od, C.c_float), p(bins, C.c_int))
    assert bins.min() >= 0 and bins.max() < total
    # every direction cell that the rays point to (several hundred) in its own half line or nearly
    assert len(np.unique(bins // 32)) >= 0.4 * len(np.unique(bins)) >= 100


def test_every_cell_has_a_bin_of_its_own(host):  # noqa: F811
    g = (np.arange(16, dtype=np.float32) + 0.5) / 16
    o = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    h = (np.arange(8, dtype=np.float32) + 0.5) / 4 - 1
    d = np.stack(np.meshgrid(h, h, h, indexing="ij"), -1).reshape(-1, 3)
    od = np.concatenate([np.repeat(o, len(d), 0), np.tile(d, (len(o), 1))], 1).astype(np.float32)
    bins = np.empty(len(od), np.int32)
    box = np.array([0, 0, 0, 1, 1, 1], np.float32)
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    total = host.rumi_host_sort_bins(len(od), p(box, C.c_float), p(od, C.c_float), p(bins, C.c_int))
    assert total == len(od) and np.array_equal(np.sort(bins), np.arange(total))
