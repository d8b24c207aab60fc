"""Every traversal scheme against the oracle's test of every primitive, where the comparison with the
reference's own BVH needs its library: rays at the million-triangle mesh, and directions with
components of exactly +0.0 and -0.0."""
import ctypes as C

import numpy as np
import pytest

import oraclelib as O
import rumi_b200
from rumi_b200 import _capi, scenes
from test_gpu_parity import _signed_zero_rays

pytestmark = pytest.mark.gpu
MODES = (0, 1, 2, 3, 4, 5)


def _scheme(gs, rays, mode, anyhit):
    t, prim = np.zeros(len(rays), np.float32), np.zeros(len(rays), np.int32)
    _capi.check(_capi.load().rumi_test_trace_scheme(
        gs.h, len(rays), rays.ctypes.data_as(C.c_void_p), int(anyhit), mode, t.ctypes.data_as(C.c_void_p),
        prim.ctypes.data_as(C.c_void_p)), "rumi_test_trace_scheme")
    return t, prim


def _camera_and_inner_rays(rng, n):
    o = np.concatenate([np.tile([[0.5, 0.5, -1.4]], (n, 1)), rng.uniform(0.05, 0.95, (n, 3))])
    d = np.concatenate([rng.uniform([0.2, 0.1, 0.2], [0.8, 0.6, 0.8], (n, 3)) - o[:n], rng.normal(size=(n, 3))])
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d, np.full((2 * n, 1), 3.4e38)], 1).astype(np.float32)


@pytest.mark.parametrize("levels,kind,n", [(9, "camera and inner", 150), (5, "signed zeros", 1024)])
def test_every_scheme_equals_a_test_of_every_primitive(levels, kind, n):
    sc = scenes.bvh_bound_pt(64, 64, 4, 10, levels=levels, seed=7)
    rng = np.random.default_rng(23)
    r7 = _signed_zero_rays(rng, n) if kind == "signed zeros" else _camera_and_inner_rays(rng, n)
    rays = np.zeros((len(r7), 8), np.float32)
    rays[:, :3], rays[:, 4:] = r7[:, :3], r7[:, 3:]
    oracle = O.OracleScene(sc)
    ot, op = oracle.trace(rays)
    assert (op >= 0).mean() > 0.5
    short = rays.copy()
    short[:, 7] = np.where(ot > 0, ot * 0.5, 0.5)
    oocc = oracle.trace(short, anyhit=True)[1]
    gs = rumi_b200.GpuScene(sc)
    try:
        for mode in MODES:
            t, prim = _scheme(gs, rays, mode, False)
            assert np.array_equal(t, ot) and np.array_equal(prim, op), mode
            assert np.array_equal(_scheme(gs, short, mode, True)[1], oocc), mode
        t, prim, _, _ = gs.trace(rays)
        assert np.array_equal(t, ot) and np.array_equal(prim, op)
        assert np.array_equal(gs.trace(short, anyhit=True)[1], oocc)
    finally:
        gs.close()
