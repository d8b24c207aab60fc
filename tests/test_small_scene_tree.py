"""Scenes around the sizes where their tree is made in another way (64 primitives: one pass of the
builder; 256: the four-wide tree by one block), and of every kind of primitive: hits against a
test of every primitive, and what the build reports."""
import numpy as np
import pytest

import oraclelib as O
import rumi_b200
from rumi_b200 import scenes
from rumi_b200.scene import Dielectric, Emissive, Film, Matte, Model, PathTracer, Rect, Scene, Sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [1.0, 0.0])  # 0: all in one place, so that no split by position exists
@pytest.mark.parametrize("n_tri,n_rect,n_sph", [(0, 0, 0), (0, 1, 0), (0, 0, 3), (61, 2, 1), (62, 2, 1), (65, 0, 0), (120, 5, 4),
                                                (250, 3, 3), (250, 4, 3), (256, 0, 0), (258, 0, 0), (1022, 1, 1)])
def test_hits_equal_a_test_of_every_primitive(n_tri, n_rect, n_sph, spread):
    rng = np.random.Generator(np.random.PCG64(n_tri + 7))
    sc = Scene()
    if n_tri:
        t = rng.uniform(-1, 1, (n_tri, 1, 3)) * spread + rng.uniform(-0.2, 0.2, (n_tri, 3, 3))
        sc.add(Model(t.astype(np.float32)), Matte(1.0, scenes.WHITE))
    for k in range(n_rect):
        p = rng.uniform(-1, 1, 3)
        sc.add(Rect(p, (0.5, 0, 0), (0, 0, 0.4), 1), Emissive(1.0, (1.0, 1.0, 1.0)) if k % 2 else Matte(1.0, (0.5, 0.5, 0.5)))
    for _ in range(n_sph):
        sc.add(Sphere(rng.uniform(-1, 1, 3), 0.2), Dielectric(1.5, 1.0, (0.0, 0.0, 0.0)))
    sc.camera, sc.image, sc.tracer = scenes.cornell_camera(), Film(8, 8, 1), PathTracer(1)
    r = np.zeros((2000, 8), np.float32)
    r[:, 0:3] = rng.uniform(-1.5, 1.5, (2000, 3))
    d = rng.uniform(-1, 1, (2000, 3)) * max(spread, 0.2) - r[:, 0:3]
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 3.4e38
    oracle = O.OracleScene(sc)
    for _ in range(2):  # the second scene takes the memory of the first
        gs = rumi_b200.GpuScene(sc)
        try:
            info = gs.bvh_info()
            n = n_tri + n_rect + n_sph
            assert info["large_levels"] == 0 if n <= 256 else info["large_levels"] > 0
            assert info["small_tasks"] == (1 if 0 < n <= 256 else info["small_tasks"])
            t, prim, _, _ = gs.trace(r)
            ot, op = oracle.trace(r)
            assert np.array_equal(t, ot) and np.array_equal(prim, op)
            _, occ, _, _ = gs.trace(r, anyhit=True)
            assert np.array_equal(occ, oracle.trace(r, anyhit=True)[1])
        finally:
            gs.close()
