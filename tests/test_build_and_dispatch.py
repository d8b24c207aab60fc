"""The tree builder at the edges of its phases, and the frames and queries that take a path of
their own by size: all exact, against the oracle's test of every primitive or the general path."""
import numpy as np
import pytest

import oraclelib as O
import rumi_b200
from rumi_b200 import scenes
from rumi_b200.scene import (Dielectric, Emissive, Film, Matte, Model, PathTracer, RayTracer, Rect, Scene, Sphere,
                             Specular)

pytestmark = pytest.mark.gpu


def _tris(shape, n):
    rng = np.random.Generator(np.random.PCG64(n))
    c = rng.uniform(-1, 1, (n, 1, 3))
    e = rng.uniform(-0.1, 0.1, (n, 3, 3))
    if shape == "clusters":   # halving distances and sizes: one side of every split stays nearly empty
        k = 0.5 ** (np.arange(n) % 40)[:, None, None]
        c, e = c * k, e * k
    elif shape == "one":      # equal triangles: no split by position exists
        c, e = c * 0.0, np.broadcast_to(e[:1], e.shape)
    elif shape == "line":     # centroids on a line, flat boxes
        c = c * np.array([1.0, 0.0, 0.0])
        e = e * np.array([1.0, 1.0, 0.0])
    elif shape == "pairs":    # two places
        c = np.where(np.arange(n)[:, None, None] % 2, 0.5, -0.5) * np.ones((n, 1, 3))
    return (c + e).astype(np.float32)


@pytest.mark.parametrize("shape,n", [("even", k) for k in (1, 2, 15, 17, 64, 65, 255, 257, 1023, 1025, 4099)] +
                         [(s, k) for s in ("clusters", "one", "line", "pairs") for k in (65, 1500)])
def test_hits_equal_a_test_of_every_triangle(shape, n):
    sc = Scene()
    sc.add(Model(_tris(shape, n)), Matte(1.0, scenes.WHITE))
    sc.camera, sc.image, sc.tracer = scenes.cornell_camera(), Film(8, 8, 1), PathTracer(1)
    rng = np.random.Generator(np.random.PCG64(7))
    r = np.zeros((2000, 8), np.float32)
    r[:, 0:3] = rng.uniform(-1.5, 1.5, (2000, 3))
    to = rng.uniform(-0.6, 0.6, (2000, 3)) * 0.5 ** rng.integers(0, 12, (2000, 1))
    d = to - r[:, 0:3]
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 3.4e38
    gs = rumi_b200.GpuScene(sc)
    try:
        t, prim, _, _ = gs.trace(r)
        ot, op = O.OracleScene(sc).trace(r)
        assert np.array_equal(t, ot) and np.array_equal(prim, op)
        _, occ, _, _ = gs.trace(r, anyhit=True)
        _, oocc = O.OracleScene(sc).trace(r, anyhit=True)
        assert np.array_equal(occ, oocc)
    finally:
        gs.close()


# triangles beside a light, a floor, a mirror and a glass sphere: one node of few records (tested in
# step) up to several nodes (walked)
@pytest.mark.parametrize("whitted", [False, True])
@pytest.mark.parametrize("n", [0, 1, 2, 3, 7, 12, 13, 14, 15, 16, 17, 40])
def test_few_primitives_render_as_the_walk_does(n, whitted):
    sc = Scene()
    sc.add(Rect((-1, -1, 3), (2, 0, 0), (0, 0, -2), 1), Matte(1.0, (0.6, 0.7, 0.5)))
    sc.add(Rect((-0.4, 0.99, 2.4), (0.8, 0, 0), (0, 0, -0.8), 1), Emissive(6.0, (1.0, 0.9, 0.8)))
    sc.add(Sphere((0.3, -0.5, 1.8), 0.35), Dielectric(1.5, 1.0, (0.1, 0.2, 0.1)))
    if n:
        tris = _tris("even", n) * 0.7 + np.array([0, 0, 2], np.float32)
        sc.add(Model(tris.astype(np.float32)), Specular(0.9, (0.9, 0.9, 0.9)) if n % 2 else Matte(0.8, scenes.WHITE))
    sc.camera, sc.image = scenes.cornell_camera(), Film(45, 37, 9)
    sc.tracer = RayTracer(5) if whitted else PathTracer(6)
    gs = rumi_b200.GpuScene(sc)
    try:
        want, sw = gs.render(seed=5, trace_mode=2)
        for mode in (0, 4):
            got, sg = gs.render(seed=5, trace_mode=mode)
            assert np.array_equal(np.asarray(want).view(np.uint32), np.asarray(got).view(np.uint32))
            assert sg["rays_extend"] == sw["rays_extend"] and sg["rays_shadow"] == sw["rays_shadow"]
    finally:
        gs.close()


# host rays up to 8192 go through the scene's page-locked staging, larger sets and device rays not
@pytest.mark.parametrize("anyhit", [False, True])
@pytest.mark.parametrize("n", [1, 33, 8191, 8192, 8193])
def test_staged_queries_equal_device_queries(n, anyhit):
    import torch
    sc = scenes.bvh_bound_pt(16, 16, 1, 1, levels=4, seed=7)
    rng = np.random.Generator(np.random.PCG64(n))
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(0.0, 1.0, (n, 3))
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 3.4e38
    gs = rumi_b200.GpuScene(sc)
    try:
        t, prim, nodes, prims = gs.trace(r, anyhit=anyhit)
        dr = torch.from_numpy(r).cuda()
        dt, dp = torch.zeros(n, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        dn, dpr = gs.trace_device(n, dr.data_ptr(), dt.data_ptr(), dp.data_ptr(), anyhit=anyhit)
        assert np.array_equal(t, dt.cpu().numpy()) and np.array_equal(prim, dp.cpu().numpy())
        assert nodes > 0 and prims > 0 and dn > 0 and dpr > 0
        if n > 1:
            t2, prim2, _, _ = gs.trace(r[:n // 2], anyhit=anyhit)  # a smaller set after a larger one
            assert np.array_equal(t2, t[:n // 2]) and np.array_equal(prim2, prim[:n // 2])
    finally:
        gs.close()
