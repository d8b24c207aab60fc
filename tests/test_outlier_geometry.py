"""Scenes with a primitive far larger than the rest (a sky sphere, a ground plane) under the
default walk: the rest costs what it costs alone.  On the CPU the walk built for the host over a
tree packed by the library's packing, on the GPU the library's own tree."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def _soup(n, seed=3):
    rng = np.random.Generator(np.random.PCG64(seed))
    c = rng.uniform(-1, 1, (n, 1, 3))
    return (c + rng.uniform(-0.1, 0.1, (n, 3, 3))).astype(np.float32)


def _rays(n, seed=5):
    rng = np.random.Generator(np.random.PCG64(seed))
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(-1.5, 1.5, (n, 3))
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 3.4e38
    return r


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    gxx = shutil.which("g++")
    inc = next((os.path.join(r, "include") for r in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                if r and os.path.isfile(os.path.join(r, "include", "cuda_runtime.h"))), None)
    if not gxx or not inc:
        pytest.skip("g++ or the CUDA headers are missing")
    so = str(tmp_path_factory.mktemp("outlier") / "liboutlier.so")
    subprocess.run([gxx, "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-I", inc, "-o", so,
                    os.path.join(HERE, "host_build", "outlier_host.cpp")], check=True)
    return C.CDLL(so)


def _prims(tri, sph):
    n = len(tri) + len(sph)
    prims = np.zeros((n, 3, 4), np.float32)
    ids = prims.view(np.int32)
    nt = len(tri)
    prims[:nt, 0, :3], prims[:nt, 1, :3], prims[:nt, 2, :3] = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    prims[nt:, 0, :3], prims[nt:, 1, 0] = sph[:, :3], sph[:, 3]
    ids[:, 0, 3] = np.arange(n)
    ids[nt:, 1, 3] = 2
    box = np.concatenate([np.concatenate([tri.min(1), tri.max(1)], 1),
                          np.concatenate([sph[:, :3] - sph[:, 3:], sph[:, :3] + sph[:, 3:]], 1)]).astype(np.float32)
    return prims, box


def _f(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))


# 600 triangles in a sphere that every ray may test: of radius 2, and of a far larger one (the same
# random tree over the same order)
@pytest.mark.parametrize("radius", [1e2, 1e4, 1e6, 1e9, 1e15])
def test_a_far_sphere_leaves_the_other_boxes_tight(host, radius):
    rays = _rays(2000)
    counts = []
    for r in (2.0, radius):
        prims, box = _prims(_soup(600), np.array([[0, 0, 0, r]], np.float32))
        counts.append(host.rumi_host_walk_tests(_f(prims), _f(box), len(prims), 11, _f(rays), len(rays)))
    assert counts[1] < 1.5 * counts[0], counts


# boxes that reach far or without end to one side: their rays are still found.  (A sphere of radius
# 10^15 beside the rest, one of infinite radius, which nothing hits, and a triangle with a far vertex.)
@pytest.mark.parametrize("sphere,vertex", [((5e15, 5e15, 5e15, 5e15), None), ((-5e15, 5e15, 0, 5e15), None),
                                           ((1, 2, 3, np.inf), None), (None, (1e16, 1e16, 1e16)),
                                           (None, (1e18, -1e18, 1e18)), (None, (-1e18, 0.3, -1e17))])
def test_a_box_without_end_hides_nothing(host, sphere, vertex):
    rays = _rays(3000)
    rays[:1000, 4:7] = 0.0
    rays[np.arange(1000), 4 + np.arange(1000) % 3] = np.where(np.arange(1000) % 2, 1.0, -1.0)  # along an axis
    tri = _soup(600)
    if vertex:
        tri[17, 1] = vertex
    prims, box = _prims(tri, np.array([sphere] if sphere else np.zeros((0, 4)), np.float32))
    m = len(rays)
    out = [(np.zeros(m, np.float32), np.zeros(m, np.int32), np.zeros((m, 2), np.float32)) for _ in range(2)]
    ip = C.POINTER(C.c_int)
    for seed in range(8):
        host.rumi_host_walk(_f(prims), _f(box), len(prims), seed, _f(rays), m, 0, _f(out[0][0]),
                            out[0][1].ctypes.data_as(ip), _f(out[0][2]), _f(out[1][0]), out[1][1].ctypes.data_as(ip),
                            _f(out[1][2]))
        assert (out[1][1] >= 0).mean() > 0.05
        for a, b in zip(*out):
            assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [1e2, 1e4, 1e6])
def test_gpu_a_far_sphere_leaves_the_other_boxes_tight(radius):
    import rumi_b200
    from rumi_b200 import scenes
    from rumi_b200.scene import Film, Matte, Model, PathTracer, Scene, Sphere
    rays = _rays(20000)
    counts = []
    for r in (2.0, radius):
        sc = Scene()
        sc.add(Model(_soup(20000) * np.float32(0.5)), Matte(1.0, scenes.WHITE))
        sc.add(Sphere((0, 0, 0), r), Matte(0.5, scenes.WHITE))
        sc.camera, sc.image, sc.tracer = scenes.cornell_camera(), Film(8, 8, 1), PathTracer(1)
        gs = rumi_b200.GpuScene(sc)
        try:
            counts.append(gs.trace(rays)[3])
        finally:
            gs.close()
    assert counts[1] < 1.5 * counts[0], counts


@pytest.mark.gpu
@pytest.mark.parametrize("sphere", [(5e15, 5e15, 5e15, 5e15), (1, 2, 3, np.inf)])
def test_gpu_a_box_without_end_hides_nothing(sphere):
    import rumi_b200
    from rumi_b200 import _capi, scenes
    from rumi_b200.scene import Film, Matte, Model, PathTracer, Scene, Sphere
    sc = Scene()
    sc.add(Model(_soup(3000)), Matte(1.0, scenes.WHITE))
    sc.add(Sphere(sphere[:3], sphere[3]), Matte(0.5, scenes.WHITE))
    sc.camera, sc.image, sc.tracer = scenes.cornell_camera(), Film(8, 8, 1), PathTracer(1)
    rays = _rays(6000)
    m = len(rays)
    gs = rumi_b200.GpuScene(sc)
    try:
        got = []
        for mode in (1, 4):  # the binary and the four-wide walk
            t, prim = np.zeros(m, np.float32), np.zeros(m, np.int32)
            _capi.check(_capi.load().rumi_test_trace_scheme(
                gs.h, m, rays.ctypes.data_as(C.c_void_p), 0, mode, t.ctypes.data_as(C.c_void_p),
                prim.ctypes.data_as(C.c_void_p)), "rumi_test_trace_scheme")
            got.append((t, prim))
        assert (got[0][1] >= 0).mean() > 0.2
        assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    finally:
        gs.close()


def _flat(kind, rng, n):
    """Triangles whose boxes are flat: a grid of y = 0.37, one of y = 0, or pieces along any axis."""
    if kind == "pieces":
        c = rng.uniform(-1, 1, (n, 1, 3))
        e = rng.uniform(-0.1, 0.1, (n, 3, 3))
        e[np.arange(n), :, rng.integers(0, 3, n)] = 0
        return (c + e).astype(np.float32)
    k = int(np.sqrt(n / 2))
    g = np.linspace(-1, 1, k + 1)
    x, z = np.meshgrid(g, g, indexing="ij")
    p = np.stack([x, np.full_like(x, 0.37 if kind == "grid" else 0.0), z], -1)
    return np.concatenate([np.stack([p[:-1, :-1], p[1:, :-1], p[:-1, 1:]], 2).reshape(-1, 3, 3),
                           np.stack([p[1:, :-1], p[1:, 1:], p[:-1, 1:]], 2).reshape(-1, 3, 3)]).astype(np.float32)


# rays from up to five times the scene's extent, at inner points and edges: exact.  (From ten times it
# two of 40000 such rays miss a flat grid, from a hundred times one in forty; the binary walk misses
# more at every distance, 8 of 40000 from one and a half times.)
@pytest.mark.parametrize("distance", [1.5, 3.0, 5.0])
@pytest.mark.parametrize("kind", ["soup", "grid", "grid at zero", "pieces"])
def test_rays_from_far_away(host, kind, distance):
    rng = np.random.Generator(np.random.PCG64(5))
    tri = _soup(600) if kind == "soup" else _flat(kind, rng, 600)
    m = 8000
    w = rng.dirichlet([0.3] * 3, m)
    w[: m // 2] = np.where(rng.random((m // 2, 3)) < 0.4, 1e-7, w[: m // 2])  # on an edge or at a vertex
    w /= w.sum(1, keepdims=True)
    at = (tri[rng.integers(0, len(tri), m)] * w[:, :, None]).sum(1)
    d = rng.normal(size=(m, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros((m, 8), np.float32)
    rays[:, :3] = at - d * (2.0 * distance) * rng.uniform(0.7, 1.0, (m, 1))
    d = at - rays[:, :3].astype(np.float64)
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = 3.4e38
    prims, box = _prims(tri, np.zeros((0, 4), np.float32))
    out = [(np.zeros(m, np.float32), np.zeros(m, np.int32), np.zeros((m, 2), np.float32)) for _ in range(2)]
    ip = C.POINTER(C.c_int)
    host.rumi_host_walk(_f(prims), _f(box), len(prims), 3, _f(rays), m, 0, _f(out[0][0]), out[0][1].ctypes.data_as(ip),
                        _f(out[0][2]), _f(out[1][0]), out[1][1].ctypes.data_as(ip), _f(out[1][2]))
    assert (out[1][1] >= 0).mean() > 0.5
    for a, b in zip(*out):
        assert np.array_equal(a, b)
