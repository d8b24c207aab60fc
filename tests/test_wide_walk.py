"""The default walk (four-wide tree, packed slabs, two triangles per record) against a test of
every primitive.

On the CPU the walk itself (traverse_queue_ww built for the host, a warp of one lane) over a
random tree packed by the library's packing, with a stack column of 8 entries so that deep walks
move entries out of it.  On the GPU the library's own tree, through trace_mode 4 against the
binary walk of trace_mode 1.  Hits are exact: the same id, distance and barycentrics."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
FP = C.POINTER(C.c_float)
IP = C.POINTER(C.c_int)

# primitive counts around a record (2), a leaf (16), a batch of a leaf's lanes (32) and the
# builder's small tasks (256)
SIZES = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (3, 1, 1), (16, 0, 0), (17, 2, 3), (33, 0, 5), (257, 9, 4),
         (1300, 3, 40)]


def _scene(n_tri, n_rect, n_sph, scale, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    c = rng.uniform(-1, 1, (n_tri, 1, 3))
    tri = (c + rng.uniform(-0.3, 0.3, (n_tri, 3, 3))) * scale
    if n_tri > 2:
        tri[n_tri // 2] = tri[0]  # coplanar duplicates tie in distance
        tri[:, :, 1][n_tri // 3: n_tri // 2] = 0.25 * scale  # flat boxes
    p = rng.uniform(-1, 1, (n_rect, 3))
    ax = rng.integers(0, 3, n_rect)
    l, w = np.zeros((n_rect, 3)), np.zeros((n_rect, 3))
    l[np.arange(n_rect), ax] = rng.uniform(0.2, 0.8, n_rect)
    w[np.arange(n_rect), (ax + 1) % 3] = rng.uniform(0.2, 0.8, n_rect)
    rect = np.concatenate([p, l, w], 1) * scale
    sph = np.concatenate([rng.uniform(-1, 1, (n_sph, 3)), rng.uniform(0.05, 0.4, (n_sph, 1))], 1) * scale
    return tri.astype(np.float32), rect.astype(np.float32), sph.astype(np.float32)


def _rays(n, scale, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(-1.5, 1.5, (n, 3)) * scale
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 7] = 3.4e38
    k = n // 8
    a = rng.integers(0, 3, k)
    r[:k, 4:7] = np.where(rng.random((k, 3)) < 0.5, 0.0, -0.0)  # along an axis, signed zeros
    r[np.arange(k), 4 + a] = rng.choice([-1.0, 1.0], k)
    r[k:2 * k, 4 + rng.integers(0, 3)] = -0.0                   # in a coordinate plane
    r[2 * k:3 * k, 7] = rng.uniform(0.0, 2.0, k) * scale        # bounded
    r[3 * k:3 * k + 4, 7] = [np.inf, 0.0, -1.0, np.nan]
    r[3 * k + 4, 4:7] = 0.0                                     # no direction
    r[4 * k:5 * k, 3] = 1.0                                     # inside an object
    r[5 * k:6 * k, 0:3] *= 1e-3                                 # origins near the centre
    return r


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    gxx = shutil.which("g++")
    inc = next((os.path.join(r, "include") for r in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                if r and os.path.isfile(os.path.join(r, "include", "cuda_runtime.h"))), None)
    if not gxx or not inc:
        pytest.skip("g++ or the CUDA headers are missing")
    so = str(tmp_path_factory.mktemp("walk") / "libwalk.so")
    subprocess.run([gxx, "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-I", inc, "-o", so,
                    os.path.join(HERE, "host_build", "walk_host.cpp")], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("anyhit", [0, 1])
@pytest.mark.parametrize("scale", [1.0, 1e-3, 2e3])
@pytest.mark.parametrize("size", SIZES)
def test_walk_equals_a_test_of_every_primitive(host, size, scale, anyhit):
    tri, rect, sph = _scene(*size, scale, 3)
    n = sum(size)
    prims = np.zeros((n, 3, 4), np.float32)
    box = np.zeros((n, 6), np.float32)
    ids = prims.view(np.int32)
    nt, nr = size[0], size[1]
    prims[:nt, 0, :3], prims[:nt, 1, :3], prims[:nt, 2, :3] = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    box[:nt, :3], box[:nt, 3:] = tri.min(1, initial=np.inf), tri.max(1, initial=-np.inf)
    for k in range(3):
        prims[nt:nt + nr, k, :3] = rect[:, 3 * k:3 * k + 3]
    far = rect[:, 0:3] + rect[:, 3:6] + rect[:, 6:9]
    box[nt:nt + nr, :3], box[nt:nt + nr, 3:] = np.minimum(rect[:, :3], far), np.maximum(rect[:, :3], far)
    prims[nt + nr:, 0, :3], prims[nt + nr:, 1, 0] = sph[:, :3], sph[:, 3]
    box[nt + nr:, :3], box[nt + nr:, 3:] = sph[:, :3] - sph[:, 3:], sph[:, :3] + sph[:, 3:]
    ids[:, 0, 3] = np.arange(n)
    ids[nt:nt + nr, 1, 3] = 1 | np.where(np.arange(nr) % 2, 0x100, 0)
    ids[nt + nr:, 1, 3] = 2 | np.where(np.arange(size[2]) % 3 == 1, 0x200, 0)
    rays = _rays(800, scale, 5)
    m = rays.shape[0]
    out = [(np.zeros(m, np.float32), np.zeros(m, np.int32), np.zeros((m, 2), np.float32)) for _ in range(2)]
    f = lambda a: a.ctypes.data_as(FP)  # noqa: E731
    host.rumi_host_walk(f(prims), f(box), n, 11, f(rays), m, anyhit, f(out[0][0]), out[0][1].ctypes.data_as(IP),
                        f(out[0][2]), f(out[1][0]), out[1][1].ctypes.data_as(IP), f(out[1][2]))
    fine = ~np.isnan(rays[:, 7])  # a NaN bound: no box is entered, while each primitive accepts it
    assert not (out[0][0][~fine] > 0).any()
    if anyhit:
        assert ((out[0][0] > 0) == (out[1][0] > 0))[fine].all()
    else:
        for a, b in zip(*out):
            assert np.array_equal(a[fine], b[fine])
    assert n < 200 or (out[1][0] > 0).mean() > 0.05


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1.0, 2e3])
@pytest.mark.parametrize("size", SIZES)
def test_gpu_four_wide_walk_equals_the_binary_walk(size, scale):
    import rumi_b200
    from rumi_b200 import _capi, scenes
    from rumi_b200.scene import Dielectric, Emissive, Film, Matte, Model, PathTracer, Rect, Scene, Sphere
    tri, rect, sph = _scene(*size, scale, 7)
    sc = Scene()
    if len(tri):
        sc.add(Model(tri), Matte(1.0, (0.5, 0.5, 0.5)))
    for k, q in enumerate(rect):
        sc.add(Rect(q[0:3], q[3:6], q[6:9], 1), Emissive(1.0, (1.0, 1.0, 1.0)) if k % 2 else Matte(1.0, (0.5, 0.5, 0.5)))
    for q in sph:
        sc.add(Sphere(q[0:3], float(q[3])), Dielectric(1.5, 1.0, (0.0, 0.0, 0.0)))
    sc.camera, sc.image, sc.tracer = scenes.cornell_camera(), Film(8, 8, 1), PathTracer(1)
    gs = rumi_b200.GpuScene(sc)
    try:
        rays = _rays(6000, scale, 13)
        m = rays.shape[0]
        got = {}
        for mode in (1, 4):
            for anyhit in (0, 1):
                t, prim = np.zeros(m, np.float32), np.zeros(m, np.int32)
                _capi.check(_capi.load().rumi_test_trace_scheme(
                    gs.h, m, rays.ctypes.data_as(C.c_void_p), anyhit, mode, t.ctypes.data_as(C.c_void_p),
                    prim.ctypes.data_as(C.c_void_p)), "rumi_test_trace_scheme")
                got[mode, anyhit] = t, prim
        assert np.array_equal(got[1, 0][0], got[4, 0][0]) and np.array_equal(got[1, 0][1], got[4, 0][1])
        assert np.array_equal(got[1, 1][1], got[4, 1][1])
        assert sum(size) < 200 or (got[1, 0][1] >= 0).mean() > 0.05
    finally:
        gs.close()
