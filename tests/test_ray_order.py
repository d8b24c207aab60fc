"""Frames of large waves, whose rays are ordered between bounces.  On the CPU the bins stay inside
their table for every origin and direction; on the GPU a path does not see its queue position, so
the films are those of small waves, whose rays are not ordered, bit for bit."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    gxx = shutil.which("g++")
    inc = next((os.path.join(r, "include") for r in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                if r and os.path.isfile(os.path.join(r, "include", "cuda_runtime.h"))), None)
    if not gxx or not inc:
        pytest.skip("g++ or the CUDA headers are missing")
    so = str(tmp_path_factory.mktemp("order") / "liborder.so")
    subprocess.run([gxx, "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-w",
                    "-I", inc, "-o", so,
                    os.path.join(HERE, "host_build", "order_host.cpp")], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("lo,hi", [((-1, -2, -3), (1, 2, 3)), ((0, 0, 0), (0, 1, 1)), ((-3e38,) * 3, (3e38,) * 3),
                                   ((1e-30,) * 3, (2e-30,) * 3)])
def test_bins_stay_in_their_table(host, lo, hi):
    rng = np.random.Generator(np.random.PCG64(3))
    od = rng.normal(size=(4096, 6)).astype(np.float32)
    odd = np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 3.4e38, -3.4e38, 1e-45], np.float32)
    od[:2048] = np.where(rng.random((2048, 6)) < 0.4, rng.choice(odd, (2048, 6)), od[:2048])
    bins = np.empty(len(od), np.int32)
    box = np.array(lo + hi, np.float32)
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))
    n = host.rumi_host_sort_bins(len(od), p(box, C.c_float), p(od, C.c_float), p(bins, C.c_int))
    assert bins.min() >= 0 and bins.max() < n


def _scene(kind, w, h, spp, depth):
    from rumi_b200 import scenes
    from rumi_b200.scene import Film, Matte, Model, PathTracer, Scene
    rng = np.random.Generator(np.random.PCG64(11))
    n = 3000
    tris = rng.uniform(0.1, 0.9, (n, 1, 3)) + rng.uniform(-0.04, 0.04, (n, 3, 3))
    if kind == "medium":
        sc = scenes.volumetric_caustic(w, h, spp, 6, 7)
    else:
        sc = Scene()
        scenes.add_cornell_box(sc)
        sc.camera = scenes.cornell_camera()
        sc.image = Film(w, h, spp)
    sc.add(Model(tris.astype(np.float32), albedo=scenes.random_albedo(n, 5)), Matte(1.0, scenes.WHITE))
    sc.tracer = PathTracer(depth)
    return sc


# just below and above the line (4194304 paths a wave), ragged; three waves, the last a small one
@pytest.mark.gpu
@pytest.mark.parametrize("kind,w,h,spp,depth,wave", [("box", 1023, 1024, 4, 3, 0), ("box", 1025, 1027, 4, 1, 0),
                                                     ("box", 1025, 1027, 4, 7, 0), ("box", 411, 640, 36, 6, 1 << 22),
                                                     ("medium", 1031, 1021, 4, 6, 0)])
def test_ordered_frames_equal_small_waves(kind, w, h, spp, depth, wave):
    import rumi_b200
    gs = rumi_b200.GpuScene(_scene(kind, w, h, spp, depth))
    try:
        want, sw = gs.render(seed=9, wave_paths=1 << 20)
        for serial in (False, True):
            got, sg = gs.render(seed=9, wave_paths=wave, serial=serial)
            assert np.array_equal(np.asarray(want).view(np.uint32), np.asarray(got).view(np.uint32))
            assert sg["rays_extend"] == sw["rays_extend"] and sg["rays_shadow"] == sw["rays_shadow"]
    finally:
        gs.close()
