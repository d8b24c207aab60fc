"""Frames whose rays are ordered between the first bounces and are too few for it in the later ones,
and the other way round over several waves: the films of small waves bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind, w, h, spp, depth):
    from rumi_b200 import scenes
    from rumi_b200.scene import Emissive, Film, Matte, Model, PathTracer, Rect, Scene
    rng = np.random.Generator(np.random.PCG64(11))
    n = 4000
    tris = rng.uniform(0.2, 0.8, (n, 1, 3)) + rng.uniform(-0.05, 0.05, (n, 3, 3))
    sc = Scene()
    if kind == "box":
        scenes.add_cornell_box(sc)
    else:  # in the open: most paths leave after a bounce or two
        sc.add(Rect((0, 2, 0), (1, 0, 0), (0, 0, 1), 1), Emissive(5.0, (1.0, 1.0, 1.0)))
    sc.add(Model(tris.astype(np.float32), albedo=scenes.random_albedo(n, 5)), Matte(1.0, scenes.WHITE))
    sc.camera, sc.image, sc.tracer = scenes.cornell_camera(), Film(w, h, spp), PathTracer(depth)
    return sc


# paths around the line for a wave (2^22); of their rays around the line for a bounce (2^21)
@pytest.mark.parametrize("kind,w,h,spp,wave", [("open", 1025, 1024, 4, 0), ("open", 2049, 1025, 4, 0), ("open", 1999, 2003, 4, 0),
                                               ("box", 1025, 1024, 4, 0), ("open", 1500, 1501, 4, 5000000)])
def test_films_equal_small_waves(kind, w, h, spp, wave):
    import rumi_b200
    gs = rumi_b200.GpuScene(_scene(kind, w, h, spp, 6))
    try:
        want, sw = gs.render(seed=9, wave_paths=1 << 20)
        for k in range(2):  # the second frame finds the counters as the first has left them
            got, sg = gs.render(seed=9, wave_paths=wave, serial=k == 1)
            assert np.array_equal(np.asarray(want).view(np.uint32), np.asarray(got).view(np.uint32))
            assert sg["rays_extend"] == sw["rays_extend"] and sg["rays_shadow"] == sw["rays_shadow"]
    finally:
        gs.close()
