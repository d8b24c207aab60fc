"""Shading comes in variants that leave the next rays in the queue in different ways (as they come, by
direction within a block, counted for the order of a large wave).  They are compiled separately and
share their arithmetic: a scene's film is the same bits whichever its frame takes, alone or in a
batch, also with textures, image-based light, subsurface and media, and a kept forward pass of an
ordered frame serves backward as its own first pass does."""
import os

import numpy as np
import pytest

import rumi_b200
import texture_cases as TC
from rumi_b200 import scenes
from rumi_b200.scene import Matte, Model, PathTracer

pytestmark = pytest.mark.gpu
DEPTH = 6
KINDS = ["caustic", "textured", "textured_medium", "ibl", "ibl_medium", "subsurface", "subsurface_medium", "medium"]


@pytest.fixture(scope="module")
def files(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("textures"))
    return TC.write_image(os.path.join(d, "a.bmp")), TC.write_sky(os.path.join(d, "s.hdr"))


def _scene(kind, files, w, h, spp, n_tris=0):
    base = kind.replace("_medium", "")
    if base == "caustic":
        sc = scenes.volumetric_caustic(w, h, spp, 6, 7)
    elif base == "textured":
        sc = TC.textured_cornell(w, h, spp, DEPTH, files[0])
    elif base == "ibl":
        sc = TC.ibl_scene(w, h, spp, DEPTH, files[1])
    elif base == "subsurface":
        sc = scenes.subsurface_cornell(w, h, spp, DEPTH)
    else:
        sc = scenes.cornell_pt(w, h, spp, DEPTH)
    if kind.endswith("medium"):
        sc = scenes.with_medium(sc)
    if n_tris:
        rng = np.random.Generator(np.random.PCG64(4))
        t = rng.uniform(0.1, 0.9, (n_tris, 1, 3)) + rng.uniform(-0.03, 0.03, (n_tris, 3, 3))
        sc.add(Model(t.astype(np.float32), albedo=scenes.random_albedo(n_tris, 5)), Matte(1.0, scenes.WHITE))
    sc.tracer = PathTracer(DEPTH)
    return sc


def _same(a, b):
    return np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32))


@pytest.mark.parametrize("kind", KINDS)
def test_few_records_and_walk(kind, files):
    gs = rumi_b200.GpuScene(_scene(kind, files, 61, 47, 9))
    try:
        want, sw = gs.render(seed=5, trace_mode=4)
        for serial in (False, True):
            got, sg = gs.render(seed=5, serial=serial)
            assert _same(got, want) and want.any()
            assert sg["rays_extend"] == sw["rays_extend"] and sg["rays_shadow"] == sw["rays_shadow"]
    finally:
        gs.close()


def test_batch_of_small_scenes_equals_their_frames(files):
    gs = [rumi_b200.GpuScene(_scene(k, files, 33 + 5 * i, 29, 4)) for i, k in enumerate(KINDS)]
    gs.append(rumi_b200.GpuScene(_scene("textured", files, 40, 24, 4, n_tris=3000)))
    b = rumi_b200.GpuBatch(gs)
    try:
        seeds = list(range(20, 20 + len(gs)))
        for graph in (False, True):
            films, _ = b.render([4] * len(gs), seeds, DEPTH, graph=graph)
            for g, s, f in zip(gs, seeds, films):
                assert _same(f, g.render(spp=4, seed=s)[0])
    finally:
        b.close()
        for g in gs:
            g.close()


@pytest.mark.parametrize("kind", ["textured", "ibl", "ibl_medium", "subsurface", "subsurface_medium"])
def test_ordered_wave_and_small_waves(kind, files):
    gs = rumi_b200.GpuScene(_scene(kind, files, 1031, 1021, 4, n_tris=3000))
    try:
        want, sw = gs.render(seed=9, wave_paths=1 << 20)
        got, sg = gs.render(seed=9)
        assert _same(got, want)
        assert sg["rays_extend"] == sw["rays_extend"] and sg["rays_shadow"] == sw["rays_shadow"]
    finally:
        gs.close()


@pytest.mark.parametrize("medium", [None, dict(sigma_s=(0.45, 0.35, 0.25), sigma_a=(0.04, 0.06, 0.09), g=0.2)])
def test_backward_after_an_ordered_forward(medium):
    w, h, spp = 1025, 1024, 4
    gs = rumi_b200.GpuScene(scenes.inverse_rendering(w, h, spp, 4, levels=5, medium=medium))
    try:
        want, _ = gs.render(seed=9, wave_paths=1 << 20)
        delta = np.random.default_rng(1).standard_normal(want.shape).astype(np.float32)
        own_a, own_v, st = gs.backward(delta, seed=9)
        film, _ = gs.forward(seed=9, keep=True)
        assert _same(film, want)
        kept_a, kept_v, sk = gs.backward(delta, seed=9)
        assert sk["extend_launches"] < st["extend_launches"]  # the kept radiance was used
        # atomic additions in another order: equal to rounding
        np.testing.assert_allclose(kept_a, own_a, rtol=1e-4, atol=1e-4 * np.abs(own_a).max())
        np.testing.assert_allclose(kept_v, own_v, rtol=1e-4, atol=1e-4 * np.abs(own_v).max())
    finally:
        gs.close()
