"""Queries and frames on a caller's stream while another thread makes and drops scenes of the same
memory pool: the workspace they take is usable on that stream at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_results_on_a_callers_stream_beside_other_scenes():
    import torch
    import rumi_b200
    from rumi_b200 import scenes
    rng = np.random.Generator(np.random.PCG64(2))
    rays = np.zeros((4000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(0.0, 1.0, (4000, 3))
    d = rng.normal(size=(4000, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = 3.4e38
    big = scenes.bvh_bound_pt(16, 16, 1, 1, levels=6, seed=3)
    small = scenes.cornell_pt(96, 80, 4, 4)
    gs = rumi_b200.GpuScene(small)
    want_t, want_id, _, _ = gs.trace(rays)
    want = gs.render(seed=4)[0].copy()
    gs.close()
    stop, errors = threading.Event(), []

    def other():
        try:
            while not stop.is_set():
                g = rumi_b200.GpuScene(big)
                g.trace(rays)
                g.close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    th = threading.Thread(target=other)
    th.start()
    try:
        stream = torch.cuda.Stream()
        film = torch.zeros((80, 96, 3), device="cuda")
        torch.cuda.synchronize()
        for _ in range(40):  # each scene's first call allocates its workspace
            g = rumi_b200.GpuScene(small)
            dr = torch.from_numpy(rays).cuda()
            dt, dp = torch.zeros(4000, device="cuda"), torch.zeros(4000, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            g.trace_device(4000, dr.data_ptr(), dt.data_ptr(), dp.data_ptr(), stream=stream.cuda_stream)
            assert np.array_equal(dt.cpu().numpy(), want_t) and np.array_equal(dp.cpu().numpy(), want_id)
            g.render(seed=4, film_device_ptr=film.data_ptr(), stream=stream.cuda_stream)
            assert np.array_equal(film.cpu().numpy(), want)
            g.close()
    finally:
        stop.set()
        th.join()
    assert not errors
