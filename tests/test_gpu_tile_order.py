"""Tile waves of several scenes: neither a job's film nor the time depends on the order of the jobs, and the waves'
kernels (of the phases, watertight ones among them) find what a render of each job alone finds."""
import numpy as np
import pytest

import azimuth_b200 as az
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, az.FLAG_WATERTIGHT], ids=["cramer", "watertight"])
def test_order_of_the_jobs(gpu, flags):
    """A scene of a few nodes first, or last.  Films as in the other tests of tile renders (1e-4: only the order of
    float sums differs).  Times of the same jobs in both orders, the best of five each, differ by less than a fifth:
    the launch configuration of the small scene, taken for all, costs a third."""
    import torch
    specs = [(az.SCENE_CORNELL, dict(width=96, height=96, spp=16)),
             (az.SCENE_FEATURES, dict(width=48, height=32, spp=4)),
             (az.SCENE_MOTION_ENV, dict(width=320, height=180, spp=9, detail=1500, max_depth=6)),
             (az.SCENE_DENSE_MESH, dict(width=400, height=400, spp=16, detail=6, max_depth=6))]
    scenes = [az.generate_scene(sid, seed=3 + k, **kw) for k, (sid, kw) in enumerate(specs)]
    gss = [az.GpuScene(s) for s in scenes]
    try:
        alone, films, jobs = [], [], []
        for k, (s, g) in enumerate(zip(scenes, gss)):
            w, h = s.resolution()
            alone.append(torch.zeros((h, w, 4), device="cuda"))
            g.render_device(alone[-1].data_ptr(), seed=30 + k, flags=flags)
            films.append(torch.zeros((h, w, 4), device="cuda"))
            jobs.append({"gpu_scene": g, "film_ptr": films[-1].data_ptr(), "seed": 30 + k})
        best = []
        for order in (jobs, jobs[::-1]):
            for f in films:
                f.zero_()
            torch.cuda.synchronize()
            per, _ = az.render_tiles(order, flags=flags)
            assert all(p["status"] == 0 for p in per)
            for k, (f, a) in enumerate(zip(films, alone)):
                a = a.cpu().numpy()
                assert a[..., 3].sum() > 0, k
                assert ol.film_compare(f.cpu().numpy(), a, 1e-4)[0] == 1.0, k
            best.append(min(az.render_tiles(order, flags=flags)[1]["gpu_ms"] for _ in range(5)))
        print("jobs in order %.2f ms, reversed %.2f ms" % tuple(best))
        assert max(best) <= 1.2 * min(best)
    finally:
        for g in gss:
            g.close()
        for s in scenes:
            s.close()
