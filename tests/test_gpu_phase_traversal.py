"""The phase-scheduled traversal kernels against one query per thread.

Launch configuration 11 runs every query of a wave by one thread to its end
(the loop the closest-hit tests check against azimuth); the others vote per
warp.  Both must find the same hits whatever the number of queries: below,
at and above a warp and a warp's batch of 64, with all lanes starting together
or in groups, for triangles, transformed instances, top-level spheres and
every kind of light.  Sums of a sample differ in their order only: at most a
few hundred float additions, 1e-5 of the largest partial sum.
"""
import numpy as np
import pytest

import azimuth_b200 as az

pytestmark = pytest.mark.gpu

LOOP = 11
SCENES = [("cornell", az.SCENE_CORNELL, {}), ("features", az.SCENE_FEATURES, {}),
          ("dense_mesh", az.SCENE_DENSE_MESH, dict(detail=4)), ("motion_env", az.SCENE_MOTION_ENV, dict(detail=300)),
          ("env_spheres", az.SCENE_ENV_SPHERES, {}), ("interior", az.SCENE_INTERIOR, dict(detail=6))]


def _samples(g, scene, w, h, **kw):
    import torch
    out = torch.zeros((w * h * 4, 4), device="cuda")
    g.render_samples(out.data_ptr(), seed=11, **kw)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("name,sid,kw", SCENES, ids=[s[0] for s in SCENES])
@pytest.mark.parametrize("w,h", [(1, 1), (8, 1), (5, 7), (16, 1), (13, 11), (48, 40)])
def test_phases_find_what_single_threads_find(gpu, name, sid, kw, w, h):
    scene = az.generate_scene(sid, seed=2, width=w, height=h, spp=4, **kw)
    with az.GpuScene(scene) as g:
        ref = _samples(g, scene, w, h, variant=LOOP)
        scale = max(float(np.abs(ref).max()), 1e-6)
        for variant in (0, 1, 8, 10, 12, 20):
            got = _samples(g, scene, w, h, variant=variant)
            assert np.abs(got - ref).max() <= 1e-5 * scale, variant
        # waves of a few samples, and queues visited in sorted order
        got = _samples(g, scene, w, h, variant=8, chunk_samples=33)
        assert np.abs(got - ref).max() <= 1e-5 * scale
        got = _samples(g, scene, w, h, variant=8, flags=az.FLAG_ORDER_SHADOW | az.FLAG_ORDER_EXTEND)
        assert np.abs(got - ref).max() <= 1e-5 * scale
