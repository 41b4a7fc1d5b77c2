"""Calls on a caller's stream that the legacy default stream does not order (a torch side stream is non-blocking)."""
import ctypes as C

import numpy as np
import pytest

import azimuth_b200 as az

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("want", ["normals", "triangles", "attrs"])
def test_mesh_postprocess_is_finished_when_it_returns(gpu, want):
    """One output alone, and no total area, whose copy would wait for the stream: bit for bit what the call on a
    stream of its own gives, also when the scratch memory holds another mesh's values."""
    import torch
    side = torch.cuda.Stream()
    scenes = [az.generate_scene(az.SCENE_DENSE_MESH, seed=s, width=8, height=8, spp=1, detail=7, soup_only=True)
              for s in (1, 2)]
    try:
        refs = [az.mesh_postprocess(s) for s in scenes]
        for turn in range(6):
            s, ref = scenes[turn % 2], refs[turn % 2]
            key = {"normals": "vertex_normals", "triangles": "triangles", "attrs": "attrs"}[want]
            out = np.full_like(np.ascontiguousarray(ref[key], np.float32), -7.0)
            ptr = [out.ctypes.data if want == k else None for k in ("normals", "triangles", "attrs")]
            rc = az.lib().az_gpu_mesh_postprocess(s.soup_ptr, *ptr, None,
                                                  C.byref(az.make_opts(stream=side.cuda_stream)))
            assert rc == 0
            assert np.array_equal(out.view(np.uint32), np.ascontiguousarray(ref[key], np.float32).view(np.uint32))
    finally:
        for s in scenes:
            s.close()
