"""The watertight and the counting kernels of the phase-scheduled traversal, which are instantiations of their own.

The watertight loop of one query per thread is behind the closest-hit call only, so the phases are compared through
what a camera sample sees: every mesh instance emits its own colour and the light list is empty, which makes a sample's
radiance the name of the entity that it hit.  The reference is the C restatement with azimuth's test; as in the test
that compares the two triangle tests, 1e-3 of the rays may take the other of two entities that meet at the same
distance (the boxes' corners, which the symmetric cameras see at the middle of pixels).
"""
import ctypes as C

import numpy as np
import pytest

import azimuth_b200 as az
import oracle_lib as ol
from test_gpu_phase_traversal import SCENES, _samples

pytestmark = pytest.mark.gpu

# byte offsets in azimuth's structs (include/az_abi.h; x86-64)
BVH_ROOT, LIGHT_COUNT = 1344, 2712
RIGHT, LEFT, RADIANCE, EMITTER, TYPE = 40, 48, 252, 264, 284
BVH_NODE = 3


def _u32(addr):
    return C.c_uint32.from_address(addr)


def _name_entities(scene):
    """Every leaf of the scene's tree emits a colour of its own; returns how many there are."""
    count = 0
    stack = [C.c_void_p.from_address(scene.scene_ptr + BVH_ROOT).value]
    while stack:
        e = stack.pop()
        if _u32(e + TYPE).value == BVH_NODE:
            stack += [C.c_void_p.from_address(e + side).value for side in (RIGHT, LEFT)]
            continue
        count += 1
        _u32(e + EMITTER).value = 1
        np.ctypeslib.as_array((C.c_float * 3).from_address(e + RADIANCE))[:] = [count, 2 * count, 0.5 * count]
    return count


@pytest.mark.parametrize("sid,kw", [(az.SCENE_DENSE_MESH, dict(detail=5)), (az.SCENE_INTERIOR, dict(detail=8)),
                                    (az.SCENE_CORNELL, {}), (az.SCENE_MOTION_ENV, dict(detail=300))],
                         ids=["dense_mesh", "interior", "cornell", "motion_env"])
def test_watertight_phases_hit_what_the_restatement_hits(gpu, sid, kw):
    import torch
    w, h = 240, 200
    scene = az.generate_scene(sid, seed=6, width=w, height=h, spp=4, max_depth=1, filter=az.FILTER_BOX, **kw)
    try:
        assert _name_entities(scene) > 1
        lights, _u32(scene.scene_ptr + LIGHT_COUNT).value = _u32(scene.scene_ptr + LIGHT_COUNT).value, 0
        want = ol.port_film(scene, seed=9)
        tight = torch.zeros((h, w, 4), device="cuda")
        with az.GpuScene(scene) as g:
            for variant in (0, 1, 8, 11, 20):
                tight.zero_()
                g.render_device(tight.data_ptr(), seed=9, variant=variant, flags=az.FLAG_WATERTIGHT)
                off = (np.abs(tight.cpu().numpy() - want) > 1e-4 * np.abs(want).max()).any(axis=-1)
                print("watertight, variant %d: %d of %d pixels differ" % (variant, int(off.sum()), w * h))
                assert off.sum() <= max(2, int(1e-3 * w * h * 4))
        _u32(scene.scene_ptr + LIGHT_COUNT).value = lights
    finally:
        scene.close()


@pytest.mark.parametrize("name,sid,kw", SCENES, ids=[s[0] for s in SCENES])
@pytest.mark.parametrize("w,h", [(1, 1), (5, 7), (13, 11), (48, 40)])
@pytest.mark.parametrize("flags", [az.FLAG_WATERTIGHT, az.FLAG_COUNT_TRAVERSAL], ids=["watertight", "counting"])
def test_launch_configurations_agree(gpu, name, sid, kw, w, h, flags):
    """Below, at and above a warp: with either flag every launch configuration finds what the first one finds, in
    waves of a few samples too (1e-5 of the largest sum, as without the flags)."""
    scene = az.generate_scene(sid, seed=2, width=w, height=h, spp=4, **kw)
    with az.GpuScene(scene) as g:
        ref = _samples(g, scene, w, h, variant=8, flags=flags)
        scale = max(float(np.abs(ref).max()), 1e-6)
        for variant in (0, 1, 10, 20):
            assert np.abs(_samples(g, scene, w, h, variant=variant, flags=flags) - ref).max() <= 1e-5 * scale, variant
        got = _samples(g, scene, w, h, variant=8, chunk_samples=33, flags=flags)
        assert np.abs(got - ref).max() <= 1e-5 * scale
        if flags == az.FLAG_COUNT_TRAVERSAL:   # the counting kernels find what the others find
            assert np.abs(_samples(g, scene, w, h, variant=8) - ref).max() <= 1e-5 * scale
