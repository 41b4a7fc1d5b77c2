"""Rays whose direction is not a unit vector against the C restatement of azimuth.

Point, area and spot lights are tested along the whole vector from the surface to the light, and a caller's ray may
have any length, while a mesh instance is traversed with a re-normalised local direction (src/azimuth_ray.h:24-66):
world and local distances then differ by the direction's length.  The interior (rooms of 8 x 4 x 8) has walls between
surfaces and lights many units apart; its meshes keep their transform, or are scaled by 2 and 0.5, or by turns, which
makes several groups.
"""
import ctypes as C

import numpy as np
import pytest

import azimuth_b200 as az
import oracle_lib as ol

pytestmark = pytest.mark.gpu

# byte offsets in azimuth's structs (include/az_abi.h; x86-64)
BVH_ROOT, LIGHTS, LIGHT_COUNT, LIGHT_SIZE, LIGHT_TYPE = 1344, 1368, 2712, 296, 292
RIGHT, LEFT, INVERSE, TRANSFORM, TYPE = 40, 48, 112, 176, 284
CAMERA_POSITION = 292
MESH_INSTANCE, BVH_NODE = 2, 3


def _floats(addr, n):
    return np.ctypeslib.as_array((C.c_float * n).from_address(addr))


def _entity(addr):
    return C.c_uint32.from_address(addr + TYPE).value


def _scale_instances(scene, factors):
    """Gives the scene's k-th mesh instance the scale factors[k % len(factors)], one for all axes or one each, and
    refits the tree's boxes."""
    turn = [0]

    def visit(e):
        box = _floats(e, 9)                     # Min, Max, Center
        if _entity(e) == BVH_NODE:
            parts = [visit(C.c_void_p.from_address(e + side).value) for side in (LEFT, RIGHT)]
            box[0:3] = np.minimum(parts[0][0:3], parts[1][0:3])
            box[3:6] = np.maximum(parts[0][3:6], parts[1][3:6])
            box[6:9] = 0.5 * (box[0:3] + box[3:6])
        else:
            assert _entity(e) == MESH_INSTANCE
            s = factors[turn[0] % len(factors)]
            turn[0] += 1
            _floats(e + TRANSFORM, 16)[[0, 5, 10]] = s
            _floats(e + INVERSE, 16)[[0, 5, 10]] = 1.0 / np.asarray(s)
            box.reshape(3, 3)[:] *= s
        return box

    visit(C.c_void_p.from_address(scene.scene_ptr + BVH_ROOT).value)


def _set_lights(scene, scale):
    """A point, an area and a spot light instead of the scene's own; returns what holds them."""
    s = np.ones(3) * scale
    buf = (C.c_ubyte * (3 * LIGHT_SIZE))()
    base = C.addressof(buf)
    _floats(base, 6)[:] = [*(s * [4, 3.4, 2]), 90, 80, 70]                                      # point, room 1
    _floats(base + LIGHT_SIZE, 15)[:] = [*(s * [20, 3.7, 5]), 60, 65, 70,                       # area, room 3
                                         s[0], 0, 0, 0, 0, s[2], 0, -1, 0]
    _floats(base + 2 * LIGHT_SIZE, 13)[:] = [*(s * [12.4, 3.8, 0.5]), 200, 190, 150,            # spot, room 2
                                             0.3, -0.5, 1, 80, 60, np.cos(np.radians(40)), np.cos(np.radians(30))]
    for k, kind in enumerate((0, 1, 3)):
        C.c_uint32.from_address(base + k * LIGHT_SIZE + LIGHT_TYPE).value = kind
    C.c_void_p.from_address(scene.scene_ptr + LIGHTS).value = base
    C.c_uint32.from_address(scene.scene_ptr + LIGHT_COUNT).value = 3
    return buf


FACTORS = {"identity": [1.0], "doubled": [2.0], "halved": [0.5], "by turns": [1.0, 2.0]}


def _lit_interior(scale, seed=3):
    """The interior under the three lights, its instances scaled; and a function that puts the scene back."""
    scene = az.generate_scene(az.SCENE_INTERIOR, seed=seed, width=96, height=54, spp=4, max_depth=2, detail=4)
    own = (C.c_void_p.from_address(scene.scene_ptr + LIGHTS).value,
           C.c_uint32.from_address(scene.scene_ptr + LIGHT_COUNT).value)
    _scale_instances(scene, [scale])
    lights = _set_lights(scene, scale)
    _floats(scene.camera_ptr + CAMERA_POSITION, 3)[:] *= scale

    def close():
        nonlocal lights
        C.c_void_p.from_address(scene.scene_ptr + LIGHTS).value, lights = own[0], None
        C.c_uint32.from_address(scene.scene_ptr + LIGHT_COUNT).value = own[1]
        scene.close()

    return scene, close


@pytest.mark.parametrize("flags", [0, az.FLAG_WATERTIGHT], ids=["cramer", "watertight"])
@pytest.mark.parametrize("case,variant", [("identity", 0), ("identity", 11), ("doubled", 0), ("doubled", 11),
                                          ("halved", 0)])   # 11: one query per thread
def test_shadows_of_lights_many_units_away(gpu, case, variant, flags):
    """The film's bar is that of the parity tests (1e-4 on all but a few pixels); the watertight test may also take
    the other side of a shared edge.  An occluder that is missed changes a pixel by the whole of a light."""
    import torch
    scene, close = _lit_interior(FACTORS[case][0])
    try:
        want = ol.port_film(scene, seed=5)
        film = torch.zeros((54, 96, 4), device="cuda")
        with az.GpuScene(scene) as g:
            g.render_device(film.data_ptr(), seed=5, variant=variant, flags=flags)
        ok, _, relmse = ol.film_compare(film.cpu().numpy(), want, 1e-4)
        print("%s: pixels within 1e-4 %.4f, relMSE %.3e" % (case, ok, relmse))
        assert ok >= (0.97 if flags else 0.99)
    finally:
        close()


@pytest.mark.parametrize("scale", [(40.0, 1.0, 0.05), (0.02, 30.0, 1.0)], ids=["long", "tall"])
def test_long_thin_boxes_and_distant_origins(gpu, scale):
    """Node boxes a thousand times as long as wide, and origins far from them in units of their width: the box tests'
    rounding stays inside the boxes' slack.  The phases find what one query per thread finds (1e-5 of the largest
    sum), and both what the restatement finds, with the parity tests' bar."""
    import torch
    scene, close = _lit_interior(np.array(scale))
    try:
        want = ol.port_film(scene, seed=6)
        assert (want[..., :3].max(axis=-1) > 0.0).mean() > 0.5
        films = []
        with az.GpuScene(scene) as g:
            for variant in (11, 0, 8, 20):
                film = torch.zeros((54, 96, 4), device="cuda")
                g.render_device(film.data_ptr(), seed=6, variant=variant)
                films.append(film.cpu().numpy())
        for f in films[1:]:
            assert np.abs(f - films[0]).max() <= 1e-5 * np.abs(films[0]).max()
        ok, _, relmse = ol.film_compare(films[1], want, 1e-4)
        print("%s: pixels within 1e-4 %.4f, relMSE %.3e" % (scale, ok, relmse))
        assert ok >= 0.99
    finally:
        close()


@pytest.mark.parametrize("length", [0.1, 1.0, 10.0])
@pytest.mark.parametrize("case", list(FACTORS))
def test_closest_hits_of_rays_of_any_length(gpu, case, length):
    """Nearest hits do not depend on the direction's length; distances are in units of it.  The bar is that of the
    closest-hit tests: the same entities but for ties, at most one in 50,000 rays."""
    scene = az.generate_scene(az.SCENE_INTERIOR, seed=3, width=8, height=8, spp=1, detail=4)
    try:
        _scale_instances(scene, FACTORS[case])
        rng = np.random.default_rng(4)
        n = 50000
        top = np.array([24.0, 3.8, 7.5]) * max(FACTORS[case])
        d = rng.normal(size=(n, 3))
        d *= length / np.linalg.norm(d, axis=1, keepdims=True)
        rays = np.concatenate([rng.uniform(0.3, 1.0, (n, 3)) * top, d, np.zeros((n, 1))], axis=1).astype(np.float32)
        ph, pu, _, pt = ol.closest_hit("port", scene, rays)
        with az.GpuScene(scene) as g:
            gh, gu, _, gt = g.closest_hit(rays)
            wh, wu, _, wt = g.closest_hit(rays, flags=az.FLAG_WATERTIGHT)
        assert ph.mean() > 0.5
        for h, u, t, bar in ((gh, gu, gt, 2e-5), (wh, wu, wt, 2e-4)):
            far = (h != ph) | ((h == 1) & (u != pu) & (np.abs(t - pt) > 1e-5 * np.abs(pt)))
            print("%s, length %g: %d of %d differ" % (case, length, int(far.sum()), n))
            assert far.sum() <= max(1, int(bar * n))
    finally:
        scene.close()
