"""Calls that no common stream orders: on a caller's non-blocking stream (a torch side stream is one), and of several
threads, each on a stream of its own."""
import ctypes as C
import threading
import time

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


@pytest.mark.parametrize("call", ["train", "infer", "eval", "params"])
def test_calls_on_one_guide_take_turns(gpu, call):
    """A call on a guide that another thread renders with begins when that render has ended: it returns later, and
    the render's film is that of the network before the call (the order of float sums apart: 1e-4)."""
    import torch
    scene = az.generate_scene(az.SCENE_INTERIOR, seed=1, width=640, height=360, spp=64, detail=8, max_depth=6)
    rng = np.random.default_rng(3)
    rows = np.zeros((4099, 16), np.float32)
    rows[:, 0:3] = rng.uniform(0.5, 3.5, (4099, 3))
    rows[:, 3] = 1.0
    rows[:, 5] = rows[:, 9] = rows[:, 13] = 1.0
    films = [torch.zeros((360, 640, 4), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    with az.GpuScene(scene) as g, az.Guide(g, seed=4) as guide:
        t0 = time.perf_counter()
        guide.render(films[0].data_ptr(), seed=7)
        alone = time.perf_counter() - t0
        end = []
        thread = threading.Thread(target=lambda: (guide.render(films[1].data_ptr(), seed=7),
                                                  end.append(time.perf_counter())))
        thread.start()
        time.sleep(min(0.02, 0.3 * alone))
        {"train": lambda: guide.train(rows, 8), "infer": lambda: guide.infer(rows), "eval": lambda: guide.eval(rows),
         "params": lambda: guide.set_params(*[0.5 * p for p in guide.params()])}[call]()
        done = time.perf_counter()
        thread.join()
    a, b = (f.cpu().numpy() for f in films)
    floor = 1e-3 * float(np.abs(a[..., :3]).mean())
    err = (np.abs(a - b) / np.maximum(np.abs(a), floor)).max(axis=-1)
    print("%s: render %.0f ms, the call ended %.1f ms after it" % (call, 1e3 * alone, 1e3 * (done - end[0])))
    assert alone > 0.04 and done > end[0] - 1e-3
    assert (err <= 1e-4).mean() >= 0.999
    scene.close()
