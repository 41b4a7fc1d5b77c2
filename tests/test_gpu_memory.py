"""What the library keeps between calls: it goes back to the driver when asked for, and does not make waves smaller."""
import pytest

import azimuth_b200 as az

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _build_and_close(torch):
    scene = az.generate_scene(az.SCENE_DENSE_MESH, seed=1, width=256, height=256, spp=16, detail=7, soup_only=True)
    film = torch.zeros((256, 256, 4), device="cuda")
    with az.GpuScene(scene, from_soup=True) as g:
        g.render_device(film.data_ptr(), seed=1)
    scene.close()


def test_kept_memory_is_given_back(gpu):
    import torch
    _build_and_close(torch)              # modules and torch's own film are in place
    az.release_memory()
    before = _free()
    for _ in range(2):
        _build_and_close(torch)
        assert _free() < before - (64 << 20)     # a scene's memory is kept for the next one
        az.release_memory()
        assert _free() >= before - (4 << 20)
    az.release_memory()                  # nothing left to give back
    with pytest.raises(az.AzError):
        az.release_memory(device=1 << 20)
    _build_and_close(torch)              # and the next call takes it again


def test_kept_memory_counts_as_free_for_the_wave_size(gpu):
    """The default wave is a power of two of which the free memory holds four in queues: 346 bytes a sample with one
    light.  With half of the kept memory missing to 2^23 samples, what the pool keeps makes up for it."""
    import torch
    az.release_memory()
    empty = _free()
    _build_and_close(torch)
    kept = empty - _free()
    assert kept > 256 << 20
    need = 4 * 346 * (1 << 23)
    scene = az.generate_scene(az.SCENE_CORNELL, seed=1, width=1024, height=1024, spp=9, max_depth=2)   # 1.1 x 2^23
    film = torch.zeros((1024, 1024, 4), device="cuda")
    with az.GpuScene(scene) as g:
        fill = torch.empty(_free() - (need - kept // 2), dtype=torch.uint8, device="cuda")
        try:
            assert _free() < need
            st = g.render_device(film.data_ptr(), seed=1, stats=True)
        finally:
            del fill
            torch.cuda.empty_cache()
    assert st["chunks"] == 2 and st["retries"] == 0, st
    scene.close()
