"""The GPU post-process at the sizes and films where its kernels can go wrong:
below, at and above the four pixels of a thread, a block and a block's share,
outputs that are not aligned for wide stores, and burn-out indices at both ends
of films whose luminances are all equal, all different or partly zero.

The reference is the same arithmetic in float64.  The kernels work in float32:
two powf (2 ulp each, amplified at most 2.2 times by the gamma) and a dozen
rounded operations, so 1e-5 relative, and one step of a byte.
"""
import numpy as np
import pytest

import azimuth_b200 as az

pytestmark = pytest.mark.gpu


def _reference(film, burnout, photographic, srgb):
    f = film.astype(np.float64)
    rgb = f[..., :3] / f[..., 3:]
    if photographic:
        lum = (rgb * [0.27, 0.67, 0.06]).sum(-1)
        flat = np.sort(lum.reshape(-1))
        factor = 0.18 / np.exp(np.log(flat + 1e-5).mean())
        at = int(np.float32(1.0 - np.float32(burnout) * np.float32(0.01)) * np.float32(flat.size - 1) + np.float32(0.5))
        white = flat[min(at, flat.size - 1)] * factor
        ls = lum * factor
        with np.errstate(divide="ignore", invalid="ignore"):
            ld = ls * (1.0 + ls / white ** 2) / (1.0 + ls)
            out = np.clip(rgb / lum[..., None] * ld[..., None], 0.0, 1.0)
        rgb = np.where(lum[..., None] != 0.0, out, rgb)
    if srgb:
        return np.where(rgb > 0.0031308, 1.055 * np.maximum(rgb, 0.0) ** (1.0 / 2.2) - 0.055, rgb * 12.92)
    return rgb ** (1.0 / 2.2)


@pytest.mark.parametrize("w,h", [(1, 1), (3, 1), (4, 1), (5, 1), (127, 1), (16, 16), (257, 31), (512, 9), (1201, 701)])
@pytest.mark.parametrize("kind", ["equal", "varied", "dark"])
@pytest.mark.parametrize("burnout", [0.0, 1.0, 100.0])
def test_sizes_and_burnout(gpu, w, h, kind, burnout):
    import torch
    rng = np.random.default_rng(w * 1000 + h)
    film = np.empty((h, w, 4), np.float32)
    film[..., 3] = 4.0
    film[..., :3] = {"equal": 2.0, "varied": rng.lognormal(0.0, 2.0, (h, w, 3)),
                     "dark": rng.random((h, w, 1)) * (rng.random((h, w, 1)) > 0.4) + 0.0}[kind]
    if kind == "dark":
        film[0, 0, :3] = 3.0          # with burn-out 100 the white point is a black pixel unless it is the only one
        if burnout == 100.0 and w * h > 1:
            pytest.skip("a white point of zero")
    dev = torch.from_numpy(film).cuda()
    n = w * h * 3
    for off in (0, 1):                # off = 1: outputs that are not aligned for wide stores
        rgb = torch.zeros(n + 4, device="cuda")
        rgb8 = torch.zeros(n + 4, dtype=torch.uint8, device="cuda")
        for photographic, srgb in ((True, True), (True, False), (False, True)):
            az.postprocess(dev.data_ptr(), w, h, burnout=burnout, photographic=photographic, srgb=srgb,
                           rgb_ptr=rgb.data_ptr() + 4 * off, rgb8_ptr=rgb8.data_ptr() + off)
            got = rgb[off:off + n].cpu().numpy().reshape(h, w, 3)
            got8 = rgb8[off:off + n].cpu().numpy().reshape(h, w, 3)
            want = _reference(film, burnout, photographic, srgb)
            assert np.abs(got - want).max() <= 1e-5 * max(1.0, float(np.abs(want).max()))
            assert np.abs(got8.astype(int) - (np.clip(got, 0, 1) * np.float32(255)).astype(int)).max() <= 0
        assert float(rgb[off + n:].abs().sum()) == 0.0 and int(rgb8[off + n:].sum()) == 0
