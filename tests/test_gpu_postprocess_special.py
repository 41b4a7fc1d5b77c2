"""The GPU post-process on films with values that a radix selection of the white point has to order: luminances below
zero, zeros of both signs, a white point of zero, infinities, NaN and pixels that no sample reached.

The reference is float64 numpy with the kernels' clamp, which takes a NaN for 0 (fmax and fmin return the other
operand).  A NaN or infinite luminance makes the log-average one too, so the tone-mapped film is black; without tone
mapping only its own pixel is affected.  Tolerance as in the test of sizes: two powf and a dozen rounded operations,
1e-5 relative.
"""
import numpy as np
import pytest

import azimuth_b200 as az

pytestmark = pytest.mark.gpu

KINDS = ["negative", "zeros", "white of zero", "infinite", "minus infinite", "nan", "negative nan", "no weight"]


def _film(kind, w, h):
    rng = np.random.default_rng(w * 100 + h)
    film = np.empty((h, w, 4), np.float32)
    film[..., 3] = 2.0
    film[..., :3] = rng.lognormal(0.0, 1.0, (h, w, 1))        # grey: the luminance has the colour's sign
    flat = film.reshape(-1, 4)
    third = np.arange(0, flat.shape[0], 3)
    if kind == "negative":
        flat[third, :3] = -1e-5 * rng.random((third.size, 1))     # log(L + 1e-5) stays finite
    elif kind == "zeros":
        flat[third, :3] = np.where(third % 2, 0.0, -0.0)[:, None]
    elif kind == "white of zero":
        flat[:, :3] = 0.0
        flat[0, :3] = 3.0
    else:
        last = flat[-1]
        last[:3] = {"infinite": np.inf, "minus infinite": -np.inf, "nan": np.nan, "negative nan": -np.float32(np.nan),
                    "no weight": 0.0}[kind]
        if kind == "no weight":
            last[3] = 0.0
    return film


def _clamp(v):
    return np.fmin(1.0, np.fmax(0.0, v))


def _reference(film, burnout, photographic, srgb):
    f = film.astype(np.float64)
    with np.errstate(all="ignore"):
        rgb = f[..., :3] / f[..., 3:]
        if photographic:
            lum = (rgb * [0.27, 0.67, 0.06]).sum(-1)
            flat = np.sort(lum.reshape(-1))                   # NaN last
            factor = 0.18 / np.exp(np.log(flat + 1e-5).mean())
            at = int(np.float32(1.0 - np.float32(burnout) * np.float32(0.01)) * np.float32(flat.size - 1)
                     + np.float32(0.5))
            white = flat[min(at, flat.size - 1)] * factor
            ls = lum * factor
            ld = ls * (1.0 + ls / white ** 2) / (1.0 + ls)
            rgb = np.where(lum[..., None] != 0.0, _clamp(rgb / lum[..., None] * ld[..., None]), rgb)
        if srgb:
            return np.where(rgb > 0.0031308, 1.055 * np.maximum(rgb, 0.0) ** (1.0 / 2.2) - 0.055, rgb * 12.92)
        return rgb ** (1.0 / 2.2)


@pytest.mark.parametrize("w,h", [(2, 1), (5, 1), (64, 33), (257, 91)])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("burnout", [0.0, 40.0, 90.0, 100.0])
def test_special_values(gpu, kind, w, h, burnout):
    import torch
    film = _film(kind, w, h)
    dev = torch.from_numpy(film).cuda()
    rgb = torch.zeros((h, w, 3), device="cuda")
    rgb8 = torch.zeros((h, w, 3), dtype=torch.uint8, device="cuda")
    for photographic, srgb in ((True, True), (False, True), (False, False)):
        az.postprocess(dev.data_ptr(), w, h, burnout=burnout, photographic=photographic, srgb=srgb,
                       rgb_ptr=rgb.data_ptr(), rgb8_ptr=rgb8.data_ptr())
        got, want = rgb.cpu().numpy(), _reference(film, burnout, photographic, srgb)
        assert np.array_equal(np.isnan(got), np.isnan(want)), (photographic, srgb)
        finite = np.isfinite(want)
        assert np.array_equal(got[~finite & ~np.isnan(want)], want[~finite & ~np.isnan(want)])
        assert np.abs(got[finite] - want[finite]).max(initial=0.0) <= 1e-5 * max(1.0, np.abs(want[finite]).max(initial=0.0))
        assert np.array_equal(rgb8.cpu().numpy(), (_clamp(got) * np.float32(255)).astype(np.uint8))
