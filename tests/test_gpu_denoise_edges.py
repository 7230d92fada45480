"""The denoiser's fused passes (csrc/denoise.cu) against the filter in float64 numpy, on images
smaller than a warp's columns, a thread's rows or the largest step (16), odd sizes, every
combination of guides, black and non-finite guide pixels.

Tolerance: a tap's weight is off by at most 2^-22 of the exponential's argument and by
128 x 4 x 2^-24 = 3e-5 from the normal stop's 128th power, so a pass moves a pixel by at most
3e-5 of the colours it averages and five passes by 1.5e-4."""
import numpy as np
import pytest

from petrichor_gb300 import capi

pytestmark = pytest.mark.gpu


def _lum(c):
    return 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]


def _reference(c, albedo, normal, hdr):
    c = c.astype(np.float64)
    H, W = c.shape[:2]
    ys, xs = np.arange(H), np.arange(W)

    def shift(t, dy, dx):
        return t[np.clip(ys + dy, 0, H - 1)][:, np.clip(xs + dx, 0, W - 1)]

    def edge(t):
        y = np.maximum(_lum(t), 0.0)
        return np.log1p(y) if hdr else np.minimum(y, 1.0)

    factor, has_a = np.ones_like(c), np.zeros((H, W), bool)
    if albedo is not None:
        a = albedo.astype(np.float64)
        has_a = np.isfinite(a).all(-1)
        lit = has_a & (_lum(np.where(np.isfinite(a), a, 0.0)) > 0.01)
        factor = np.where(lit[..., None], np.maximum(np.where(np.isfinite(a), a, 1.0), 1e-3), 1.0)
    c = c / factor
    n, has_n = np.zeros_like(c), np.zeros((H, W), bool)
    if normal is not None:
        n = np.where(np.isfinite(normal), normal, 0.0).astype(np.float64)
        l2 = (n * n).sum(-1)
        has_n = np.isfinite(normal).all(-1) & (l2 > 0.25)
        n = np.where(has_n[..., None], n / np.sqrt(np.maximum(l2, 0.25))[..., None], 0.0)
    near = [(dy, dx) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    lum = edge(c)
    m1 = sum(shift(lum, *d) for d in near) / 9
    m2 = sum(shift(lum * lum, *d) for d in near) / 9
    var = np.maximum(m2 - m1 * m1, 0.0)
    h = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
    sigma = 2.0 if albedo is None and normal is None else 4.0
    for k in range(5):
        scale = 1.0 / (sigma * np.sqrt(sum(shift(var, *d) for d in near) / 9) + 1e-4)
        sc, sw, sv = np.zeros_like(c), np.zeros((H, W)), np.zeros((H, W))
        for i in range(5):
            for j in range(5):
                dy, dx = (i - 2) << k, (j - 2) << k
                w = np.ones((H, W))
                if (i, j) != (2, 2):
                    w = np.exp(-np.abs(lum - shift(lum, dy, dx)) * scale)
                    dot = np.maximum((n * shift(n, dy, dx)).sum(-1), 0.0)
                    w = np.where(has_n & shift(has_n, dy, dx), w * dot ** 128, w)
                    d = factor - shift(factor, dy, dx)
                    w = np.where(has_a & shift(has_a, dy, dx), w * np.exp(-(d * d).sum(-1) * 100.0), w)
                w = w * h[i] * h[j]
                sc += w[..., None] * shift(c, dy, dx)
                sw += w
                sv += w * w * shift(var, dy, dx)
        c, var = sc / sw[..., None], sv / (sw * sw)
        lum = edge(c)
    return c * factor


@pytest.mark.parametrize("guides", ["", "a", "n", "an"])
@pytest.mark.parametrize("height,width", [(1, 1), (1, 40), (47, 1), (3, 31), (13, 33), (50, 65), (97, 61)])
def test_small_images_match_float64(gpu_ctx, height, width, guides):
    rng = np.random.default_rng(1000 * height + width)
    color = np.exp(0.7 * rng.normal(size=(height, width, 3))).astype(np.float32)
    albedo = rng.uniform(0.0, 0.9, (height, width, 3)).astype(np.float32)
    base = np.array([0.3, 0.5, 0.8]) + 0.05 * rng.normal(size=(height, width, 3))
    normal = (base * rng.uniform(0.7, 1.4, (height, width, 1))).astype(np.float32)
    if height * width > 8:
        albedo[0, :3] = 0.0
        albedo[height // 2, width // 2] = np.inf
        normal[height // 3, width // 2] = np.nan
        normal[-1, -1] = 0.1
    a, n = (albedo if "a" in guides else None), (normal if "n" in guides else None)
    for hdr in (True, False):
        img = color if hdr else color / (1 + color)
        got = gpu_ctx.denoise(img, a, n, hdr=hdr)
        want = _reference(img, a, n, hdr)
        assert np.all(np.abs(got - want) <= 1.5e-4 * (np.abs(want) + np.abs(want).mean()))
