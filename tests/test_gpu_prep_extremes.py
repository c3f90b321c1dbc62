"""Image preprocessing of images whose rows exceed one table of the background
sums (5,888 rows), against float64 sums on the GPU, and of pixels whose
squares add up to more than FP32 holds, against the float64 oracle.

Tolerances: as in test_gpu_prep_sizes.py, 10 log2(N^2) 2^-24 of the largest
value; the statistics are FP64 results rounded to FP32."""
import numpy as np
import pytest
import torch

import tg3
from oracle import preprocess as PP

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _prepare(img, r, iCol, iRow):
    n, N, _ = img.shape
    ctx = tg3.Context(0)
    try:
        ctx.set_pixels(iCol, iRow, N)
        dat = torch.empty((n, len(iCol)), dtype=torch.complex64, device=DEV)
        stats = torch.empty((n, 3), dtype=torch.float32, device=DEV)
        torch.cuda.synchronize()
        ctx.prepare_images(img, r, dat, stats=stats)
        ctx.sync()
    finally:
        ctx.close()
    return dat.cpu().numpy(), stats.cpu().numpy()


def _pixels(rU):
    i, j = np.meshgrid(np.arange(rU + 1), np.arange(-rU, rU + 1))
    k = i * i + j * j <= rU * rU
    return i[k].astype(np.int32), j[k].astype(np.int32)


@pytest.mark.parametrize("N", [5888, 6000, 29160])
def test_large_images(N):
    r = 0.4 * N + 0.3
    g = torch.Generator(device=DEV).manual_seed(N)
    img = torch.empty((1, N, N), dtype=torch.float32, device=DEV)
    c = torch.arange(N, device=DEV, dtype=torch.float64) - N // 2
    rows = max(1, 2 ** 26 // N)
    for y in range(0, N, rows):
        img[0, y:y + rows].normal_(2.0, 3.0, generator=g)
        img[0, y:y + rows] += 2 * torch.exp(-((c[y:y + rows, None] - 0.1 * N) ** 2 + c ** 2)
                                            / (0.02 * N * N)).float()
    iCol, iRow = _pixels(8)
    dat, stats = _prepare(img, r, iCol, iRow)

    def chunks():
        for y in range(0, N, rows):
            q = (c[y:y + rows, None] ** 2 + c ** 2)
            yield y, img[0, y:y + rows].double(), q

    n = s1 = s2 = 0
    for _, x, q in chunks():
        b = x[q > np.floor(r * r)]
        n, s1, s2 = n + b.numel(), s1 + float(b.sum()), s2 + float((b - 2).square().sum())
    m = s1 / n
    sd = np.sqrt((s2 - n * (m - 2) ** 2) / (n - 1))
    sn = np.sqrt((s2 - n * (m - 2) ** 2) / sd ** 2 / (n - 1))
    np.testing.assert_allclose(stats[0], [m, sd, sn], rtol=2e-6)
    ex = torch.exp(-2j * np.pi * c[:, None] * torch.arange(9, device=DEV) / N)
    ey = torch.exp(-2j * np.pi * torch.arange(-8, 9, device=DEV)[:, None] * c / N)
    F = torch.zeros((17, 9), dtype=torch.complex128, device=DEV)
    for y, x, q in chunks():
        u = q.sqrt()
        w = torch.where(u < r, torch.ones_like(u), 0.5 + 0.5 * torch.cos((u - r) / 6 * np.pi))
        v = (x - m) / (sd * sn) * torch.where(u > r + 6, torch.zeros_like(u), w)
        F += ey[:, y:y + rows] @ (v.to(torch.complex128) @ ex)
    ref = F.cpu().numpy()[iRow + 8, iCol]
    assert np.abs(dat[0] - ref).max() <= 10 * np.log2(float(N) ** 2) * 2.0 ** -24 * np.abs(ref).max()


@pytest.mark.parametrize("N", [48, 64, 94, 256])
def test_large_pixels(N):
    """Squares of 1e36, a few thousand to the sum: the statistics and the scaled
    image are those of the oracle."""
    rng = np.random.default_rng(N)
    imgs = (1e18 * rng.standard_normal((3, N, N))).astype(np.float32)
    imgs[1] *= 1e-18
    iCol, iRow = _pixels(N // 4)
    r = 0.3 * N
    dat, stats = _prepare(torch.as_tensor(imgs).to(DEV), r, iCol, iRow)
    ref, st, _ = PP.preprocess(imgs, r, iCol, iRow)
    unit = np.stack([st[:, 1], st[:, 1], np.ones(3)], 1)
    np.testing.assert_allclose(stats / unit, st / unit, rtol=0, atol=2e-6)
    assert np.abs(dat - ref).max() <= 10 * np.log2(float(N) ** 2) * 2.0 ** -24 * np.abs(ref).max()


@pytest.mark.parametrize("N", [64, 94, 256])
def test_pixels_not_finite(N):
    """A NaN background pixel, an infinite one, a NaN corner (the sums' pivot) and a
    NaN inside the circle: such an image's mean or deviation is not a finite number
    (the last one's are, only its pixel data is not), the other images' results are
    the same bits as without them."""
    g = torch.Generator(device=DEV).manual_seed(N)
    img = torch.randn((6, N, N), generator=g, device=DEV) * 3 + 2
    iCol, iRow = _pixels(N // 4)
    r = 0.4 * N

    def run(x):
        ctx = tg3.Context(0)
        try:
            ctx.set_pixels(iCol, iRow, N)
            dat = torch.empty((6, len(iCol)), dtype=torch.complex64, device=DEV)
            stats = torch.empty((6, 3), dtype=torch.float32, device=DEV)
            torch.cuda.synchronize()
            ctx.prepare_images(x, r, dat, std_n=1.0, stats=stats)
            ctx.sync()
        finally:
            ctx.close()
        return dat, stats

    dat, stats = run(img)
    bad = img.clone()
    bad[0, 1, N // 2] = bad[2, 0, 0] = bad[3, N // 2, N // 2] = float("nan")
    bad[1, N - 1, 3] = float("inf")
    dat2, stats2 = run(bad)
    for k in (4, 5):
        assert torch.equal(dat[k], dat2[k]) and torch.equal(stats[k], stats2[k])
    assert not stats2[:3].isfinite().all(1).any()
    assert torch.equal(stats[3], stats2[3]) and dat2[:4].isnan().all()
