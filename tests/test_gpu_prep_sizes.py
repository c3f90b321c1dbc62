"""Image preprocessing at sides of every radix of the on-chip transform, one
with no factors for it, pixel lists that reach the edge of the half plane and
lists short of it, sides whose columns take several CTAs, and a repeated pixel,
against the float64 oracle.

Tolerance: an FP32 transform of N^2 points is off by about log2(N^2) 2^-24 of
the points' root mean square, the pixels entering it by a few 2^-24; 1e-5 of
the largest value is ten times log2(400^2) 2^-24."""
import numpy as np
import pytest
import torch

import tg3
from oracle import preprocess as PP

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _pixels(N, rU):
    i, j = np.meshgrid(np.arange(0, min(rU, N // 2) + 1), np.arange(-min(rU, N // 2), min(rU, N // 2) + 1))
    k = i * i + j * j <= rU * rU
    return i[k].astype(np.int32), j[k].astype(np.int32)


@pytest.mark.parametrize("N,n,r,rU,mask,std_n", [
    (24, 3, 9.0, 24, 1, 0.0), (64, 5, 24.5, 20, 1, 0.0), (48, 4, 20.0, 48, 0, 0.0),
    (70, 3, 30.0, 25, 1, 1.3), (90, 2, 36.0, 32, 1, 0.0), (98, 2, 39.2, 35, 1, 0.0),
    (110, 2, 44.0, 38, 1, 0.0), (130, 2, 52.0, 52, 1, 0.0), (144, 2, 71.9, 50, 1, 0.0),
    (198, 2, 80.0, 60, 1, 0.0), (200, 2, 80.0, 60, 0, 0.7), (220, 1, 88.0, 80, 1, 0.0),
    (256, 200, 102.4, 80, 1, 0.0), (256, 2, 102.4, 182, 1, 0.0), (320, 2, 128.0, 128, 1, 0.0),
    (400, 1, 270.0, 100, 1, 0.0), (94, 3, 37.6, 30, 1, 0.0), (94, 2, 40.0, 30, 0, 0.0)])
def test_sizes(N, n, r, rU, mask, std_n):
    rng = np.random.default_rng(N + rU)
    imgs = (10 + 3 * rng.standard_normal((n, N, N))).astype(np.float32)
    imgs += 5 * rng.random((n, 1, 1)).astype(np.float32)
    iCol, iRow = _pixels(N, rU)
    p = rng.permutation(len(iCol))
    iCol, iRow = np.append(iCol[p], iCol[p[0]]), np.append(iRow[p], iRow[p[0]])
    ctx = tg3.Context(0)
    try:
        ctx.set_pixels(iCol, iRow, N)
        store = torch.empty(n * N * N + 1, dtype=torch.float32, device=DEV)
        img = store[1:].view(n, N, N)          # 4-byte aligned only
        img.copy_(torch.as_tensor(imgs))
        dat = torch.full((n, len(iCol)), float("nan"), dtype=torch.complex64, device=DEV)
        stats = torch.empty((n, 3), dtype=torch.float32, device=DEV)
        torch.cuda.synchronize()
        ctx.prepare_images(img, r, dat, mask=bool(mask), std_n=std_n, stats=stats)
        ctx.sync()
    finally:
        ctx.close()
    ref, st, _ = PP.preprocess(imgs, r, iCol, iRow, mask=bool(mask), std_n=std_n or None)
    got = dat.cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
    np.testing.assert_allclose(stats.cpu().numpy(), st, rtol=2e-6)
