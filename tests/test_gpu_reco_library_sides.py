"""Reconstruction at sides that go to the library's transforms, 3-D and the single
plane of a 2-D class, from accumulators whose column x = 0 is as insertion leaves
it: (0, y, z) and (0, -y, -z) come from different pixels and are not conjugates.
The real transform along x takes the real part of that column's sums, as the
float64 oracle does.  Tolerance as in test_gpu_reco_sides.py: 2e-5 of the map's
peak is ten times log2(n^3) 2^-24."""
import numpy as np
import pytest
import torch

import tg3
from oracle import reconstruct as RC

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _half(vdim, dim, rng):
    q = np.fft.fftfreq(vdim, 1.0 / vdim)
    k = np.meshgrid(*([q] * (dim - 1)), np.arange(vdim // 2 + 1), indexing="ij")
    r = np.sqrt(sum(v * v for v in k))
    T = 10.0 * np.exp(-r / (0.3 * vdim)) + 0.5
    F = np.fft.rfftn(rng.standard_normal((vdim,) * dim)) * T / np.sqrt(float(vdim) ** dim)
    shape = (vdim,) * (dim - 1)
    F[..., 0] += 0.3 * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))
    T[..., 0] *= rng.uniform(0.5, 1.5, shape)
    return F.astype(np.complex64), T.astype(np.float32)


def _reference(F, T, pf, max_r, fsc, grid):
    return RC.reconstruct(F.astype(np.complex128), T.astype(np.float64), pf, max_r, fsc, True, grid,
                          "mkb")


@pytest.mark.parametrize("grid", [True, False])
@pytest.mark.parametrize("N", [16, 32, 50, 22])
def test_3d(N, grid):
    pf, max_r = 2, N // 2 - 2
    F, T = _half(N * pf, 3, np.random.default_rng(N))
    fsc = np.clip(1.05 - np.arange(N // 2 + 1) / (N / 2), 0, 1)
    ctx = tg3.Context(0)
    try:
        ctx.insert_begin(N * pf, pf)
        ctx.insert_load(torch.as_tensor(F).to(DEV), torch.as_tensor(T).to(DEV))
        vol = torch.empty((N, N, N), dtype=torch.float32, device=DEV)
        rounds = ctx.reconstruct(vol, max_r, fsc=torch.as_tensor(fsc).to(DEV), join_half=True,
                                 grid_corr=grid, kernel=tg3.KERNEL_MKB)
        ctx.sync()
        got = vol.cpu().numpy()
    finally:
        ctx.close()
    ref, n = _reference(F, T, pf, max_r, fsc, grid)
    assert rounds == n
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("grid", [True, False])
@pytest.mark.parametrize("N", [32, 64, 128, 50, 256, 512, 1024])
def test_2d(N, grid):
    pf, max_r = 2, N // 2 - 3
    F, T = _half(N * pf, 2, np.random.default_rng(N))
    fsc = np.clip(1.05 - np.arange(N // 2 + 1) / (N / 2), 0, 1)
    img, rounds = np.zeros((N, N), np.float32), np.zeros(1, np.int32)
    tg3.check(tg3.lib().tg3_Reconstruct2D(tg3.ptr(F), tg3.ptr(T), N * pf, pf, tg3.ptr(fsc), len(fsc),
                                          1, max_r, int(grid), tg3.KERNEL_MKB, 1.9, 15.0,
                                          tg3.ptr(img), tg3.ptr(rounds)))
    ref, n = _reference(F, T, pf, max_r, fsc, grid)
    assert int(rounds[0]) == n
    assert np.abs(img - ref).max() <= 2e-5 * np.abs(ref).max()


def test_3d_1024():
    """Box 512 at padding 2, the largest grid; the reference in float64 by torch,
    the column made of conjugates first."""
    N, pf, max_r = 512, 2, 100
    v = N * pf
    g = torch.Generator(device=DEV).manual_seed(8)
    c = torch.cat([torch.arange(v // 2), torch.arange(-v // 2, 0)]).to(DEV)
    q = c[:, None, None] ** 2 + c[None, :, None] ** 2 + torch.arange(v // 2 + 1, device=DEV) ** 2
    inside = q < (max_r * pf) ** 2
    del q
    F = torch.randn((v, v, v // 2 + 1), generator=g, device=DEV, dtype=torch.complex64)
    T = 0.5 + torch.rand((v, v, v // 2 + 1), generator=g, device=DEV)
    ctx = tg3.Context(0)
    try:
        ctx.insert_begin(v, pf)
        torch.cuda.synchronize()
        ctx.insert_load(F, T)
        vol = torch.empty((N, N, N), dtype=torch.float32, device=DEV)
        ctx.reconstruct(vol, max_r, grid_corr=False, kernel=tg3.KERNEL_TRILINEAR)
        ctx.sync()
    finally:
        ctx.close()
    V = torch.where(inside, F.to(torch.complex128) / T, 0)
    del F, T, inside
    i = torch.arange(v, device=DEV)
    V[..., 0] = 0.5 * (V[..., 0] + V[..., 0][-i % v][:, -i % v].conj())
    m = torch.fft.irfftn(V, s=(v, v, v))
    del V
    j = torch.arange(-N // 2, N // 2, device=DEV)
    m = m[j % v][:, j % v][:, :, j % v]
    r2 = (j[:, None, None] ** 2 + j[None, :, None] ** 2 + j ** 2).double()
    m /= torch.sinc(r2.sqrt() / v) ** 2
    assert float((vol - m).abs().max()) <= 2e-5 * float(m.abs().max())
    del m, r2, vol
    torch.cuda.empty_cache()
