"""The reconstruction's own transform passes at sides with every radix (2, 3, 4,
5, 8 and their composites), radii that fill and that leave half of the grid,
and a side that goes to the library's transforms, against the float64 oracle.

Tolerance: a transform of n^3 points in FP32 is off by about log2(n^3) 2^-24 of
the points' root mean square; the balancing divides by the result round
after round, which keeps its last round's errors only.  2e-5 of the map's peak
is ten times log2(144^3) 2^-24."""
import numpy as np
import pytest
import torch

import tg3
from oracle import reconstruct as RC

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _half(vdim, rng):
    q = np.fft.fftfreq(vdim, 1.0 / vdim)
    kz, ky, kx = np.meshgrid(q, q, np.arange(vdim // 2 + 1), indexing="ij")
    r = np.sqrt(kx * kx + ky * ky + kz * kz)
    T = 10.0 * np.exp(-r / (0.3 * vdim)) + 0.5
    F = np.fft.rfftn(rng.standard_normal((vdim, vdim, vdim))) * T / np.sqrt(vdim ** 3)
    return F, T


@pytest.mark.parametrize("N,pf,max_r,grid,kernel", [
    (48, 2, 23, True, "mkb"), (48, 2, 10, True, "trilinear"), (32, 4, 15, True, "mkb"),
    (72, 2, 30, True, "mkb"), (36, 4, 18, False, "mkb"), (80, 2, 36, False, "trilinear"),
    (60, 3, 25, False, "mkb"), (96, 2, 47, False, "mkb"), (54, 4, 20, False, "mkb"),
    (50, 2, 20, True, "mkb")])
def test_sides(N, pf, max_r, grid, kernel):
    F, T = _half(N * pf, np.random.default_rng(N + max_r))
    _check(N, pf, max_r, grid, kernel, F, T)


@pytest.mark.parametrize("N,grid", [(48, True), (64, True), (64, False), (72, True)])
def test_unpaired_plane(N, grid):
    """The column x = 0 as insertion leaves it: the writes to (0, y, z) and to
    (0, -y, -z) come from different pixels, so the two are not conjugates.  The
    real transform along x takes the real part of that column's sums."""
    vdim = 2 * N
    rng = np.random.default_rng(N)
    F, T = _half(vdim, rng)
    F[:, :, 0] += 0.3 * (rng.standard_normal((vdim, vdim)) + 1j * rng.standard_normal((vdim, vdim)))
    T[:, :, 0] *= rng.uniform(0.5, 1.5, (vdim, vdim))
    _check(N, 2, N // 2 - 3, grid, "mkb", F, T)


def _check(N, pf, max_r, grid, kernel, F, T):
    vdim = N * pf
    fsc = np.clip(1.05 - np.arange(N // 2 + 1) / (N / 2), 0, 1)
    ctx = tg3.Context(0)
    try:
        ctx.insert_begin(vdim, pf)
        ctx.insert_load(torch.as_tensor(F.astype(np.complex64)).to(DEV),
                        torch.as_tensor(T.astype(np.float32)).to(DEV))
        vol = torch.empty((N, N, N), dtype=torch.float32, device=DEV)
        rounds = ctx.reconstruct(vol, max_r, fsc=torch.as_tensor(fsc).to(DEV), join_half=True,
                                 grid_corr=grid,
                                 kernel=tg3.KERNEL_MKB if kernel == "mkb" else tg3.KERNEL_TRILINEAR)
        ctx.sync()
        got = vol.cpu().numpy()
    finally:
        ctx.close()
    ref, n = RC.reconstruct(F.astype(np.complex64).astype(np.complex128),
                            T.astype(np.float32).astype(np.float64), pf, max_r, fsc, True, grid,
                            kernel)
    assert rounds == n
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max()
