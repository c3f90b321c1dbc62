"""The reconstruction's own passes at their larger sides (every pair of factors
from 16 x 15 to 32 x 16), all rounds and both directions of the transforms,
against the same chain in float64 by torch on the GPU.  F and T are Hermitian
(the transform of a real map, a radial T).  Tolerance as in
test_gpu_reco_sides.py: 2e-5 of the map's peak, ten times log2(n^3) 2^-24."""
import numpy as np
import pytest
import torch

import tg3
from oracle import reconstruct as RC

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
A, ALPHA, STEP = 1.9, 15.0, 1.0 / 100000


def _q(c, x):
    return c[:, None, None] ** 2 + c[None, :, None] ** 2 + x[None, None, :] ** 2


def _table(fn, n, device_index):
    return torch.as_tensor(fn(np.arange(n, dtype=np.float64)), device=DEV)[device_index]


def _reference(F, T, N, pf, max_r):
    """RC.reconstruct with grid correction and the MKB kernel, without an FSC."""
    v = N * pf
    c = torch.cat([torch.arange(v // 2), torch.arange(-v // 2, 0)]).to(DEV)
    half = torch.arange(v // 2 + 1, device=DEV)
    inside = _q(c, half) < (max_r * pf) ** 2
    krl = _table(lambda q: RC.mkb_rl(np.sqrt(np.rint(q / float(v) ** 2 / STEP) * STEP), A, ALPHA),
                 3 * (v // 2) ** 2 + 1, _q(c, c)) / RC.mkb_rl(0.0, A, ALPHA)
    T = T.double()
    W = inside.double()
    diff, no_dec = np.inf, 0
    for m in range(30):
        C = torch.fft.rfftn(torch.fft.irfftn(torch.complex(T * W, torch.zeros_like(T)),
                                             s=(v, v, v)) * krl).abs()
        W = torch.where(inside, W / C.clamp_min(1e-6), W)
        prev, diff = diff, float((C - 1).abs()[inside].max())
        no_dec = no_dec + 1 if diff > prev * 0.95 else 0
        if diff < 1e-2 or (m >= 10 and no_dec == 2):
            break
    del krl, T, C
    pad = torch.fft.irfftn(torch.where(inside, F.to(torch.complex128) * W, 0), s=(v, v, v))
    i = torch.arange(-N // 2, N // 2, device=DEV)
    k = _table(lambda q: RC.mkb_rl(np.sqrt(q) / v, A * pf, ALPHA), 3 * (N // 2) ** 2 + 1,
               _q(i, i)) / RC.mkb_rl(0.0, A * pf, ALPHA)
    return pad[i % v][:, i % v][:, :, i % v] / k, m + 1


@pytest.mark.parametrize("side", [240, 256, 288, 320, 360, 384, 400, 432, 480, 512])
def test_sides(side):
    pf = 2
    N = side // pf
    max_r = N // 2 - 1 if side % 3 else N // 3
    g = torch.Generator(device=DEV).manual_seed(side)
    c = torch.cat([torch.arange(side // 2), torch.arange(-side // 2, 0)]).to(DEV)
    r = _q(c, torch.arange(side // 2 + 1, device=DEV)).double().sqrt()
    T = (10.0 * torch.exp(-r / (0.3 * side)) + 0.5).float()
    F = torch.fft.rfftn(torch.randn((side,) * 3, generator=g, device=DEV, dtype=torch.float64))
    F = (F * T / side ** 1.5).to(torch.complex64).contiguous()
    del r
    ctx = tg3.Context(0)
    try:
        ctx.insert_begin(side, pf)
        torch.cuda.synchronize()
        ctx.insert_load(F, T)
        vol = torch.empty((N, N, N), dtype=torch.float32, device=DEV)
        rounds = ctx.reconstruct(vol, max_r, grid_corr=True, kernel=tg3.KERNEL_MKB, a=A, alpha=ALPHA)
        ctx.sync()
    finally:
        ctx.close()
    ref, n = _reference(F, T, N, pf, max_r)
    assert rounds == n
    assert float((vol - ref).abs().max()) <= 2e-5 * float(ref.abs().max())
    torch.cuda.empty_cache()
