"""The FP32 cross term's tiles (launch_gemm_nt_fp32 chooses the tile from the
sizes): log-likelihoods of the local phase at sizes on and off the tile
edges, against the same sums in float64 over the library's own projections.

Tolerance: an FP32 chain of n multiply-adds is within n 2^-24 sum |a b| of
the exact sum, and its operands (the shifted data, formed in FP32 from
sincospif phases, and the norm) carry a few roundings more: (2 K + 64) 2^-24
times the sum of the terms' magnitudes."""
import numpy as np
import pytest
import torch

import tg3
from tg3 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def case():
    rng = np.random.default_rng(7)
    box, px, pf = 32, 1.5, 2
    bm = synth.blob_map(rng, 16, (2.0, 4.0), px, 8.0)
    iCol, iRow, _, _ = synth.pixel_index(box, 9, 1)
    ctx = tg3.Context(0)
    ctx.set_volume(0, synth.padded_volume(bm, box, pf, device=DEV, dtype=torch.float32), pf)
    ctx.set_pixels(iCol, iRow, box)
    yield dict(ctx=ctx, box=box, iCol=iCol, iRow=iRow)
    ctx.close()


# one column to two column tiles, one row to many tiles of every height
@pytest.mark.parametrize("nP,nR,nT", [(1, 1, 1), (1, 17, 16), (1, 33, 17), (3, 129, 129),
                                      (2, 1000, 100), (64, 200, 9), (8, 500, 50), (24, 250, 33),
                                      (20, 257, 121), (40, 1000, 100), (12, 2049, 84),
                                      (4, 900, 256)])
def test_tiles(case, nP, nR, nT):
    ctx, box, K = case["ctx"], case["box"], len(case["iCol"])
    g = torch.Generator(device=DEV).manual_seed(nP * 1000 + nR + nT)
    f64 = dict(dtype=torch.float64, device=DEV)
    rnd = lambda *s: torch.randn(*s, generator=g, **f64)  # noqa: E731
    quat = torch.nn.functional.normalize(rnd(nP, nR, 4), dim=-1).contiguous()
    trans = (2 * rnd(nP, nT, 2)).contiguous()
    dat = torch.complex(rnd(nP, K), rnd(nP, K)).to(torch.complex64)
    ctf = rnd(nP, K).float()
    sig = (-0.5 - rnd(nP, K).abs()).float()
    out = [torch.empty(s, **f64) for s in ((nP,), (nP, nR), (nP, nT), (nP,))]
    dvp = torch.empty((nP, nR, nT), dtype=torch.float32, device=DEV)
    ctx.local_phase(nP, nR, nT, dat, ctf, sig, quat, trans, torch.full((nP, nR), 1.0 / nR, **f64),
                    torch.full((nP, nT), 1.0 / nT, **f64), torch.ones(nP, **f64), None, *out, dvp,
                    tg3.SCORE_FP32)
    P = torch.empty((nP * nR, K), dtype=torch.complex64, device=DEV)
    mats = torch.empty((nP * nR, 9), **f64)
    torch.cuda.synchronize()
    tg3.check(tg3.lib().tg3_rotmat_d(tg3.ptr(quat), nP * nR, tg3.ptr(mats), None))
    torch.cuda.synchronize()
    ctx.project(0, mats, nP * nR, P)
    ctx.sync()
    P = P.reshape(nP, nR, K).to(torch.complex128)
    i, j = (torch.as_tensor(case[k], **f64) for k in ("iCol", "iRow"))
    t = trans.float().double()
    S = torch.exp(-2j * np.pi * (t[..., :1] * i + t[..., 1:] * j) / box)      # (nP, nT, K)
    X, c, w = dat.to(torch.complex128), ctf.double(), sig.double()
    A = (w * c * X)[:, None] * S.conj()
    flat = lambda z: torch.view_as_real(z).flatten(-2)     # noqa: E731
    x0 = (w * X.abs().square()).sum(1)[:, None, None]
    nrm = torch.einsum("lrk,lk->lr", P.abs().square(), w * c * c)[..., None]
    ref = x0 + nrm - 2 * torch.einsum("lrk,ltk->lrt", flat(P), flat(A))
    mag = x0.abs() + nrm.abs() + 2 * torch.einsum("lrk,ltk->lrt", flat(P).abs(),
                                                  (w * c * X).abs()[:, None].expand_as(A)
                                                  .repeat_interleave(2, -1))
    assert ((dvp.double() - ref).abs() <= (2 * K + 64) * 2.0 ** -24 * mag).all()
