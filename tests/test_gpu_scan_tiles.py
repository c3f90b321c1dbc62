"""The split search's tiles and the maxima that its GEMM hands the weights
kernel: scans whose translations, rotations and images end on and off the
tiles (128 rows, 256 columns, 32-column chunks that hold one, two or many
images; row groups of a chunked search).

The scan is held against its own log-likelihoods: the reported best is the
largest of them exactly (both round x0 + D, the one in FP64), and the
marginals are the sums of exp(L - best) over them.  A log-likelihood is
rounded to FP32 at |L| (2^-24 |L|), the exponential and the sums are FP32:
relative 2^-23 |L| + 1e-5 of a marginal."""
import numpy as np
import pytest
import torch

import tg3
from tg3 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ctx():
    rng = np.random.default_rng(3)
    box, pf = 32, 2
    bm = synth.blob_map(rng, 12, (2.0, 4.0), 1.5, 8.0)
    c = tg3.Context(0)
    c.set_volume(0, synth.padded_volume(bm, box, pf, device=DEV, dtype=torch.float32), pf)
    c.set_pixels(*synth.pixel_index(box, 9, 1)[:2], box)
    yield c
    c.close()


@pytest.mark.parametrize("nImg,nR,nT", [(1, 1, 1), (3, 127, 9), (5, 129, 31), (7, 300, 32),
                                        (2, 256, 33), (9, 640, 49), (310, 128, 25), (1, 1300, 256),
                                        (40, 77, 3), (306, 515, 64), (3, 70, 300)])
def test_best_and_marginals(ctx, nImg, nR, nT):
    iCol, _, _, _ = synth.pixel_index(32, 9, 1)
    K = len(iCol)
    g = torch.Generator(device=DEV).manual_seed(nImg + nR + nT)
    f64 = dict(dtype=torch.float64, device=DEV)
    rnd = lambda *s: torch.randn(*s, generator=g, **f64)  # noqa: E731
    q = torch.nn.functional.normalize(rnd(nR, 4), dim=-1).contiguous()
    mats = torch.empty((nR, 9), **f64)
    tg3.check(tg3.lib().tg3_rotmat_d(tg3.ptr(q), nR, tg3.ptr(mats), None))
    trans = (2 * rnd(nT, 2)).contiguous()
    dat = (0.2 * torch.complex(rnd(nImg, K), rnd(nImg, K))).to(torch.complex64)
    ctf = rnd(nImg, K).float()
    sig = (-0.05 - 0.1 * rnd(nImg, K).abs()).float()
    pR, pT = torch.rand(nR, generator=g, **f64), torch.rand(nT, generator=g, **f64)
    wC, wR = torch.empty(nImg, **f64), torch.empty((nImg, nR), **f64)
    wT, base = torch.empty((nImg, nT), **f64), torch.empty(nImg, **f64)
    dvp = torch.empty((nImg, nR, nT), dtype=torch.float32, device=DEV)
    torch.cuda.synchronize()
    ctx.global_scan(0, nImg, nR, nT, dat, ctf, sig, mats, trans, pR, pT, wC, wR, wT, base, dvp,
                    tg3.SCORE_BF16X3)
    ctx.sync()
    L = dvp.double()
    assert torch.equal(base.float(), dvp.amax((1, 2)))
    e = torch.exp(L - base[:, None, None])
    tol = 2.0 ** -23 * float(L.abs().max()) + 1e-5
    for got, want in ((wR, e @ pT), (wT, torch.einsum("lrt,r->lt", e, pR)),
                      (wC, torch.einsum("lrt,r,t->l", e, pR, pT))):
        assert ((got - want).abs() <= tol * want.abs() + 1e-30).all()
