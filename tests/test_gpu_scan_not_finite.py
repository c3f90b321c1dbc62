"""Global searches with a rotation that is not a number, an image that is not,
and log-likelihoods of -inf: the best log-likelihood is the largest of the
numbers, and one rotation's NaN reaches its own weight and the sums over
rotations, not the other rotations' weights.

As in test_gpu_scan_tiles.py the scan is held against its own log-likelihoods:
the reported best is the largest of them exactly, a marginal the sum of exp(L -
best) to 2^-23 |L| + 1e-5 relative (a log-likelihood is rounded to FP32, the
exponential and the sums are FP32)."""
import pytest
import torch

import tg3
from tg3 import synth

import numpy as np

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = dict(dtype=torch.float64, device=DEV)
BOX = 32


@pytest.fixture(scope="module")
def ctx():
    rng = np.random.default_rng(3)
    bm = synth.blob_map(rng, 12, (2.0, 4.0), 1.5, 8.0)
    c = tg3.Context(0)
    c.set_volume(0, synth.padded_volume(bm, BOX, 2, device=DEV, dtype=torch.float32), 2)
    c.set_pixels(*synth.pixel_index(BOX, 9, 1)[:2], BOX)
    yield c
    c.close()


def _inputs(ctx, nImg, nR, nT):
    K = len(synth.pixel_index(BOX, 9, 1)[0])
    g = torch.Generator(device=DEV).manual_seed(nImg + nR + nT)
    rnd = lambda *s: torch.randn(*s, generator=g, **F64)  # noqa: E731
    q = torch.nn.functional.normalize(rnd(nR, 4), dim=-1).contiguous()
    mats = torch.empty((nR, 9), **F64)
    tg3.check(tg3.lib().tg3_rotmat_d(tg3.ptr(q), nR, tg3.ptr(mats), None))
    torch.cuda.synchronize()
    return dict(mats=mats, trans=(2 * rnd(nT, 2)).contiguous(),
                dat=(0.2 * torch.complex(rnd(nImg, K), rnd(nImg, K))).to(torch.complex64),
                ctf=rnd(nImg, K).float(), sig=(-0.05 - 0.1 * rnd(nImg, K).abs()).float(),
                pR=torch.rand(nR, generator=g, **F64), pT=torch.rand(nT, generator=g, **F64))


def _scan(ctx, i, nImg, nR, nT, precision):
    wC, base = torch.empty(nImg, **F64), torch.empty(nImg, **F64)
    wR, wT = torch.empty((nImg, nR), **F64), torch.empty((nImg, nT), **F64)
    dvp = torch.empty((nImg, nR, nT), dtype=torch.float32, device=DEV)
    torch.cuda.synchronize()
    ctx.global_scan(0, nImg, nR, nT, i["dat"], i["ctf"], i["sig"], i["mats"], i["trans"], i["pR"],
                    i["pT"], wC, wR, wT, base, dvp, precision)
    ctx.sync()
    return wC, wR, wT, base, dvp.double()


SIZES = [(3, 127, 9), (5, 300, 32), (2, 256, 33), (4, 640, 49), (2, 1300, 256), (40, 77, 1)]
PRECISIONS = [tg3.SCORE_BF16X3, tg3.SCORE_FP32]


@pytest.mark.parametrize("precision", PRECISIONS, ids=["split", "fp32"])
@pytest.mark.parametrize("nImg,nR,nT", SIZES)
def test_nan(ctx, nImg, nR, nT, precision):
    i = _inputs(ctx, nImg, nR, nT)
    bad, img = nR // 3, nImg - 1
    i["mats"][bad] = float("nan")
    i["dat"][img, 5] = float("nan")
    wC, wR, wT, base, L = _scan(ctx, i, nImg, nR, nT, precision)
    r = torch.arange(nR, device=DEV) != bad
    assert L[:, bad].isnan().all() and L[img].isnan().all()
    assert wR[:, bad].isnan().all() and wR[img].isnan().all()
    assert wT.isnan().all() and wC.isnan().all()
    L, base, wR = L[:img, r], base[:img], wR[:img, r]
    assert torch.equal(base.float(), L.amax((1, 2)).float())
    want = torch.exp(L - base[:, None, None]) @ i["pT"]
    tol = 2.0 ** -23 * float(L.abs().max()) + 1e-5
    assert ((wR - want).abs() <= tol * want.abs() + 1e-30).all()


@pytest.mark.parametrize("precision", PRECISIONS, ids=["split", "fp32"])
@pytest.mark.parametrize("nImg,nR,nT", SIZES)
def test_minus_infinity(ctx, nImg, nR, nT, precision):
    """A CTF whose square times |P|^2 leaves FP32 for half of the rotations."""
    i = _inputs(ctx, nImg, nR, nT)
    P = torch.empty((nR, i["dat"].shape[1]), dtype=torch.complex64, device=DEV)
    torch.cuda.synchronize()
    ctx.project(0, i["mats"], nR, P)
    ctx.sync()
    p = int(P.abs().double().std(0).argmax())
    power = P[:, p].abs().double().square()
    i["ctf"].zero_()
    i["ctf"][:, p] = float((3.4e38 / 0.1 / power.median()).sqrt())
    i["sig"][:, p] = -0.1
    wC, wR, wT, base, L = _scan(ctx, i, nImg, nR, nT, precision)
    rows = L.isinf().all(2)
    assert rows.any() and not rows.all() and not L.isnan().any()
    assert torch.equal(base.float(), L.amax((1, 2)).float())
    # neighbouring FP32 numbers of this size are far more than 100 apart: the largest alone count
    e = (L == L.amax((1, 2), keepdim=True)).double()
    for got, want in ((wR, e @ i["pT"]), (wT, torch.einsum("lrt,r->lt", e, i["pR"])),
                      (wC, torch.einsum("lrt,r,t->l", e, i["pR"], i["pT"]))):
        torch.testing.assert_close(got, want, rtol=1e-5, atol=0)


@pytest.mark.parametrize("precision", PRECISIONS, ids=["split", "fp32"])
@pytest.mark.parametrize("nImg,nR,nT", [(3, 5, 9), (2, 130, 33), (5, 64, 49), (2, 70, 200)])
def test_infinite_prior(ctx, nImg, nR, nT, precision):
    """An infinite prior of one translation and log-likelihoods within a few units
    of one another: every rotation's weight and the image's are infinite, the
    translations' finite."""
    i = _inputs(ctx, nImg, nR, nT)
    i["sig"] *= 1e-5
    i["pT"][nT // 2] = float("inf")
    wC, wR, wT, base, L = _scan(ctx, i, nImg, nR, nT, precision)
    assert float((base[:, None, None] - L).max()) < 60
    assert (wR == float("inf")).all() and (wC == float("inf")).all()
    torch.testing.assert_close(wT, torch.einsum("lrt,r->lt", torch.exp(L - base[:, None, None]),
                                                i["pR"]), rtol=1e-4, atol=0)
