"""MKB insertion where its work is cut.

- Lists that end within a run of 8 pixels, an item of 64 and a warp, against the
  same list inserted in two parts cut elsewhere: the same terms in another
  order.  With a table in shared memory (padding 2, 3) and one that does not
  fit (padding 1), also against the sums over all candidates in float64, within
  the relative L2 of 1e-4 that insertion is held to elsewhere.
- The order by radius (many draws, a far reach) against the order by draw (the
  same draws in two calls).
A voxel sums some tens of terms in FP32: 64 2^-24 of the sum of their
magnitudes, which for weights of one sign is the T accumulator's value itself
(and 12 times that for the values: |dat| <= 6, ctf >= 0.5)."""
import numpy as np
import pytest
import torch

import tg3

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _reference(box, pf, ic, ir, dat, ctf, mats, w):
    vdim = box * pf
    nx, a, alpha = vdim // 2 + 1, 1.9, 15.0
    F = np.zeros((vdim, vdim, nx), complex)
    T = np.zeros((vdim, vdim, nx))
    o = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    for l in range(len(mats)):
        v = (pf * (ic[:, None] * mats[l][:, 0] + ir[:, None] * mats[l][:, 1]))    # (K, 3): x, y, z
        n = np.ceil(v - 1.9).astype(int)[:, None] + o
        r2 = ((v[:, None] - n) ** 2).sum(-1)
        s = (1.9 * pf) ** 2 * 1e-5
        r2 = np.rint(r2 / s) * s
        k = np.where(r2 <= a * a, np.i0(alpha * np.sqrt(np.maximum(1 - r2 / (a * a), 0))) / np.i0(alpha), 0)
        val = k * (w[l] * ctf[l] * dat[l])[:, None]
        wt = k * (w[l] * ctf[l] ** 2)[:, None]
        flip = n[..., 0] < 0
        n = np.where(flip[..., None], -n, n)
        val = np.where(flip, val.conj(), val)
        at = (n[..., 2] % vdim, n[..., 1] % vdim, n[..., 0])
        ok = k > 0
        np.add.at(F, tuple(q[ok] for q in at), val[ok])
        np.add.at(T, tuple(q[ok] for q in at), wt[ok])
    return F, T


def _insert(box, pf, parts, draws, quat, dat, ctf, w, t):
    """F, T after inserting the (columns, rows, slice) of `parts`, `draws` at a time."""
    vdim = box * pf
    ctx = tg3.Context(0)
    try:
        ctx.set_pixels(*parts[0][:2], box)
        ctx.insert_begin(vdim, pf)
        for ic, ir, s in parts:
            ctx.set_pixels(ic, ir, box)
            for a in range(0, len(quat), draws):
                b = slice(a, a + draws)
                ctx.insert(len(quat[b]), dat[b, s].contiguous(), ctf[b, s].contiguous(), quat[b],
                           t[b], None, w[b], tg3.KERNEL_MKB)
                ctx.sync()
        F = torch.empty((vdim, vdim, vdim // 2 + 1), dtype=torch.complex64, device=DEV)
        T = torch.empty((vdim, vdim, vdim // 2 + 1), dtype=torch.float32, device=DEV)
        ctx.insert_read(F, T)
        ctx.sync()
        return F, T
    finally:
        ctx.close()


def _draws(rng, n, K):
    d = lambda x: torch.as_tensor(np.ascontiguousarray(x)).to(DEV)   # noqa: E731
    quat = rng.standard_normal((n, 4))
    dat = (rng.standard_normal((n, K)) + 1j * rng.standard_normal((n, K))).astype(np.complex64)
    out = (d(quat / np.linalg.norm(quat, axis=1, keepdims=True)), d(dat),
           d(rng.uniform(0.5, 1, (n, K)).astype(np.float32)),
           d(rng.uniform(0.5, 1, n).astype(np.float32)), d(rng.standard_normal((n, 2))))
    torch.cuda.synchronize()
    return out


def _same(a, b):
    (F0, T0), (F1, T1) = a, b
    assert ((T0 - T1).abs() <= 64 * 2.0 ** -24 * T1).all()
    assert ((F0 - F1).abs() <= 12 * 64 * 2.0 ** -24 * T1).all()


@pytest.mark.parametrize("box,pf,K,n,cut", [(16, 2, 2, 3, 1), (16, 2, 7, 5, 3), (20, 2, 64, 4, 31),
                                            (20, 2, 65, 3, 8), (24, 1, 100, 6, 63), (20, 3, 77, 4, 5),
                                            (32, 2, 200, 170, 129)])
def test_runs(box, pf, K, n, cut):
    rng = np.random.default_rng(K + n)
    R = (box * pf // 2 - 3) // pf
    j, i = np.mgrid[-R:R + 1, 0:R + 1]
    keep = (i * i + j * j <= R * R) & ~((i == 0) & (j < 0))
    i, j = i[keep], j[keep]
    q = rng.permutation(len(i))[:K]
    ic, ir = i[q].astype(np.int32), j[q].astype(np.int32)
    quat, dat, ctf, w, t = _draws(rng, n, K)
    w[n // 2] = 0
    t = torch.zeros_like(t)
    whole = _insert(box, pf, [(ic, ir, slice(0, K))], n, quat, dat, ctf, w, t)
    _same(whole, _insert(box, pf, [(ic[:cut], ir[:cut], slice(0, cut)), (ic[cut:], ir[cut:], slice(cut, K))],
                         n, quat, dat, ctf, w, t))
    mats = torch.empty((n, 9), dtype=torch.float64, device=DEV)
    tg3.check(tg3.lib().tg3_rotmat_d(tg3.ptr(quat), n, tg3.ptr(mats), None))
    torch.cuda.synchronize()
    ref = _reference(box, pf, ic, ir, dat.cpu().numpy(), ctf.cpu().numpy(),
                     mats.cpu().numpy().reshape(n, 3, 3), w.cpu().numpy())
    for got, r in zip(whole, ref):
        assert np.linalg.norm(got.cpu().numpy() - r) <= 1e-4 * np.linalg.norm(r)


def test_order_by_radius():
    rng = np.random.default_rng(5)
    box, pf, n = 256, 2, 200
    j, i = np.mgrid[-120:121, 0:121]
    keep = (i * i + j * j <= 120 * 120) & (i % 5 == 0) & (j % 7 == 0) & ~((i == 0) & (j < 0))
    ic, ir = i[keep].astype(np.int32), j[keep].astype(np.int32)
    quat, dat, ctf, w, t = _draws(rng, n, len(ic))
    parts = [(ic, ir, slice(0, len(ic)))]
    by_radius = _insert(box, pf, parts, n, quat, dat, ctf, w, t)
    assert (by_radius[1] > 0).sum() > 1e6
    _same(by_radius, _insert(box, pf, parts, n // 2, quat, dat, ctf, w, t))
