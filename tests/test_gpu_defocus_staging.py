"""tg3_ExpectLocal3D_ctf stages its arrays in one pinned buffer that grows, inputs
and results in an order of their own: calls below, above and again below the
buffer's first size (256 KB), with and without the log-likelihoods, give what the
batched device call gives for the same particle, bit for bit.  The CTFs of the
batched call are the same FP64 formula on the GPU, rounded to float (its sine
and cosine; a last-bit difference of the FP64 value moves one float in 10^8)."""
import ctypes

import numpy as np
import pytest
import torch

import tg3
from tg3 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_sizes_in_turn():
    rng = np.random.default_rng(12)
    box, pf = 32, 2
    bm = synth.blob_map(rng, 12, (2.0, 4.0), 1.5, 8.0)
    vol = synth.padded_volume(bm, box, pf, device=DEV, dtype=torch.float32)
    iCol, iRow = (np.ascontiguousarray(x, np.int32) for x in synth.pixel_index(box, 9, 1)[:2])
    K, p, lib = len(iCol), tg3.ptr, tg3.lib()
    host = np.ascontiguousarray(vol.cpu().numpy().astype(np.complex64))
    h = ctypes.c_void_p()
    tg3.check(lib.tg3_volume_create(ctypes.byref(h), p(host), box * pf, pf))
    ctx = tg3.Context(0)
    k1, k2, ps, con = (float(np.float32(x)) for x in (0.06, 3e4, 0.2, 0.1))
    try:
        ctx.set_volume(0, vol, pf)
        ctx.set_pixels(iCol, iRow, box)
        for nR, nT, nD, with_dvp in ((40, 9, 3, True), (9000, 7, 5, True), (9000, 7, 1, False),
                                     (7, 3, 16, True), (33, 5, 2, False)):
            quat = rng.standard_normal((nR, 4))
            quat /= np.linalg.norm(quat, axis=1, keepdims=True)
            trans = rng.standard_normal((nT, 2))
            dat = (rng.standard_normal(K) + 1j * rng.standard_normal(K)).astype(np.complex64)
            defO = (-2e4 + 1e3 * rng.standard_normal(K)).astype(np.float32)
            freQ = (np.hypot(iCol, iRow) / (1.5 * box)).astype(np.float32)
            sig = (-0.05 - 0.1 * rng.random(K)).astype(np.float32)
            dpara = 1 + 0.05 * rng.standard_normal(nD)
            pR, pT, pD = rng.random(nR), rng.random(nT), rng.random(nD)
            wC, base = np.empty(1, np.float32), np.empty(1, np.float32)
            wR, wT, wD = (np.empty(n, np.float32) for n in (nR, nT, nD))
            dvp = np.empty((nD, nR, nT), np.float32) if with_dvp else None
            tg3.check(lib.tg3_ExpectLocal3D_ctf(
                h, p(dat), p(defO), p(freQ), k1, k2, ps, con, p(sig), p(iCol), p(iRow), K, box, p(quat),
                nR, p(trans), nT, p(dpara), nD, p(pR), p(pT), p(pD), 0.7, p(wC), p(wR), p(wT), p(wD),
                p(dvp), p(base)))
            d = lambda x: torch.as_tensor(np.ascontiguousarray(x)[None]).to(DEV)   # noqa: E731
            f2 = d(freQ).double() ** 2
            ki = k1 * d(defO).double() * d(dpara)[0][:, None] * f2 + k2 * f2 * f2 - ps
            ctf = (-np.sqrt(1 - con * con) * torch.sin(ki) + con * torch.cos(ki)).float()[None]
            o = [torch.empty(s, dtype=torch.float64, device=DEV)
                 for s in (1, (1, nR), (1, nT), (1, nD), 1)]
            dv = torch.empty((1, nD, nR, nT), dtype=torch.float32, device=DEV)
            one = torch.full((1,), 0.7, dtype=torch.float64, device=DEV)
            args = [d(dat), ctf.contiguous()] + [d(x) for x in (sig, quat, trans, pR, pT, pD)] + [one]
            torch.cuda.synchronize()
            ctx.local_phase_ctf(1, nR, nT, nD, *args, None, *o, dv, tg3.SCORE_FP32)
            ctx.sync()
            for got, ref in ((wC, o[0]), (wR, o[1][0]), (wT, o[2][0]), (wD, o[3][0]), (base, o[4])):
                np.testing.assert_array_equal(got, ref.float().cpu().numpy())
            if with_dvp:
                np.testing.assert_array_equal(dvp, dv[0].cpu().numpy())
    finally:
        ctx.close()
        lib.tg3_volume_destroy(h)
