"""tg3_ExpectLocal3D stages its arrays in one pinned buffer that grows: calls below, above and again below its first size (256 KB)
give what the batched device call gives for the same particle, bit for bit (the
same kernels at the same sizes, rounded to float)."""
import ctypes

import numpy as np
import pytest
import torch

import tg3
from tg3 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_sizes_in_turn():
    rng = np.random.default_rng(11)
    box, pf = 32, 2
    bm = synth.blob_map(rng, 12, (2.0, 4.0), 1.5, 8.0)
    vol = synth.padded_volume(bm, box, pf, device=DEV, dtype=torch.float32)
    iCol, iRow = (np.ascontiguousarray(x, np.int32) for x in synth.pixel_index(box, 9, 1)[:2])
    K, p, lib = len(iCol), tg3.ptr, tg3.lib()
    host = np.ascontiguousarray(vol.cpu().numpy().astype(np.complex64))
    h = ctypes.c_void_p()
    tg3.check(lib.tg3_volume_create(ctypes.byref(h), p(host), box * pf, pf))
    ctx = tg3.Context(0)
    try:
        ctx.set_volume(0, vol, pf)
        ctx.set_pixels(iCol, iRow, box)
        for nR, nT in ((40, 9), (9000, 25), (7, 3)):
            quat = rng.standard_normal((nR, 4))
            quat /= np.linalg.norm(quat, axis=1, keepdims=True)
            trans = rng.standard_normal((nT, 2))
            dat = (rng.standard_normal(K) + 1j * rng.standard_normal(K)).astype(np.complex64)
            ctf = rng.standard_normal(K).astype(np.float32)
            sig = (-0.05 - 0.1 * rng.random(K)).astype(np.float32)
            pR, pT = rng.random(nR), rng.random(nT)
            wC, base = np.empty(1, np.float32), np.empty(1, np.float32)
            wR, wT, dvp = (np.empty(s, np.float32) for s in (nR, nT, (nR, nT)))
            tg3.check(lib.tg3_ExpectLocal3D(h, p(dat), p(ctf), p(sig), p(iCol), p(iRow), K, box, p(quat),
                                            nR, p(trans), nT, p(pR), p(pT), 0.7, p(wC), p(wR), p(wT),
                                            p(dvp), p(base)))
            d = lambda x: torch.as_tensor(np.ascontiguousarray(x)[None]).to(DEV)   # noqa: E731
            o = [torch.empty(s, dtype=torch.float64, device=DEV) for s in (1, (1, nR), (1, nT), 1)]
            dv = torch.empty((1, nR, nT), dtype=torch.float32, device=DEV)
            args = [d(x) for x in (dat, ctf, sig, quat, trans, pR, pT)]
            one = torch.full((1,), 0.7, dtype=torch.float64, device=DEV)
            torch.cuda.synchronize()
            ctx.local_phase(1, nR, nT, *args, one, None, *o, dv, tg3.SCORE_FP32)
            ctx.sync()
            for got, ref in ((wC, o[0]), (wR, o[1][0]), (wT, o[2][0]), (base, o[3])):
                np.testing.assert_array_equal(got, ref.float().cpu().numpy())
            np.testing.assert_array_equal(dvp, dv[0].cpu().numpy())
    finally:
        ctx.close()
        lib.tg3_volume_destroy(h)
