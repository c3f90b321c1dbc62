"""Two host threads, each with a context of its own, whose calls launch the same
kernels with different amounts of shared memory: what each gets is, bit for
bit, what the same calls give one after another (the reconstruction's sums
have a fixed order)."""
import threading

import numpy as np
import pytest
import torch

import tg3

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_reconstruction_radii():
    """Maps of one padded side (512) with radii whose rows need 70 and 45 KB a
    CTA; a call's launches are spread over its balancing rounds."""
    N, pf = 256, 2
    v = N * pf
    g = torch.Generator(device=DEV).manual_seed(5)
    F = torch.randn(v, v, v // 2 + 1, generator=g, device=DEV, dtype=torch.complex64)
    T = 0.5 + torch.rand(v, v, v // 2 + 1, generator=g, device=DEV)
    ctxs = {r: tg3.Context(0) for r in (120, 20)}
    out, errors = {}, []

    def maps(radius, n):
        vols = []
        try:
            for _ in range(n):
                vol = torch.empty((N, N, N), dtype=torch.float32, device=DEV)
                ctxs[radius].reconstruct(vol, radius)
                ctxs[radius].sync()
                vols.append(vol)
        except tg3.TG3Error as e:
            errors.append(str(e))
        out[radius] = vols

    try:
        for c in ctxs.values():
            c.insert_begin(v, pf)
            c.insert_load(F, T)
            c.sync()
        torch.cuda.synchronize()
        for r in ctxs:
            maps(r, 1)
        alone = {r: vols[0].cpu().numpy() for r, vols in out.items()}
        threads = [threading.Thread(target=maps, args=a) for a in ((120, 6), (20, 12))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        for c in ctxs.values():
            c.close()
    assert not errors
    for r, vols in out.items():
        for vol in vols:
            np.testing.assert_array_equal(vol.cpu().numpy(), alone[r])
