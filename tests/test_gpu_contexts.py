"""A local phase while its context is the only one of its device that runs local
phases, beside a second one, and alone again: the launches differ (stages of the
split cross term, the SMs' split between shared memory and L1), the results do
not, to the last bit; nor do those of a plan that was captured alone."""
import numpy as np
import pytest
import torch

import tg3
from test_gpu_ragged import _outputs, setup  # noqa: F401
from tg3 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _context(vol, box):
    c = tg3.Context(0)
    c.set_volume(0, vol, 2)
    c.set_pixels(*synth.pixel_index(box, 9, 1)[:2], box)
    return c


def _phase(ctx, K, nP, nR, nT, precision):
    g = torch.Generator(device=DEV).manual_seed(nR)
    f64 = dict(dtype=torch.float64, device=DEV)
    rnd = lambda *s: torch.rand(*s, generator=g, **f64)  # noqa: E731
    quat = torch.nn.functional.normalize(rnd(nP, nR, 4) - 0.5, dim=-1).contiguous()
    dat = torch.complex(rnd(nP, K), rnd(nP, K)).to(torch.complex64)
    o = [torch.empty(s, **f64) for s in (nP, (nP, nR), (nP, nT), nP)]
    dvp = torch.empty((nP, nR, nT), dtype=torch.float32, device=DEV)
    torch.cuda.synchronize()
    ctx.local_phase(nP, nR, nT, dat, rnd(nP, K).float(), -rnd(nP, K).float(), quat, rnd(nP, nT, 2),
                    rnd(nP, nR), rnd(nP, nT), rnd(nP), None, *o, dvp, precision)
    ctx.sync()
    return [x.cpu().numpy() for x in (*o, dvp)]


@pytest.mark.parametrize("precision", [tg3.SCORE_FP32, tg3.SCORE_BF16X3], ids=["fp32", "bf16x3"])
def test_alone_and_beside(precision):
    box = 32
    rng = np.random.default_rng(3)
    bm = synth.blob_map(rng, 12, (2.0, 4.0), 1.5, 8.0)
    vol = synth.padded_volume(bm, box, 2, device=DEV, dtype=torch.float32)
    K = len(synth.pixel_index(box, 9, 1)[0])
    sizes = [(5, 300, 100), (3, 129, 256), (40, 64, 9)]
    a = _context(vol, box)
    b = None
    try:
        alone = [_phase(a, K, *s, precision) for s in sizes]
        b = _context(vol, box)
        other = [_phase(b, K, *s, precision) for s in sizes]
        beside = [_phase(a, K, *s, precision) for s in sizes]
        b.close()
        again = [_phase(a, K, *s, precision) for s in sizes]
    finally:
        a.close()
        if b:
            b.close()
    for runs in (other, beside, again):
        for x, y in zip(alone, runs):
            for u, v in zip(x, y):
                np.testing.assert_array_equal(u, v)


def test_plan_captured_alone(setup):                                # noqa: F811
    s, ctx = setup, setup["ctx"]
    out = _outputs(len(s["cls"]), s["nR"], s["nT"])
    plan = tg3.RaggedPlan(ctx, s["cls"], s["nR"], s["nT"], s["dev"], out, tg3.SCORE_BF16X3,
                          budget=1 << 20, graph=True)
    rng = np.random.default_rng(3)
    bm = synth.blob_map(rng, 12, (2.0, 4.0), 1.5, 8.0)
    vol = synth.padded_volume(bm, 32, 2, device=DEV, dtype=torch.float32)
    b = _context(vol, 32)
    got = []
    try:
        for step in range(3):
            if step == 1:
                _phase(b, len(synth.pixel_index(32, 9, 1)[0]), 2, 50, 9, tg3.SCORE_BF16X3)
            if step == 2:
                b.close()
            for v in out.values():
                v.zero_()
            torch.cuda.synchronize()
            plan.run()
            ctx.sync()
            got.append({k: v.cpu().numpy() for k, v in out.items()})
    finally:
        plan.close()
        b.close()
    for g in got[1:]:
        for k in g:
            np.testing.assert_array_equal(got[0][k], g[k])
