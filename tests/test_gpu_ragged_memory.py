"""An uneven-batch plan that replays a captured graph, after the context's buffers
were replaced: by a call whose workspace is larger, by a second plan, by volumes
and pixel sets uploaded again at other sizes.  The plan's outputs stay the same,
bit for bit, and a pixel slot of another size is refused."""
import numpy as np
import pytest
import torch

import tg3
from test_gpu_ragged import BOX, DEV, PF, PX, _outputs, setup  # noqa: F401
from tg3 import synth

pytestmark = pytest.mark.gpu


def _run(plan, ctx, out):
    for v in out.values():
        v.zero_()
    torch.cuda.synchronize()
    plan.run()
    ctx.sync()
    return {k: v.cpu().numpy() for k, v in out.items()}


def _local(ctx, K, nP, nR, nT, precision):
    g = torch.Generator(device=DEV).manual_seed(1)
    f64 = dict(dtype=torch.float64, device=DEV)
    rnd = lambda *s: torch.rand(*s, generator=g, **f64)  # noqa: E731
    quat = torch.nn.functional.normalize(rnd(nP, nR, 4) - 0.5, dim=-1).contiguous()
    dat = torch.complex(rnd(nP, K), rnd(nP, K)).to(torch.complex64)
    o = [torch.empty(s, **f64) for s in (nP, (nP, nR), (nP, nT), nP)]
    torch.cuda.synchronize()
    ctx.local_phase(nP, nR, nT, dat, rnd(nP, K).float(), -rnd(nP, K).float(), quat, rnd(nP, nT, 2),
                    rnd(nP, nR), rnd(nP, nT), rnd(nP), None, *o, None, precision)
    ctx.sync()


@pytest.mark.parametrize("precision", [tg3.SCORE_FP32, tg3.SCORE_BF16X3], ids=["fp32", "bf16x3"])
def test_larger_workspace(setup, precision):                        # noqa: F811
    s, ctx = setup, setup["ctx"]
    out, out2 = (_outputs(len(s["cls"]), s["nR"], s["nT"]) for _ in range(2))
    args = (s["cls"], s["nR"], s["nT"], s["dev"])
    plan = tg3.RaggedPlan(ctx, *args, out, precision, budget=96 << 10, graph=True)
    try:
        first = _run(plan, ctx, out)
        held = ctx.workspace_bytes()
        ctx.use_pixels(-1)
        nP = 32
        for _ in range(2):
            while ctx.workspace_bytes() == held:
                nP *= 2
                _local(ctx, s["K"][0], nP, 400, 25, precision)
            held = ctx.workspace_bytes()
            torch.cuda.empty_cache()
            again = _run(plan, ctx, out)
            for k in first:
                np.testing.assert_array_equal(first[k], again[k])
        other = tg3.RaggedPlan(ctx, *args, out2, precision, budget=64 << 20, graph=True)
        try:
            for p, o in ((plan, out), (other, out2), (plan, out)):
                again = _run(p, ctx, o)
                for k in first:
                    np.testing.assert_array_equal(first[k], again[k])
        finally:
            other.close()
    finally:
        plan.close()


def test_volumes_and_pixels_again():
    rng = np.random.default_rng(5)
    ctx = tg3.Context(0)
    maps = [synth.blob_map(rng, 12, (2.0, 4.0), 1.5, 8.0) for _ in range(2)]
    vols = [synth.padded_volume(m, BOX, PF, device=DEV, dtype=torch.float32) for m in maps]
    st = synth.make_stack(9, [maps[0]], BOX, PX, PF, 9, synth.config_rL(BOX, PX), 6, 2.0, 0.1)
    nP, K = 6, len(st.iCol)
    nR, nT = rng.integers(20, 60, nP), rng.integers(3, 9, nP)
    R, T = int(nR.sum()), int(nT.sum())
    host = dict(dat=st.dat[:nP].astype(np.complex64).ravel(), ctf=st.ctf[:nP].astype(np.float32).ravel(),
                sig=st.sigRcp[:nP].astype(np.float32).ravel(),
                quat=synth.haar_quaternions(rng, R), trans=rng.standard_normal((T, 2)),
                pwR=rng.random(R) + 0.1, pwT=rng.random(T) + 0.1, pwC=np.ones(nP),
                permR=np.concatenate([rng.permutation(int(n)) for n in nR]).astype(np.int32),
                u0R=rng.random(nP) / nR, peakR=np.full(nP, np.nan),
                permT=np.concatenate([rng.permutation(int(n)) for n in nT]).astype(np.int32),
                u0T=rng.random(nP) / nT, peakT=np.zeros(nP))
    dev = {k: torch.as_tensor(np.ascontiguousarray(v)).to(DEV) for k, v in host.items()}
    out = _outputs(nP, nR, nT)

    def upload(vol):
        ctx.set_volume(0, vol, PF)
        ctx.set_pixels_slot(0, st.iCol, st.iRow, BOX)
        ctx.set_pixels(st.iCol, st.iRow, BOX)

    plan = None
    try:
        upload(vols[0])
        plan = tg3.RaggedPlan(ctx, np.zeros(nP, np.int32), nR, nT, dev, out, tg3.SCORE_FP32,
                              budget=1 << 20, graph=True)
        first = _run(plan, ctx, out)
        # other sizes, then the plan's again: every buffer is another one
        small = synth.padded_volume(maps[1], BOX // 2, PF, device=DEV, dtype=torch.float32)
        ctx.set_volume(0, small, PF)
        ctx.set_pixels_slot(0, st.iCol[:5], st.iRow[:5], BOX)
        torch.cuda.synchronize()
        ctx.set_volume(0, vols[0], PF)
        with pytest.raises(tg3.TG3Error):
            plan.run()
        upload(vols[0])
        again = _run(plan, ctx, out)
        for k in first:
            np.testing.assert_array_equal(first[k], again[k])
        upload(vols[1])                                   # in place: the new map is seen
        assert not np.array_equal(_run(plan, ctx, out)["wR"], first["wR"])
    finally:
        if plan:
            plan.close()
        ctx.close()
