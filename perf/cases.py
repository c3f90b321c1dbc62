"""The work that users of this library have it do, as cases that can be timed and compared.

Sizes come from the library's own benchmark workloads and tests (box 64 to 256, padding 2, the
cutoffs, hypothesis counts and batch sizes of the particle-filter rounds, the global search, 2-D
classification, uneven batches, the learned E-step and its training, insertion, reconstruction and
preprocessing), and the ranges around them.  Inputs are synthetic and made from a seed: Gaussian-blob
maps, whose transforms are analytic, and noisy central slices of them at known poses."""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "thunder-refactor-expectation_gb300"))
import tg3  # noqa: E402

DEV = "cuda:0"
PF = 2
F64, F32, I32, C64, C128 = (torch.float64, torch.float32, torch.int32, torch.complex64,
                            torch.complex128)


# ------------------------------------------------------------------------------- the cases --
def listed():
    return [
        # one particle through the reference-shaped host call, as the reference's optimiser makes
        # it once per particle: the smallest work, where launches and host calls count
        dict(name="particle_box64", path="particle", box=64, rU=16, nR=100, nT=9),
        # a particle-filter round at production size, plain precision: 1,000 x 100 hypotheses
        dict(name="local_fp32_box256", path="local", box=256, rU=80, nP=32, nR=1000, nT=100, nD=1,
             prec="fp32"),
        # the same in the split precision, on a batch whose size divides nothing
        dict(name="local_bf16_box256", path="local", box=256, rU=80, nP=61, nR=1000, nT=100, nD=1,
             prec="bf16"),
        # uneven batches after narrowing: four classes, own cutoffs and set sizes per particle
        dict(name="ragged_box192", path="ragged", box=192, rU=96, nC=4, nP=192, nR_lo=200,
             nR_hi=8000, nT_lo=9, nT_hi=81, prec="bf16"),
        # the first iteration's global search over one map, plain precision (6,912 x 49)
        dict(name="global_fp32_box64", path="global", box=64, rU=16, nImg=333, nDir=192, nPsi=36,
             half=3, prec="fp32"),
        # the same in the split precision, on the whole set of a small refinement
        dict(name="global_bf16_box64", path="global", box=64, rU=16, nImg=2000, nDir=192, nPsi=36,
             half=3, prec="bf16"),
        # 2-D classification: 16 class images, 72 in-plane rotations x 49 shifts
        dict(name="class2d_box128", path="class2d", box=128, rU=24, nK=16, nImg=1000, nR=72,
             half=3, prec="bf16"),
        # the learned E-step as one call: network, matching, rescoring, fallback search
        dict(name="learned_box256", path="learned", box=256, rU=80, nC=2, nP=1000, nDir=192,
             nPsi=36, nRot=256, nTrans=25, half=3, fall=0.12, prec="bf16"),
        # one minibatch of the pose network's training: forward of both halves, loss, gradients
        dict(name="train_batch256", path="train", n=256),
        # insertion of a batch's best poses into fresh accumulators, read out at the end
        dict(name="insert_box256", path="insert", box=256, rU=80, nP=2000, kernel="mkb"),
        # one map from its accumulators, with the balancing of the weights
        dict(name="reconstruct_box256", path="reconstruct", box=256, rU=120, kernel="mkb",
             grid=True),
        # a stack's images to the likelihood's pixel data
        dict(name="prepare_box256", path="prepare", box=256, rU=80, n=1024),
    ]


def draw(rng):
    log = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    even = lambda v: 2 * int(round(v / 2))                                # noqa: E731
    path = rng.choice(["particle", "local", "local", "local", "ragged", "global", "global",
                       "class2d", "learned", "train", "insert", "reconstruct", "prepare"])
    prec = rng.choice(["fp32", "bf16"])
    if path == "particle":
        box = even(log(40, 160))
        return dict(path=path, box=box, rU=int(box * rng.uniform(0.2, 0.35)),
                    nR=int(log(50, 1000)), nT=int(log(5, 100)))
    if path == "local":
        box = even(log(48, 288))
        c = dict(path=path, box=box, rU=int(box * rng.uniform(0.2, 0.4)), nP=int(log(2, 96)),
                 nR=int(log(60, 2000)), nT=int(log(9, 121)),
                 nD=rng.choice([1, 1, 1, rng.randint(3, 9)]), prec=prec)
        c["nT"] = min(c["nT"], 200 // c["nD"])
        K = n_pixels(c["rU"])
        most = 32 * 1000 * 9930
        while c["nP"] * c["nR"] * K * max(1.0, c["nD"] * c["nT"] / 100) > most:
            c["nP" if c["nP"] > 2 else "nR"] //= 2
        return c
    if path == "ragged":
        box = even(log(96, 192))
        return dict(path=path, box=box, rU=int(box * rng.uniform(0.3, 0.48)),
                    nC=rng.randint(1, 4), nP=rng.randint(40, 150), nR_lo=rng.randint(100, 300),
                    nR_hi=rng.randint(1000, 6000), nT_lo=9, nT_hi=rng.randint(20, 81), prec=prec)
    if path == "global":
        box = even(log(48, 160))
        c = dict(path=path, box=box, rU=int(box * rng.uniform(0.2, 0.3)), nImg=int(log(20, 1500)),
                 nDir=rng.randint(40, 192), nPsi=rng.randint(12, 36), half=rng.randint(1, 4),
                 prec=prec)
        while c["nImg"] * c["nDir"] * c["nPsi"] * (2 * c["half"] + 1) ** 2 * n_pixels(c["rU"]) > 8e10:
            c["nImg"] = max(1, c["nImg"] // 2)
        return c
    if path == "class2d":
        box = even(log(64, 160))
        return dict(path=path, box=box, rU=int(box * rng.uniform(0.15, 0.25)),
                    nK=rng.randint(2, 20), nImg=int(log(50, 1000)), nR=rng.randint(24, 90),
                    half=rng.randint(1, 3), prec=prec)
    if path == "learned":
        box = even(log(96, 200))
        return dict(path=path, box=box, rU=int(box * rng.uniform(0.2, 0.32)),
                    nC=rng.randint(1, 3), nP=int(log(60, 900)), nDir=rng.randint(60, 192),
                    nPsi=rng.randint(20, 36), nRot=rng.randint(64, 256), nTrans=rng.randint(9, 25),
                    half=rng.randint(1, 3), fall=round(rng.uniform(0.05, 0.25), 3), prec=prec)
    if path == "train":
        return dict(path=path, n=int(log(32, 320)))
    if path == "insert":
        box = even(log(64, 256))
        return dict(path=path, box=box, rU=int(box * rng.uniform(0.2, 0.32)),
                    nP=int(log(60, 2000)), kernel=rng.choice(["mkb", "mkb", "trilinear"]))
    if path == "reconstruct":
        box = rng.choice([48, 64, 72, 90, 96, 108, 120, 128, 144, 160, 180, 192])
        return dict(path=path, box=box, rU=int(box * rng.uniform(0.35, 0.47)),
                    kernel=rng.choice(["mkb", "trilinear"]), grid=rng.random() < 0.8)
    box = even(log(48, 256))
    return dict(path=path, box=box, rU=int(box * rng.uniform(0.2, 0.4)), n=int(log(40, 1000)))


# ------------------------------------------------------------------- geometry and synthetic data --
def pixels(rU):
    """Half-plane pixels 1 <= |k| < rU: columns and rows, int32."""
    j = np.arange(-rU, rU + 1)
    i = np.arange(0, rU + 1)
    jj, ii = np.meshgrid(j, i, indexing="ij")
    jj, ii = jj.ravel(), ii.ravel()
    u = ii * ii + jj * jj
    keep = ~((ii == 0) & (jj < 0)) & (u < rU * rU) & (u >= 1) & (np.rint(np.sqrt(u)) < rU)
    return ii[keep].astype(np.int32), jj[keep].astype(np.int32)


def n_pixels(rU):
    return len(pixels(rU)[0])


def generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) + 77)
    return g


def uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=DEV, dtype=F64)


def normal(g, *shape, dtype=F64):
    return torch.randn(*shape, generator=g, device=DEV, dtype=dtype)


def unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def haar(g, *shape):
    q = unit(normal(g, *shape, 4))
    return torch.where(q[..., :1] < 0, -q, q)


def quat_mul(a, b):
    aw, ax, ay, az = a.unbind(-1)
    bw, bx, by, bz = b.unbind(-1)
    return torch.stack([aw * bw - ax * bx - ay * by - az * bz, aw * bx + ax * bw + ay * bz - az * by,
                        aw * by - ax * bz + ay * bw + az * bx,
                        aw * bz + ax * by - ay * bx + az * bw], -1)


def near(g, q, spread, n):
    """n rotations about each of q (..., 4): turned by rotation vectors of deviation `spread`."""
    v = 0.5 * spread * normal(g, *q.shape[:-1], n, 3)
    th = v.norm(dim=-1, keepdim=True)
    d = torch.cat([torch.cos(th), torch.sin(th) * v / th.clamp_min(1e-12)], -1)
    return unit(quat_mul(q[..., None, :].expand(*d.shape), d))


def matrix(q):
    """Rotation matrices (..., 3, 3) of unit quaternions (w, x, y, z)."""
    w, x, y, z = q.unbind(-1)
    r = [1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
         2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
         2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]
    return torch.stack(r, -1).reshape(*q.shape[:-1], 3, 3)


def rotation_grid(nDir, nPsi):
    """nDir directions on a spiral over the sphere x nPsi in-plane angles, as quaternions."""
    k = torch.arange(nDir, device=DEV, dtype=F64)
    th = torch.acos(1 - 2 * (k + 0.5) / nDir)
    ph = k * (math.pi * (3 - math.sqrt(5)))
    psi = torch.arange(nPsi, device=DEV, dtype=F64) * (2 * math.pi / nPsi)
    z0 = torch.zeros_like(k)
    qd = quat_mul(torch.stack([torch.cos(ph / 2), z0, z0, torch.sin(ph / 2)], -1),
                  torch.stack([torch.cos(th / 2), z0, torch.sin(th / 2), z0], -1))
    z1 = torch.zeros_like(psi)
    qp = torch.stack([torch.cos(psi / 2), z1, z1, torch.sin(psi / 2)], -1)
    return quat_mul(qd[:, None].expand(nDir, nPsi, 4), qp[None].expand(nDir, nPsi, 4)).reshape(-1, 4)


def shift_grid(half):
    g = torch.arange(-half, half + 1, device=DEV, dtype=F64)
    ty, tx = torch.meshgrid(g, g, indexing="ij")
    return torch.stack([ty.reshape(-1), tx.reshape(-1)], 1).contiguous()


def blobs(g, n, box):
    """n Gaussian blobs: amplitudes, widths and centres in pixels, inside 0.31 box of the centre."""
    c = unit(normal(g, n, 3)) * (0.31 * box) * uniform(g, 0, 1, n, 1) ** (1 / 3)
    return uniform(g, 0.5, 1, n), uniform(g, 1.4, 2.7, n), c


def axis_factors(sig, c, f):
    """The blobs' transforms along one axis at frequencies f (cycles per pixel): (blobs, f)."""
    e = torch.exp(-2 * math.pi ** 2 * sig[:, None] ** 2 * f[None] ** 2)
    return e * torch.exp(-2j * math.pi * c[:, None] * f[None])


def volume(bl, box):
    """The blobs' transform on the padded half grid [z][y][x], complex64."""
    amp, sig, c = bl
    v = PF * box
    f = torch.fft.fftfreq(v, device=DEV, dtype=F64)
    x = torch.arange(v // 2 + 1, device=DEV, dtype=F64) / v
    gz, gy, gx = (axis_factors(sig, c[:, a], t).to(C64) for a, t in ((2, f), (1, f), (0, x)))
    w = (amp * (2 * math.pi * sig ** 2) ** 1.5).to(C64)
    yx = (gy[:, :, None] * gx[:, None, :]).reshape(len(amp), -1)
    return torch.matmul((gz * w[:, None]).T, yx).reshape(v, v, v // 2 + 1).contiguous()


def slices(bl, R, box, iCol, iRow, rU):
    """Central slices of the blobs' transform at rotations R (n, 3, 3): (n, K) complex64."""
    amp, sig, c = bl
    i = torch.arange(0, rU + 1, device=DEV, dtype=F64) / box
    j = torch.arange(-rU, rU + 1, device=DEV, dtype=F64) / box
    w = (amp * (2 * math.pi * sig ** 2) ** 1.5)
    at = ((torch.as_tensor(iRow, device=DEV).long() + rU) * (rU + 1)
          + torch.as_tensor(iCol, device=DEV).long())
    out = torch.empty(len(R), len(iCol), device=DEV, dtype=C64)
    p = c @ R                                           # (n, blobs, 3): the centres' plane coordinates
    for s in range(0, len(R), 64):
        gi = torch.exp(-2 * math.pi ** 2 * sig[:, None] ** 2 * i ** 2) * torch.exp(
            -2j * math.pi * p[s:s + 64, :, 0, None] * i)
        gj = torch.exp(-2 * math.pi ** 2 * sig[:, None] ** 2 * j ** 2) * torch.exp(
            -2j * math.pi * p[s:s + 64, :, 1, None] * j)
        grid = torch.matmul((gj * w[:, None]).to(C64).transpose(1, 2), gi.to(C64))
        out[s:s + 64] = grid.reshape(len(grid), -1)[:, at]
    return out


def ctf_attributes(g, n):
    a = torch.zeros(n, 7, device=DEV, dtype=F64)
    a[:, 0], a[:, 4], a[:, 5] = 3e5, 2.7e7, 0.1
    a[:, 1:3] = uniform(g, 1e4, 3e4, n, 2)
    a[:, 3] = uniform(g, 0, math.pi, n)
    return a


def ctf_values(a, box, px, iCol, iRow, scale=1.0):
    """Contrast transfer at the pixels for the attributes a (n, 7), defocus times `scale`."""
    i = torch.as_tensor(iCol, device=DEV, dtype=F64)
    j = torch.as_tensor(iRow, device=DEV, dtype=F64)
    V, dU, dV, th, Cs, A = (a[:, k, None] for k in range(6))
    lam = 12.2643247 / torch.sqrt(V * (1 + V * 0.978466e-6))
    u2 = (i * i + j * j) / (px * box) ** 2
    d = -0.5 * scale * (dU + dV + (dU - dV) * torch.cos(2 * (torch.atan2(j, i) - th)))
    ki = math.pi * lam * d * u2 + 0.5 * math.pi * Cs * lam ** 3 * u2 * u2
    return -torch.sqrt(1 - A * A) * torch.sin(ki) + A * torch.cos(ki)


def phases(t, box, iCol, iRow, dtype=F64):
    """exp(-2 pi i k.t / box) for shifts t (..., 2)."""
    i = torch.as_tensor(iCol, device=DEV, dtype=F64)
    j = torch.as_tensor(iRow, device=DEV, dtype=F64)
    return torch.exp(-2j * math.pi * (t[..., :1] * i + t[..., 1:] * j) / box)


def particles(g, bl, n, box, iCol, iRow, rU, snr, shift):
    """n particle images at the pixels, with their poses: white noise at `snr`."""
    px = 1.1 * 256 / box
    q, t = haar(g, n), uniform(g, -shift, shift, n, 2)
    ctf = ctf_values(ctf_attributes(g, n), box, px, iCol, iRow)
    x = slices(bl, matrix(q), box, iCol, iRow, rU) * ctf
    for s in range(0, n, 256):
        x[s:s + 256] *= phases(t[s:s + 256], box, iCol, iRow).to(C64)
    s2 = float(x.abs().double().square().mean()) / snr / 2
    K = len(iCol)
    for s in range(0, n, 256):
        m = len(x[s:s + 256])
        x[s:s + 256] += math.sqrt(s2) * torch.complex(normal(g, m, K, dtype=F32),
                                                      normal(g, m, K, dtype=F32))
    sig = torch.full((n, K), -0.5 / s2, device=DEV, dtype=F32)
    return dict(dat=x.to(C64).contiguous(), ctf=ctf.float().contiguous(), sig=sig, q=q, t=t, px=px)


def network_images(g, bl, q, box):
    """64 x 64 images of the map at rotations q, noisy, centred, normalised."""
    k = 32
    j = np.concatenate([np.arange(0, k), np.arange(-k, 0)])
    jj, ii = np.meshgrid(j, np.arange(0, k + 1), indexing="ij")
    F = slices(bl, matrix(q), box, ii.ravel(), jj.ravel(), k).reshape(-1, 64, 33)
    x = torch.fft.fftshift(torch.fft.irfft2(F, s=(64, 64)), dim=(-2, -1)).float()
    x = x / x.std(dim=(-2, -1), keepdim=True)
    x = x + 3.0 * normal(g, *x.shape, dtype=F32)
    x = x - x.mean(dim=(-2, -1), keepdim=True)
    return (x / x.std(dim=(-2, -1), keepdim=True)).contiguous()


def network_params(g):
    """He-initialised parameters of the pose network, layer after layer: weights, then biases."""
    parts = []
    for cin, cout in ((9, 32), (288, 32), (288, 64), (576, 64), (576, 128), (1152, 128), (8192, 256),
                      (256, 68)):
        parts += [normal(g, cout * cin, dtype=F32) * math.sqrt(2.0 / cin),
                  0.01 * normal(g, cout, dtype=F32)]
    return torch.cat(parts)


def permutations(g, n, m):
    return torch.argsort(torch.rand(n, m, generator=g, device=DEV), dim=1).to(I32).contiguous()


def precision(c):
    return tg3.SCORE_BF16X3 if c["prec"] == "bf16" else tg3.SCORE_FP32


def empty(dtype, *shape):
    return torch.empty(*shape, device=DEV, dtype=dtype)


def inputs(c, seed):
    """A case's inputs, from the seed alone."""
    g = generator(seed)
    path = c["path"]
    x = {}
    if path in ("particle", "local", "global", "insert", "learned"):
        x["iCol"], x["iRow"] = pixels(c["rU"])
    if path in ("particle", "local"):
        box, nP, nR, nT = c["box"], c.get("nP", 1), c["nR"], c["nT"]
        bl = blobs(g, 120, box)
        x["vol"] = volume(bl, box)
        p = particles(g, bl, nP, box, x["iCol"], x["iRow"], c["rU"], 0.04, 5.0)
        x.update(p)
        x["quat"] = near(g, p["q"], 0.07, nR).contiguous()
        x["trans"] = (p["t"][:, None] + 2.0 * normal(g, nP, nT, 2)).contiguous()
        x["pwR"] = torch.full((nP, nR), 1.0 / nR, device=DEV, dtype=F64)
        x["pwT"] = torch.full((nP, nT), 1.0 / nT, device=DEV, dtype=F64)
        x["pwC"] = torch.ones(nP, device=DEV, dtype=F64)
        nD = c.get("nD", 1)
        if nD > 1:
            a = ctf_attributes(g, nP)
            f = torch.linspace(0.9, 1.1, nD)
            x["ctfD"] = torch.stack([ctf_values(a, box, p["px"], x["iCol"], x["iRow"], float(d))
                                     for d in f], 1).float().contiguous()
            x["pwD"] = torch.full((nP, nD), 1.0 / nD, device=DEV, dtype=F64)
        for k, m in (("R", nR), ("T", nT)):
            x["perm" + k] = permutations(g, nP, m)
            x["u0" + k] = uniform(g, 0, 1.0 / m, nP)
        x["peakR"] = torch.full((nP,), float("nan"), device=DEV, dtype=F64)
        x["peakT"] = torch.zeros(nP, device=DEV, dtype=F64)
    elif path == "ragged":
        box, nP, nC = c["box"], c["nP"], c["nC"]
        cls = torch.arange(nP) % nC
        sizes, gs = {}, generator(nP)         # the set sizes belong to the case, not to the seed
        for k in ("nR", "nT"):
            lo, hi = math.log(c[k + "_lo"]), math.log(c[k + "_hi"])
            sizes[k] = torch.exp(uniform(gs, lo, hi, nP)).round().int().cpu().numpy()
        cut = [int(c["rU"] * f) for f in (1.0, 0.75, 0.58, 0.42)[:nC]]
        x.update(cls=cls.int().numpy(), nR=sizes["nR"], nT=sizes["nT"], cut=cut, vols=[], pix=[])
        rows = {}
        for k in range(nC):
            bl = blobs(g, 120, box)
            x["vols"].append(volume(bl, box))
            x["pix"].append(pixels(cut[k]))
            p = particles(g, bl, int((cls == k).sum()), box, *x["pix"][k], cut[k], 0.04, 5.0)
            for n, l in enumerate(torch.nonzero(cls == k).ravel().tolist()):
                rows[l] = {"dat": p["dat"][n], "ctf": p["ctf"][n], "sig": p["sig"][n],
                           "quat": near(g, p["q"][n:n + 1], 0.07, int(sizes["nR"][l]))[0],
                           "trans": p["t"][n] + 2.0 * normal(g, int(sizes["nT"][l]), 2)}
        cat = {k: torch.cat([rows[l][k].reshape(-1) for l in range(nP)]).contiguous()
               for k in ("dat", "ctf", "sig", "quat", "trans")}
        for k, ax in (("nR", "R"), ("nT", "T")):
            cat["pw" + ax] = torch.cat([torch.full((int(m),), 1.0 / m, device=DEV, dtype=F64)
                                        for m in sizes[k]])
            cat["perm" + ax] = torch.cat([permutations(g, 1, int(m))[0] for m in sizes[k]])
            cat["u0" + ax] = uniform(g, 0, 1, nP) / torch.as_tensor(sizes[k], device=DEV)
        cat["pwC"] = torch.ones(nP, device=DEV, dtype=F64)
        cat["peakR"] = torch.full((nP,), float("nan"), device=DEV, dtype=F64)
        cat["peakT"] = torch.zeros(nP, device=DEV, dtype=F64)
        x["inp"] = cat
    elif path == "global":
        bl = blobs(g, 40, c["box"])
        x["vol"] = volume(bl, c["box"])
        x.update(particles(g, bl, c["nImg"], c["box"], x["iCol"], x["iRow"], c["rU"], 0.05,
                           float(c["half"])))
        x["quat"] = rotation_grid(c["nDir"], c["nPsi"])
        x["mats"] = matrix(x["quat"]).reshape(-1, 9).contiguous()
        x["grid"] = shift_grid(c["half"])
    elif path == "class2d":
        box, nK, n = c["box"], c["nK"], c["nImg"]
        x["iCol"], x["iRow"] = pixels(c["rU"])
        v = PF * box
        f = torch.fft.fftfreq(v, device=DEV, dtype=F64)
        fx = torch.arange(v // 2 + 1, device=DEV, dtype=F64) / v
        psi = uniform(g, 0, 2 * math.pi, n)
        z = torch.zeros_like(psi)
        q = torch.stack([torch.cos(psi / 2), z, z, torch.sin(psi / 2)], -1)
        px = 1.1 * 256 / box
        ctf = ctf_values(ctf_attributes(g, n), box, px, x["iCol"], x["iRow"])
        dat = torch.empty(n, len(x["iCol"]), device=DEV, dtype=C64)
        x["imgs"] = torch.empty(nK, v, v // 2 + 1, device=DEV, dtype=C64)
        for k in range(nK):
            bl = blobs(g, 80, box)
            w = bl[0] * (2 * math.pi * bl[1] ** 2) ** 1.5
            x["imgs"][k] = torch.matmul((axis_factors(bl[1], bl[2][:, 1], f) * w[:, None]).T,
                                        axis_factors(bl[1], bl[2][:, 0], fx)).to(C64)
            dat[k::nK] = slices(bl, matrix(q[k::nK]), box, x["iCol"], x["iRow"], c["rU"])
        t = uniform(g, -c["half"], c["half"], n, 2)
        dat = dat * ctf * phases(t, box, x["iCol"], x["iRow"])
        s2 = float(dat.abs().square().mean()) / 0.1 / 2
        dat = dat + math.sqrt(s2) * torch.complex(normal(g, *dat.shape), normal(g, *dat.shape))
        x.update(dat=dat.to(C64).contiguous(), ctf=ctf.float().contiguous(),
                 sig=torch.full(dat.shape, -0.5 / s2, device=DEV, dtype=F32))
        a = torch.arange(c["nR"], device=DEV, dtype=F64) * (2 * math.pi / c["nR"])
        x["rot"] = torch.stack([torch.cos(a), torch.sin(a)], 1).contiguous()
        x["grid"] = shift_grid(c["half"])
    elif path == "learned":
        nP, nC, box = c["nP"], c["nC"], c["box"]
        cls = torch.arange(nP, device=DEV) % nC
        K = len(x["iCol"])
        x.update(cls=cls.int(), vols=[], images=empty(F32, nP, 64, 64), dat=empty(C64, nP, K),
                 ctf=empty(F32, nP, K), sig=empty(F32, nP, K))
        for k in range(nC):
            bl = blobs(g, 120, box)
            x["vols"].append(volume(bl, box))
            sel = torch.nonzero(cls == k).ravel()
            p = particles(g, bl, len(sel), box, x["iCol"], x["iRow"], c["rU"], 0.04, 2.0)
            x["images"][sel] = network_images(g, bl, p["q"], box)
            for name in ("dat", "ctf", "sig"):
                x[name][sel] = p[name]
        x["params"] = network_params(g)
        x["quat"] = rotation_grid(c["nDir"], c["nPsi"]).contiguous()
        x["grid"] = shift_grid(c["half"])
    elif path == "train":
        bl = blobs(g, 120, 128)
        q = haar(g, c["n"])
        x["img"] = network_images(g, bl, q, 128)
        x["ref"] = network_images(g, bl, q, 128)
        x["t"] = uniform(g, -3, 3, c["n"], 2).contiguous()
        x["params"] = network_params(g)
    elif path == "insert":
        bl = blobs(g, 60, c["box"])
        x.update(particles(g, bl, c["nP"], c["box"], x["iCol"], x["iRow"], c["rU"], 0.05, 5.0))
        x["off"] = (0.5 * normal(g, c["nP"], 2)).contiguous()
        x["w"] = uniform(g, 0.5, 1.0, c["nP"]).float()
    elif path == "reconstruct":
        v = PF * c["box"]
        r = torch.sqrt(half_grid(v))
        x["T"] = ((40 + float(uniform(g, 0, 20, 1))) * torch.exp(-r / (0.4 * v)) + 0.5).float()
        del r
        F = volume(blobs(g, 80, c["box"]), c["box"])
        x["F"] = (F * x["T"]).contiguous()
        n = c["box"] // 2 + 1
        x["fsc"] = (1.05 - torch.arange(n, device=DEV, dtype=F64) / (n - 1)).clamp(0, 1)
    elif path == "prepare":
        n, N = c["n"], c["box"]
        a = torch.arange(N, device=DEV, dtype=F32) - N // 2
        mid = 0.1 * N * normal(g, n, 2, 1, dtype=F32)
        w = 0.1 * N * (0.7 + torch.rand(n, 1, generator=g, device=DEV))
        gx, gy = (torch.exp(-0.5 * ((a[None] - mid[:, k]) / w) ** 2) for k in (0, 1))
        img = normal(g, n, N, N, dtype=F32)
        img += gy[:, :, None] * gx[:, None, :]
        x["img"] = (img.mul_(3.0).add_(10.0)).contiguous()
        x["iCol"], x["iRow"] = pixels(c["rU"])
    return x


def half_grid(v):
    """Squared radii of the padded half grid [z][y][x], float32."""
    f = torch.fft.fftfreq(v, 1.0 / v, device=DEV, dtype=F32) ** 2
    h = torch.arange(v // 2 + 1, device=DEV, dtype=F32) ** 2
    return f[:, None, None] + f[None, :, None] + h[None, None, :]


# -------------------------------------------------------------------------- a user's program --
def prepare(case, seed):
    c = case
    x = inputs(c, seed)
    path = c["path"]
    if path == "particle":
        host = {k: np.ascontiguousarray(x[k][0].cpu().numpy()) for k in
                ("dat", "ctf", "sig", "quat", "trans", "pwR", "pwT")}
        vol = x["vol"].cpu().numpy()
        h = ctypes.c_void_p()
        tg3.check(tg3.lib().tg3_volume_create(ctypes.byref(h), tg3.ptr(vol), PF * c["box"], PF))
        return dict(c=c, vol=VolumeHandle(h), iCol=x["iCol"], iRow=x["iRow"], **host,
                    wC=np.zeros(1, np.float32), wR=np.zeros(c["nR"], np.float32),
                    wT=np.zeros(c["nT"], np.float32), base=np.zeros(1, np.float32))
    if path == "train":
        net = tg3.Cnn(0, seed=1)
        net.set_params(x["params"].cpu().numpy())
        return dict(c=c, net=net, img=x["img"], ref=x["ref"], t=x["t"],
                    out=[empty(F32, c["n"], tg3.Cnn.N_OUT) for _ in range(4)])
    ctx = tg3.Context(0)
    s = dict(c=c, ctx=ctx)
    if path == "local":
        nP, nR, nT, nD = c["nP"], c["nR"], c["nT"], c["nD"]
        ctx.set_volume(0, x.pop("vol"), PF)
        ctx.set_pixels(x["iCol"], x["iRow"], c["box"])
        s.update(x, o=dict(wC=empty(F64, nP), wR=empty(F64, nP, nR), wT=empty(F64, nP, nT),
                           base=empty(F64, nP), srcR=empty(I32, nP, nR), wOutR=empty(F64, nP, nR),
                           topR=empty(I32, nP), srcT=empty(I32, nP, nT), wOutT=empty(F64, nP, nT),
                           topT=empty(I32, nP)))
        if nD > 1:
            s["o"]["wD"] = empty(F64, nP, nD)
    elif path == "ragged":
        for k in range(c["nC"]):
            ctx.set_volume(k, x["vols"][k], PF)
            ctx.set_pixels_slot(k, *x["pix"][k], c["box"])
        nP, R, T = c["nP"], int(x["nR"].sum()), int(x["nT"].sum())
        o = dict(wC=empty(F64, nP), base=empty(F64, nP), wR=empty(F64, R), wT=empty(F64, T),
                 srcR=empty(I32, R), wOutR=empty(F64, R), srcT=empty(I32, T), wOutT=empty(F64, T),
                 topR=empty(I32, nP), topT=empty(I32, nP))
        s.update(o=o, plan=tg3.RaggedPlan(ctx, x["cls"], x["nR"], x["nT"], x["inp"], o,
                                          precision(c), budget=6 << 30, graph=True))
    elif path == "global":
        nR, nT = c["nDir"] * c["nPsi"], len(x["grid"])
        ctx.set_volume(0, x.pop("vol"), PF)
        ctx.set_pixels(x["iCol"], x["iRow"], c["box"])
        n = c["nImg"]
        s.update(x, nR=nR, nT=nT, pR=torch.full((nR,), 1.0 / nR, device=DEV, dtype=F64),
                 pT=torch.full((nT,), 1.0 / nT, device=DEV, dtype=F64),
                 o=dict(wC=empty(F64, n), wR=empty(F64, n, nR), wT=empty(F64, n, nT),
                        base=empty(F64, n)))
    elif path == "class2d":
        ctx.set_pixels(x["iCol"], x["iRow"], c["box"])
        n, nK, nR, nT = c["nImg"], c["nK"], c["nR"], len(x["grid"])
        s.update(x, nT=nT, pR=torch.full((nR,), 1.0 / nR, device=DEV, dtype=F64),
                 pT=torch.full((nT,), 1.0 / nT, device=DEV, dtype=F64),
                 o=dict(wC=empty(F32, n, nK), wR=empty(F32, n, nK, nR), wT=empty(F32, n, nK, nT),
                        base=empty(F32, n)))
    elif path == "learned":
        net = tg3.Cnn(0, seed=1)
        net.set_params(x["params"].cpu().numpy())
        nB, nP, nRot, nT = len(x["quat"]), c["nP"], c["nRot"], c["nTrans"]
        mats = matrix(x["quat"]).reshape(-1, 9).contiguous()
        for k in range(c["nC"]):
            ctx.set_volume(k, x["vols"][k], PF)
        ctx.set_pixels(x["iCol"], x["iRow"], c["box"])
        for k in range(c["nC"]):
            refs, out, z = empty(F32, nB, 64, 64), empty(F32, nB, 68), empty(F32, nB, 64)
            ctx.render_references(k, mats, nB, 64, refs)
            ctx.sync()
            net.infer(refs, out)
            net.embed(out, z)
            torch.cuda.synchronize()
            ctx.set_bank(k, x["quat"], nB)
            ctx.set_references(k, z)
        s.update({k: x[k] for k in ("images", "dat", "ctf", "sig", "cls", "grid")}, net=net,
                 peak=-math.inf,
                 o=dict(bestQuat=empty(F64, nP, 4), bestTrans=empty(F64, nP, 2),
                        baseL=empty(F64, nP), peak=empty(F32, nP), fellBack=empty(I32, nP),
                        propIdx=empty(I32, nP, nRot), propWR=empty(F64, nP, nRot),
                        propWT=empty(F64, nP, nT), propBase=empty(F64, nP)))
        # the confidence threshold that sends the wanted share of particles to the global search,
        # half way between two particles' values
        run_learned(s)
        p = torch.sort(s["o"]["peak"].double()).values
        k = min(nP - 1, max(1, int(round(c["fall"] * nP))))
        s["peak"] = float(0.5 * (p[k - 1] + p[k]))
    elif path == "insert":
        ctx.set_pixels(x["iCol"], x["iRow"], c["box"])
        v = PF * c["box"]
        s.update(x, F=empty(C64, v, v, v // 2 + 1), T=empty(F32, v, v, v // 2 + 1),
                 O=empty(F64, 3), count=empty(I32, 1),
                 stream=torch.cuda.ExternalStream(ctx.stream))
    elif path == "reconstruct":
        ctx.insert_begin(PF * c["box"], PF)
        N = c["box"]
        s.update(x, out=empty(F32, N, N, N))
    elif path == "prepare":
        ctx.set_pixels(x["iCol"], x["iRow"], c["box"])
        s.update(x, dat=empty(C64, c["n"], len(x["iCol"])), stats=empty(F32, c["n"], 3))
    ctx.sync()
    torch.cuda.synchronize()
    return s


class VolumeHandle:
    """A tg3_volume, destroyed with this object."""

    def __init__(self, h):
        self.h = h

    def __del__(self):
        tg3.lib().tg3_volume_destroy(self.h)


def run_learned(s):
    c = s["c"]
    s["ctx"].learned_expect(s["net"], s["images"], s["dat"], s["ctf"], s["sig"], s["cls"], c["nRot"],
                            c["nTrans"], 5, s["grid"], s["peak"], precision(c), s["o"])
    return s["o"]


def run(state):
    s, c = state, state["c"]
    path = c["path"]
    if path == "particle":
        p = tg3.ptr
        tg3.check(tg3.lib().tg3_ExpectLocal3D(
            s["vol"].h, p(s["dat"]), p(s["ctf"]), p(s["sig"]), p(s["iCol"]), p(s["iRow"]),
            len(s["iCol"]), c["box"], p(s["quat"]), c["nR"], p(s["trans"]), c["nT"], p(s["pwR"]),
            p(s["pwT"]), 1.0, p(s["wC"]), p(s["wR"]), p(s["wT"]), None, p(s["base"])))
        return dict(wC=s["wC"], wR=s["wR"], wT=s["wT"], base=s["base"])
    if path == "train":
        net, (oP, oR, dP, dR) = s["net"], s["out"]
        net.forward(s["img"], oP)
        net.forward(s["ref"], oR)
        net.zero_grads()
        loss = net.contrastive(oP, oR, s["t"], 0.1, dP, dR)
        net.backward(s["img"], dP)
        net.backward(s["ref"], dR)
        return dict(outP=oP, outR=oR, loss=loss, dP=dP, dR=dR, grads=net.grads())
    ctx = s["ctx"]
    if path == "local":
        nP, nR, nT, o = c["nP"], c["nR"], c["nT"], s["o"]
        if c["nD"] > 1:
            ctx.local_phase_ctf(nP, nR, nT, c["nD"], s["dat"], s["ctfD"], s["sig"], s["quat"],
                                s["trans"], s["pwR"], s["pwT"], s["pwD"], s["pwC"], None, o["wC"],
                                o["wR"], o["wT"], o["wD"], o["base"], None, precision(c))
        else:
            ctx.local_phase(nP, nR, nT, s["dat"], s["ctf"], s["sig"], s["quat"], s["trans"],
                            s["pwR"], s["pwT"], s["pwC"], None, o["wC"], o["wR"], o["wT"],
                            o["base"], None, precision(c))
        for k, n in (("R", nR), ("T", nT)):
            ctx.resample(nP, n, o["w" + k], s["pw" + k], s["perm" + k], s["u0" + k], s["peak" + k],
                         n, o["src" + k], o["wOut" + k], o["top" + k])
        return o
    if path == "ragged":
        s["plan"].run()
        return s["o"]
    if path == "global":
        o = s["o"]
        ctx.global_scan(0, c["nImg"], s["nR"], s["nT"], s["dat"], s["ctf"], s["sig"], s["mats"],
                        s["grid"], s["pR"], s["pT"], o["wC"], o["wR"], o["wT"], o["base"], None,
                        precision(c))
        return o
    if path == "class2d":
        o = s["o"]
        ctx.global_scan2d_classes(s["imgs"], PF, c["nImg"], c["nR"], s["nT"], s["dat"], s["ctf"],
                                  s["sig"], s["rot"], s["grid"], s["pR"], s["pT"], o["wC"],
                                  o["wR"], o["wT"], o["base"], precision(c))
        return o
    if path == "learned":
        return run_learned(s)
    if path == "insert":
        ctx.insert_begin(PF * c["box"], PF)
        with torch.cuda.stream(s["stream"]):
            s["O"].zero_()
            s["count"].zero_()
        ctx.insert(c["nP"], s["dat"], s["ctf"], s["q"], s["t"], s["off"], s["w"], kernel_of(c),
                   s["O"], s["count"])
        ctx.insert_read(s["F"], s["T"])
        return dict(F=s["F"], T=s["T"], O=s["O"], count=s["count"])
    if path == "reconstruct":
        ctx.insert_load(s["F"], s["T"])
        rounds = ctx.reconstruct(s["out"], c["rU"], fsc=s["fsc"], join_half=True,
                                 grid_corr=c["grid"], kernel=kernel_of(c))
        return dict(map=s["out"], rounds=rounds)
    ctx.prepare_images(s["img"], 0.4 * c["box"], s["dat"], mask=True, std_n=0.0, stats=s["stats"])
    return dict(dat=s["dat"], stats=s["stats"])


def kernel_of(c):
    return tg3.KERNEL_MKB if c["kernel"] == "mkb" else tg3.KERNEL_TRILINEAR


# ------------------------------------------------------------- what a pass cannot do without --
def work(case):
    c = case
    path = c["path"]
    if path == "train":
        # 69.4 M multiply-adds an image forward, twice that backward, for particle and reference
        macs = 69.4e6 * 3 * 2 * c["n"]
        return dict(bytes=2 * c["n"] * (64 * 64 * 4 + 68 * 8) + 2 * 4 * 2.4e6, flops=2 * macs)
    box = c["box"]
    if path == "reconstruct":
        nh = (PF * box) ** 2 * (box + 1)
        # F and T read and the map written: the balancing works on arrays of its own
        return dict(bytes=12 * nh + 4 * box ** 3,
                    flops=(20 if c["grid"] else 1) * 5.0 * nh * math.log2((PF * box) ** 3) * 2)
    if path == "ragged":
        K = np.array([n_pixels(int(c["rU"] * f)) for f in (1.0, 0.75, 0.58, 0.42)[:c["nC"]]])
        mean = lambda k: (c[k + "_hi"] - c[k + "_lo"]) / math.log(c[k + "_hi"] / c[k + "_lo"])  # noqa: E731
        nR, nT, n = mean("nR"), mean("nT"), c["nP"] / c["nC"]
        return dict(bytes=float(n * (16 * K.sum() + c["nC"] * (60 * nR + 44 * nT))),
                    flops=float(n * K.sum() * nR * (48 + 4 * nT)))
    K = n_pixels(c["rU"])
    ball = min((PF * box) ** 2 * (box + 1), 2.1 * (PF * c["rU"]) ** 3) * 8
    if path in ("particle", "local"):
        nP, nR, nT, nD = c.get("nP", 1), c["nR"], c["nT"], c.get("nD", 1)
        return dict(bytes=nP * (K * (12 + 4 * nD) + 72 * nR + 56 * nT) + min(ball, 64.0 * K * nR * nP),
                    flops=float(nP) * nR * K * (48 + 4 * nT * nD))
    if path == "global":
        nR, nT = c["nDir"] * c["nPsi"], (2 * c["half"] + 1) ** 2
        return dict(bytes=c["nImg"] * (16 * K + 8 * (nR + nT)) + ball,
                    flops=4.0 * K * nR * (nT + 1) * c["nImg"])
    if path == "class2d":
        nT = (2 * c["half"] + 1) ** 2
        return dict(bytes=c["nImg"] * (16 * K + 4 * c["nK"] * (c["nR"] + nT))
                    + c["nK"] * 8.0 * PF * box * (box + 1),
                    flops=4.0 * K * c["nK"] * c["nR"] * (nT + 1) * c["nImg"])
    if path == "learned":
        nB, nTg = c["nDir"] * c["nPsi"], (2 * c["half"] + 1) ** 2
        hyp = c["nRot"] * c["nTrans"] + c["fall"] * nB * nTg
        return dict(bytes=c["nP"] * (16 * K + 4 * 4096 + 16 * c["nRot"]) + c["nC"] * nB * 8 * K,
                    flops=c["nP"] * (4.0 * K * hyp + 1.39e8 + 128 * nB))
    if path == "insert":
        nh = (PF * box) ** 2 * (box + 1)
        per = 28.7 if c["kernel"] == "mkb" else 8
        return dict(bytes=16.0 * K * c["nP"] + 12 * nh, flops=c["nP"] * K * (20 + 6 * per))
    return dict(bytes=c["n"] * (4.0 * box * box + 8 * K),
                flops=c["n"] * (2.5 * box * box * math.log2(box * box) + 10 * box * box))


# -------------------------------------------------------------------- the same in 64 bits --
def sample(vol, R, iCol, iRow):
    """Trilinear samples of the half volume vol (complex64) at R (n, 3, 3): (n, K) complex128."""
    v, nx = vol.shape[0], vol.shape[2]
    flat = vol.reshape(-1)
    a = torch.as_tensor(iCol, device=DEV, dtype=F64) * PF
    b = torch.as_tensor(iRow, device=DEV, dtype=F64) * PF
    out = torch.empty(len(R), len(iCol), device=DEV, dtype=C128)
    step = max(1, 4_000_000 // len(iCol))
    for s in range(0, len(R), step):
        r = R[s:s + step]
        p = [r[:, k, :1] * a + r[:, k, 1:2] * b for k in range(3)]
        neg = p[0] < 0
        p = [torch.where(neg, -t, t) for t in p]
        lo = [torch.floor(t) for t in p]
        fr = [t - l for t, l in zip(p, lo)]
        lo = [l.long() for l in lo]
        acc = torch.zeros(len(r), len(iCol), device=DEV, dtype=C128)
        for dz in (0, 1):
            for dy in (0, 1):
                row = ((lo[2] + dz) % v * v + (lo[1] + dy) % v) * nx
                wzy = (fr[2] if dz else 1 - fr[2]) * (fr[1] if dy else 1 - fr[1])
                for dx in (0, 1):
                    acc += flat[row + lo[0] + dx] * (wzy * (fr[0] if dx else 1 - fr[0]))
        out[s:s + step] = torch.where(neg, acc.conj(), acc)
    return out


def score(P, dat, ctf, sig, S):
    """Log-likelihoods (R, T) of one particle: projections P (R, K), phases S (T, K)."""
    X, c, w = dat.to(C128), ctf.double(), sig.double()
    const = (w * X.abs().square()).sum()
    nrm = P.abs().square() @ (w * c * c)
    A = w * c * X * S.conj()
    cross = torch.view_as_real(P).reshape(len(P), -1) @ torch.view_as_real(A).reshape(len(A), -1).T
    return const + nrm[:, None] - 2 * cross


def marginals(L, pR, pT):
    m = L.max()
    e = torch.exp(L - m)
    r = e @ pT
    return r @ pR, r, pR @ e, m


def f32_shifts(t):
    return t.float().double()


def exact(case, seed):
    c = case
    path = c["path"]
    if path == "learned":
        return None                     # the network's roundings decide the proposals
    x = inputs(c, seed)
    if path in ("particle", "local"):
        o = dict(wC=[], wR=[], wT=[], base=[], wD=[])
        for l in range(c.get("nP", 1)):
            P = sample(x["vol"], matrix(x["quat"][l]), x["iCol"], x["iRow"])
            S = phases(f32_shifts(x["trans"][l]), c["box"], x["iCol"], x["iRow"])
            pR, pT = x["pwR"][l], x["pwT"][l]
            if c.get("nD", 1) == 1:
                got = marginals(score(P, x["dat"][l], x["ctf"][l], x["sig"][l], S), pR, pT)
            else:
                part = [marginals(score(P, x["dat"][l], x["ctfD"][l, d], x["sig"][l], S), pR, pT)
                        for d in range(c["nD"])]
                m = max(p[3] for p in part)
                e = [torch.exp(p[3] - m) for p in part]
                w = [float(t) for t in x["pwD"][l]]
                got = [sum(w[d] * e[d] * part[d][k] for d in range(c["nD"])) for k in range(3)] + [m]
                o["wD"].append(torch.stack([e[d] * part[d][0] for d in range(c["nD"])]))
            for k, v in zip(("wC", "wR", "wT", "base"), got):
                o[k].append(v)
        o = {k: torch.stack(v) for k, v in o.items() if v}
        if path == "particle":
            return dict(wC=o["wC"], wR=o["wR"][0], wT=o["wT"][0], base=o["base"])
        return dict(o, srcR=None, wOutR=None, topR=None, srcT=None, wOutT=None, topT=None)
    if path == "ragged":
        o = dict(wC=[], wR=[], wT=[], base=[])
        at = dict(K=0, R=0, T=0)
        i = x["inp"]
        for l in range(c["nP"]):
            k = int(x["cls"][l])
            iCol, iRow = x["pix"][k]
            K, nR, nT = len(iCol), int(x["nR"][l]), int(x["nT"][l])
            a, r, t = at["K"], at["R"], at["T"]
            q = i["quat"].reshape(-1, 4)[r:r + nR]
            S = phases(f32_shifts(i["trans"].reshape(-1, 2)[t:t + nT]), c["box"], iCol, iRow)
            L = torch.cat([score(sample(x["vols"][k], matrix(q[b:b + 1024]), iCol, iRow),
                                 i["dat"][a:a + K], i["ctf"][a:a + K], i["sig"][a:a + K], S)
                           for b in range(0, nR, 1024)])
            for n, v in zip(("wC", "wR", "wT", "base"),
                            marginals(L, i["pwR"][r:r + nR], i["pwT"][t:t + nT])):
                o[n].append(v)
            at = dict(K=a + K, R=r + nR, T=t + nT)
        return dict(wC=torch.stack(o["wC"]), base=torch.stack(o["base"]), wR=torch.cat(o["wR"]),
                    wT=torch.cat(o["wT"]), srcR=None, wOutR=None, srcT=None, wOutT=None, topR=None,
                    topT=None)
    if path in ("global", "class2d"):
        S = phases(f32_shifts(x["grid"]), c["box"], x["iCol"], x["iRow"])
        if path == "global":
            P = [sample(x["vol"], x["mats"].reshape(-1, 3, 3), x["iCol"], x["iRow"])]
        else:
            P = [sample_2d(img, x["rot"].float().double(), x["iCol"], x["iRow"]) for img in x["imgs"]]
        n, nR, nT = c["nImg"], len(P[0]), len(S)
        wC, wR, wT = (empty(F64, n, len(P), *k) for k in ((), (nR,), (nT,)))
        base = empty(F64, n)
        for l in range(n):
            L = [score(p, x["dat"][l], x["ctf"][l], x["sig"][l], S) for p in P]
            m = torch.stack([t.max() for t in L]).max()
            for k, t in enumerate(L):
                e = torch.exp(t - m)
                wR[l, k], wT[l, k], wC[l, k] = e.mean(1), e.mean(0), e.mean()
            base[l] = m
        if path == "global":
            wC, wR, wT = wC[:, 0], wR[:, 0], wT[:, 0]
        return dict(wC=wC, wR=wR, wT=wT, base=base)
    if path == "train":
        return exact_train(c, x)
    if path == "insert":
        return exact_insert(c, x)
    if path == "reconstruct":
        return exact_reconstruct(c, x)
    return exact_prepare(c, x)


def sample_2d(img, rot, iCol, iRow):
    """Bilinear samples of one class image at in-plane rotations rot (n, 2) = (cos, sin)."""
    v, nx = img.shape
    a = torch.as_tensor(iCol, device=DEV, dtype=F64) * PF
    b = torch.as_tensor(iRow, device=DEV, dtype=F64) * PF
    cs, sn = rot[:, :1], rot[:, 1:]
    px, py = cs * a - sn * b, sn * a + cs * b
    neg = px < 0
    px, py = torch.where(neg, -px, px), torch.where(neg, -py, py)
    x0, y0 = torch.floor(px), torch.floor(py)
    fx, fy = px - x0, py - y0
    x0, y0 = x0.long(), y0.long()
    acc = torch.zeros(px.shape, device=DEV, dtype=C128)
    for dy in (0, 1):
        for dx in (0, 1):
            acc += img.reshape(-1)[(y0 + dy) % v * nx + x0 + dx] * (
                (fy if dy else 1 - fy) * (fx if dx else 1 - fx))
    return torch.where(neg, acc.conj(), acc)


def exact_train(c, x):
    shapes = ((32, 1, 3, 3), (32, 32, 3, 3), (64, 32, 3, 3), (64, 64, 3, 3), (128, 64, 3, 3),
              (128, 128, 3, 3), (256, 8192), (68, 256))
    ws, bs, at = [], [], 0
    for sh in shapes:
        n = math.prod(sh)
        # weights enter the products as bf16, their gradients go to the 32-bit masters
        ws.append(x["params"][at:at + n].bfloat16().double().reshape(sh).requires_grad_())
        bs.append(x["params"][at + n:at + n + sh[0]].double().requires_grad_())
        at += n + sh[0]

    def forward(img):
        h = img.double()[:, None]
        for k in range(6):
            # a convolution as one product: 64-bit convolutions of the library are slow
            s = 2 if k % 2 else 1
            u = torch.nn.functional.unfold(h, 3, padding=1, stride=s)
            y = ws[k].reshape(len(ws[k]), -1) @ u + bs[k][:, None]
            h = torch.relu(y.reshape(len(img), len(ws[k]), h.shape[-1] // s, h.shape[-1] // s))
        h = torch.relu(h.reshape(len(img), -1) @ ws[6].T + bs[6])
        return h @ ws[7].T + bs[7]

    n = c["n"]
    grad = torch.zeros(at, device=DEV, dtype=F64)
    with torch.no_grad():
        outs = [torch.cat([forward(v[b:b + 32]) for b in range(0, n, 32)]) for v in (x["img"], x["ref"])]
    oP, oR = (o.detach().requires_grad_() for o in outs)
    u, v = (o[:, :64] / torch.sqrt(o[:, :64].square().sum(1, keepdim=True) + 1e-12)
            for o in (oP, oR))
    S = u @ v.T / 0.1
    d = x["t"] - oP[:, 64:66]
    lv = oP[:, 66:68]
    loss = (0.5 * (torch.logsumexp(S, 1) + torch.logsumexp(S, 0)) - S.diagonal()
            + 0.5 * (d * d * torch.exp(-lv) + lv).sum(1)).mean()
    dP, dR = torch.autograd.grad(loss, (oP, oR))
    for img, g in ((x["img"], dP), (x["ref"], dR)):
        for b in range(0, n, 32):
            p = [t for pair in zip(ws, bs) for t in pair]
            got = torch.autograd.grad(forward(img[b:b + 32]), p, g[b:b + 32])
            grad += torch.cat([t.reshape(-1) for t in got])
    return dict(outP=oP.detach(), outR=oR.detach(), loss=loss.detach(), dP=dP, dR=dR, grads=grad)


def exact_insert(c, x):
    box, v = c["box"], PF * c["box"]
    nx = v // 2 + 1
    F = torch.zeros(v * v * nx, 2, device=DEV, dtype=F64)
    T = torch.zeros(v * v * nx, device=DEV, dtype=F64)
    a = torch.as_tensor(x["iCol"], device=DEV, dtype=F64) * PF
    b = torch.as_tensor(x["iRow"], device=DEV, dtype=F64) * PF
    R, t = matrix(x["q"]), x["t"] - x["off"]
    step = max(1, 1_000_000 // len(a))
    i0a = torch.special.i0(torch.tensor(15.0, device=DEV, dtype=F64))

    def add(ijk, val, wt):
        neg = ijk[0] < 0
        i, j, k = (torch.where(neg, -p, p) for p in ijk)
        val = torch.where(neg, val.conj(), val)
        at = ((k % v) * v + j % v) * nx + i
        F.index_add_(0, at.reshape(-1), torch.view_as_real(val).reshape(-1, 2))
        T.index_add_(0, at.reshape(-1), wt.reshape(-1))

    for s in range(0, c["nP"], step):
        r = R[s:s + step]
        cf, w = x["ctf"][s:s + step].double(), x["w"][s:s + step].double()[:, None]
        val = x["dat"][s:s + step].to(C128) * phases(-t[s:s + step], box, x["iCol"], x["iRow"])
        val, wt = val * (cf * w), cf * cf * w
        p = [r[:, k, :1] * a + r[:, k, 1:2] * b for k in range(3)]
        if c["kernel"] == "trilinear":
            neg = p[0] < 0
            p = [torch.where(neg, -q, q) for q in p]
            val = torch.where(neg, val.conj(), val)
            lo = [torch.floor(q) for q in p]
            for e in range(8):
                d = (e & 1, e >> 1 & 1, e >> 2)
                k = math_prod((q - l) if n else (1 - (q - l)) for q, l, n in zip(p, lo, d))
                add([(l + n).long() for l, n in zip(lo, d)], val * k, wt * k)
            continue
        lo = [torch.ceil(q - 1.9) for q in p]
        for e in range(64):
            at = [l + n for l, n in zip(lo, (e & 3, e >> 2 & 3, e >> 4))]
            r2 = sum((q - n) ** 2 for q, n in zip(p, at))
            # the kernel is tabulated at 1e5 steps of r^2 over [0, (pf a)^2]
            h = (PF * 1.9) ** 2 / 1e5
            k2 = 1 - torch.round(r2 / h) * h / 1.9 ** 2
            k = torch.where(k2 >= 0, torch.special.i0(15.0 * torch.sqrt(k2.clamp_min(0))) / i0a, 0.0)
            on = k > 0
            add([n[on].long() for n in at], val[on] * k[on], wt[on] * k[on])
    z = torch.cat([t, torch.zeros_like(t[:, :1])], 1)
    O = -(R @ z[:, :, None])[:, :, 0].sum(0)
    return dict(F=torch.view_as_complex(F).reshape(v, v, nx), T=T.reshape(v, v, nx), O=O,
                count=torch.tensor([c["nP"]], dtype=I32))


def math_prod(vs):
    out = 1.0
    for v in vs:
        out = out * v
    return out


def mkb_real(r, a, alpha=15.0):
    """Real-space form of the order-0 modified Kaiser-Bessel kernel over its value at 0, inside
    2 pi a r <= alpha: I_1.5(v) / v^1.5 with I_1.5 in closed form."""
    def f(v):
        v = v.clamp_min(1e-3)
        return (torch.cosh(v) - torch.sinh(v) / v) / v ** 2
    v2 = alpha ** 2 - (2 * math.pi * a * r) ** 2
    inner = f(torch.sqrt(v2.clamp_min(0)))
    u = torch.sqrt((-v2).clamp_min(0)).clamp_min(1e-3)
    outer = (torch.sin(u) / u - torch.cos(u)) / u ** 2
    return torch.where(v2 >= 0, inner, outer) / f(torch.tensor(alpha, device=DEV, dtype=F64))


def exact_reconstruct(c, x):
    N, v = c["box"], PF * c["box"]
    q = half_grid(v).double()
    r2max = float((c["rU"] * PF) ** 2)
    inside = q < r2max
    T = x["T"].double()
    u = (torch.round(torch.sqrt(q)).long() // PF).clamp_max(10 ** 6)
    fsc = x["fsc"]
    f = torch.where(u < len(fsc), fsc[u.clamp_max(len(fsc) - 1)], 0.0).clamp(1e-3, 1 - 1e-3)
    f = torch.sqrt(2 * f / (1 + f))
    T = torch.where((q >= (5 * PF) ** 2) & inside, T / f, T).clamp_min(1e-25)
    del u, f, q
    W = inside.double()
    rounds = 0
    if c["grid"]:
        g = torch.fft.fftfreq(v, 1.0 / v, device=DEV, dtype=F64) ** 2
        r2 = (g[:, None, None] + g[None, :, None] + g[None, None, :]) / float(v) ** 2
        r2 = torch.round(r2 * 1e5) / 1e5
        k = mkb_real(torch.sqrt(r2), 1.9)
        del r2
        diff, still = math.inf, 0
        for m in range(30):
            C = torch.fft.rfftn(torch.fft.irfftn((T * W).to(C128), s=(v, v, v)) * k).abs()
            W = torch.where(inside, W / C.clamp_min(1e-6), W)
            last, diff = diff, float((C[inside] - 1).abs().max())
            still = still + 1 if diff > last * 0.95 else 0
            rounds = m + 1
            if diff < 1e-2 or (m >= 10 and still == 2):
                break
    else:
        W = torch.where(inside, 1 / T.clamp_min(1e-6), 0.0)
    pad = torch.fft.irfftn(torch.where(inside, x["F"].to(C128) * W, 0), s=(v, v, v))
    i = torch.arange(N, device=DEV) - N // 2
    out = pad[(i % v)[:, None, None], (i % v)[None, :, None], (i % v)[None, None, :]]
    a = i.double() ** 2
    r = torch.sqrt(a[:, None, None] + a[None, :, None] + a[None, None, :]) / v
    k = mkb_real(r, 1.9 * PF) if c["kernel"] == "mkb" else torch.sinc(r) ** 2
    return dict(map=out / k, rounds=rounds)


def exact_prepare(c, x):
    N, r = c["box"], 0.4 * c["box"]
    a = torch.arange(N, device=DEV, dtype=F64) - N // 2
    d2 = a[:, None] ** 2 + a[None, :] ** 2
    bg, d = d2 > r * r, torch.sqrt(d2)
    w = torch.where(d < r, 1.0, 1 - (0.5 - 0.5 * torch.cos((d - r) / 6.0 * math.pi)))
    w = torch.where(d > r + 6, 0.0, w)
    stats = empty(F64, c["n"], 3)
    n = int(bg.sum())
    for s in range(0, c["n"], 64):
        y = x["img"][s:s + 64].double()
        b = y[:, bg]
        m, sd = b.mean(1), b.std(1)
        sn = torch.sqrt((((b - m[:, None]) / sd[:, None]) ** 2).sum(1) / (n - 1))
        stats[s:s + 64] = torch.stack([m, sd, sn], 1)
    std_n = stats[:, 2].mean()
    rows = torch.as_tensor(x["iRow"], device=DEV).long() % N
    cols = torch.as_tensor(x["iCol"], device=DEV).long()
    dat = empty(C128, c["n"], len(cols))
    for s in range(0, c["n"], 64):
        y = (x["img"][s:s + 64].double() - stats[s:s + 64, 0, None, None]) / stats[s:s + 64, 1, None, None]
        F = torch.fft.rfft2(torch.fft.ifftshift(y * w / std_n, dim=(-2, -1)))
        dat[s:s + 64] = F[:, rows, cols]
    return dict(dat=dat, stats=stats)
