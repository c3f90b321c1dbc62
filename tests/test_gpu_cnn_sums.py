"""The network's FP32 convolutions at training batch sizes (the forms that a CTA
of 32 channels takes, shares of the batch in the weight gradient), the
rounding of the weight gradients' long sums, and images with a pixel that is
not a number, against float64 (torch's convolutions on the GPU).

Weights are -1, 0 and 1, inputs and output gradients whole numbers, so the forward pass and the
gradients with respect to the activations are exact in FP32 (the largest sums
are checked to stay below 2^24), and what differs in a weight's gradient is
the rounding of its own sum.  The sums' partials are chains of at most 64
products, which meet in FP64: an FP32 chain of m incoherent terms is off by
about 0.3 2^-24 sqrt(m / 2) of its size, 1.0e-7, and the last rounding adds
2^-25; 1.7e-7 of a layer's norm."""
import numpy as np
import pytest
import torch
import torch.nn.functional as Fn
from torch.nn import grad as G

import tg3
from oracle import cnn_oracle as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _params(rng):
    lay, total = C.layout()
    p = np.zeros(total, np.float32)
    for wo, ws, bo, co in lay:
        nw = int(np.prod(ws))
        p[wo:wo + nw] = rng.integers(0, 2, nw) * 2 - 1.0
        p[wo:wo + nw] *= rng.random(nw) < min(0.25, 12.0 / (nw // ws[0]))
        p[bo:bo + co] = rng.integers(-1, 2, co)
    return p


def _reference(params, img, g_out, bad=None):
    """Outputs, gradients (the parameter layout) and the largest sum of |terms|
    met on the way; `bad` marks the pixels that are not numbers, whose first
    layer's outputs are 0 and pass no gradient."""
    lay, total = C.layout()
    p = torch.as_tensor(params, dtype=torch.float64, device=DEV)
    x = torch.as_tensor(img, dtype=torch.float64, device=DEV)[:, None]
    hit = None
    if bad is not None:
        x = torch.where(bad[:, None], torch.zeros_like(x), x)
        hit = Fn.max_pool2d(bad[:, None].double(), 3, 1, 1) > 0
    W = [p[wo:wo + int(np.prod(ws))].reshape(ws) for wo, ws, _, _ in lay]
    acts, largest = [x], 0.0
    for i, (_, _, bo, co) in enumerate(lay):
        b, s = p[bo:bo + co], C.SHAPES[i][4]
        conv = (lambda a, w: Fn.conv2d(a, w, None, s, 1)) if s else (lambda a, w: a.flatten(1) @ w.T)  # noqa: E731,B023
        y = conv(acts[i], W[i]) + (b[:, None, None] if s else b)
        largest = max(largest, float(conv(acts[i].abs(), W[i].abs()).max()))
        if i < len(lay) - 1:
            y = y.clamp_min(0)
        if i == 0 and hit is not None:
            y = torch.where(hit, torch.zeros_like(y), y)
        acts.append(y)
    grad = torch.zeros(total, dtype=torch.float64, device=DEV)
    gy = torch.as_tensor(g_out, dtype=torch.float64, device=DEV)
    for i in range(len(lay) - 1, -1, -1):
        (wo, ws, bo, co), s = lay[i], C.SHAPES[i][4]
        if i < len(lay) - 1:
            gy = gy.reshape(acts[i + 1].shape) * (acts[i + 1] > 0)
        if s:
            back = lambda g, w: G.conv2d_input(acts[i].shape, w, g, s, 1)      # noqa: E731,B023
            gW, gb = G.conv2d_weight(acts[i], ws, gy, s, 1), gy.sum((0, 2, 3))
        else:
            back = lambda g, w: (g @ w).reshape(acts[i].shape)                 # noqa: E731,B023
            gW, gb = gy.T @ acts[i].flatten(1), gy.sum(0)
        grad[wo:wo + gW.numel()], grad[bo:bo + co] = gW.flatten(), gb
        if i:
            largest = max(largest, float(back(gy.abs(), W[i].abs()).max()))
            gy = back(gy, W[i])
    return acts[-1], grad.cpu().numpy(), largest


def _run(params, img, g_out):
    n = len(img)
    net = tg3.Cnn(0, seed=1)
    try:
        net.set_params(params)
        out = torch.empty((n, tg3.Cnn.N_OUT), dtype=torch.float32, device=DEV)
        im = torch.as_tensor(img).to(DEV)
        net.forward(im, out)
        net.zero_grads()
        net.backward(im, torch.as_tensor(g_out).to(DEV))
        return out, net.grads().astype(np.float64)
    finally:
        net.close()


@pytest.mark.parametrize("n", [1, 7, 80, 160, 256, 320, 640])
def test_sums(n):
    rng = np.random.default_rng(n)
    params = _params(rng)
    img = rng.integers(-400, 401, (n, 64, 64)).astype(np.float32)
    g_out = rng.integers(-400, 401, (n, tg3.Cnn.N_OUT)).astype(np.float32)
    ref_out, ref, largest = _reference(params, img, g_out)
    assert largest < 2 ** 24
    out, g = _run(params, img, g_out)
    assert torch.equal(out.double(), ref_out)
    for i, (wo, ws, bo, co) in enumerate(C.layout()[0]):
        if not C.SHAPES[i][4]:
            continue
        for a, b in ((wo, bo), (bo, bo + co)):
            d, r = np.linalg.norm(g[a:b] - ref[a:b]), np.linalg.norm(ref[a:b])
            assert d <= 1.7e-7 * r, (i, d / r)


def test_sums_keep_their_order():
    """The same batch twice: the gradients are equal to the last bit."""
    rng = np.random.default_rng(3)
    params = rng.standard_normal(C.layout()[1]).astype(np.float32) * 0.05
    img = rng.standard_normal((40, 64, 64)).astype(np.float32)
    g_out = rng.standard_normal((40, tg3.Cnn.N_OUT)).astype(np.float32)
    a, b = (_run(params, img, g_out) for _ in range(2))
    for i, (wo, _, bo, co) in enumerate(C.layout()[0]):
        if C.SHAPES[i][4]:
            np.testing.assert_array_equal(a[1][wo:bo + co], b[1][wo:bo + co])


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("n", [3, 40])
def test_pixels_not_finite(n, value):
    """A pixel that is not a number: the first layer's outputs over it are 0 by
    the ReLU and pass no gradient, so all gradients stay finite.  An infinite
    one with weights of one sign over it does the same where the outputs are
    -inf."""
    rng = np.random.default_rng(n)
    params = _params(rng)
    if np.isinf(value):
        w0, ws, _, _ = C.layout()[0][0]
        params[w0:w0 + int(np.prod(ws))] = -1.0
    img = rng.integers(-400, 401, (n, 64, 64)).astype(np.float32)
    img[1, 20, 31] = img[2, 0, 0] = value
    g_out = rng.integers(-400, 401, (n, tg3.Cnn.N_OUT)).astype(np.float32)
    bad = torch.as_tensor(~np.isfinite(img)).to(DEV)
    ref_out, ref, largest = _reference(params, np.nan_to_num(img, nan=0, posinf=0), g_out, bad)
    assert largest < 2 ** 24
    out, g = _run(params, img, g_out)
    assert torch.equal(out.double(), ref_out)
    for i, (wo, ws, bo, co) in enumerate(C.layout()[0]):
        if C.SHAPES[i][4]:
            d, r = np.linalg.norm(g[wo:bo + co] - ref[wo:bo + co]), np.linalg.norm(ref[wo:bo + co])
            assert d <= 1.7e-7 * r, (i, d / r)
