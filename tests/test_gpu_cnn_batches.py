"""The network's FP32 convolutions at batch sizes on and off their tiles (four
images a tile at 8 x 8, shares of the batch in the weight gradient), against
the float64 oracle.

Inputs and weights are small whole numbers, so every sum of the forward pass
is exact in FP32: the outputs must be equal, and no ReLU sits on another side
of zero than the oracle's.  The gradients are FP32 sums of up to 4,096 n
products: sqrt(4096 n) 2^-24 of the root sum of squares of the terms, which
for these incoherent sums is the size of the sum; 3e-5 of the norm at n = 33,
for every layer's weights and biases."""
import numpy as np
import pytest
import torch

import tg3
from oracle import cnn_oracle as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [1, 3, 4, 6, 33])
def test_whole_numbers(n):
    rng = np.random.default_rng(n)
    lay, total = C.layout()
    params = np.zeros(total, np.float32)
    for wo, ws, bo, co in lay:
        nw = int(np.prod(ws))
        share = min(0.25, 12.0 / (nw // ws[0]))         # about 12 taps an output
        params[wo:wo + nw] = rng.integers(0, 2, nw) * 2 - 1.0
        params[wo:wo + nw] *= rng.random(nw) < share
        params[bo:bo + co] = rng.integers(-1, 2, co)
    img = rng.integers(-1, 2, (n, 64, 64)).astype(np.float32)
    g_out = rng.integers(-1, 2, (n, tg3.Cnn.N_OUT)).astype(np.float32)
    acts = C.forward(params, img)
    assert max(np.abs(a).max() for a in acts) < 2 ** 20
    ref = C.grad_from_output(params, img, g_out, acts=acts)
    net = tg3.Cnn(0, seed=1)
    try:
        net.set_params(params)
        out = torch.empty((n, tg3.Cnn.N_OUT), dtype=torch.float32, device=DEV)
        im = torch.as_tensor(img).to(DEV)
        net.forward(im, out)
        np.testing.assert_array_equal(out.cpu().numpy(), acts[-1].astype(np.float32))
        net.zero_grads()
        net.backward(im, torch.as_tensor(g_out).to(DEV))
        g = net.grads().astype(np.float64)
    finally:
        net.close()
    for li, (wo, ws, bo, co) in enumerate(lay):
        nw = int(np.prod(ws))
        for a, b in ((wo, wo + nw), (bo, bo + co)):
            d, r = np.linalg.norm(g[a:b] - ref[a:b]), np.linalg.norm(ref[a:b])
            assert d <= 3e-5 * r, (li, d / r)
