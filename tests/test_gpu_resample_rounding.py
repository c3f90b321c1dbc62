"""The resampler's parallel sums against sequential double sums, bit for bit,
on sets that stress the rounding: like terms (binade ends at every
doubling, ties), powers of two, terms over hundreds of binades, zeros,
subnormals; set sizes around the serial start (16) and the window (256), and
outputs shorter and longer than the set."""
import numpy as np
import pytest

import tg3
from oracle import oracle as O

pytestmark = pytest.mark.gpu

KINDS = {
    "uniform": lambda r, n: r.random(n),
    "equal": lambda r, n: np.full(n, 0.1),
    "powers": lambda r, n: 2.0 ** -r.integers(0, 60, n),
    "halves": lambda r, n: np.where(np.arange(n) == 0, 2.0 ** 40, 2.0 ** -13 * r.integers(1, 8, n)),
    "steep": lambda r, n: np.exp(-200 * r.random(n)),
    "zeros": lambda r, n: np.where(r.random(n) < 0.7, 0.0, r.random(n)),
    "small": lambda r, n: 2.0 ** -1020 * r.integers(1, 9, n),
}


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("n,n_out", [(1, 1), (2, 5), (15, 15), (16, 16), (17, 17), (100, 300),
                                     (255, 255), (257, 200), (272, 272), (1000, 1000),
                                     (2049, 4000), (8192, 8192)])
def test_sums_round_in_order(kind, n, n_out):
    rng = np.random.default_rng(n)
    nP = 3
    u = np.stack([KINDS[kind](rng, n) for _ in range(nP)])
    u[:, -1] = np.maximum(u[:, -1], u.max(axis=1) / 4)
    u[:, -1] = np.where(u[:, -1] > 0, u[:, -1], 0.5)         # a set of zeros is refused
    w = 2.0 ** rng.integers(-2, 3, (nP, n)) if kind != "uniform" else rng.random((nP, n))
    perm = np.stack([rng.permutation(n) for _ in range(nP)]).astype(np.int32)
    u0 = rng.random(nP) / n_out
    peaks = np.array([np.nan, 0.0, 0.3])
    if kind == "small":
        peaks[:] = 0.0
    src, top = np.zeros((nP, n_out), np.int32), np.zeros(nP, np.int32)
    wout = np.zeros((nP, n_out))
    tg3.check(tg3.lib().tg3_resample(nP, n, tg3.ptr(u), tg3.ptr(w), tg3.ptr(perm), tg3.ptr(u0),
                                     tg3.ptr(peaks), n_out, tg3.ptr(src), tg3.ptr(wout),
                                     tg3.ptr(top)))
    for b in range(nP):
        pf = O.peak_factor_r(u[b]) if np.isnan(peaks[b]) else peaks[b]
        s_ref, w_ref, t_ref = O.resample(u[b], w[b], perm[b], u0[b], pf, n_out)
        np.testing.assert_array_equal(src[b], s_ref)
        np.testing.assert_array_equal(wout[b], w_ref)
        assert top[b] == t_ref
