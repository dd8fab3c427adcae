"""The device field generator's periodic Gaussian passes against a NumPy
restatement of the whole generator (SplitMix64 noise, Box-Muller, three
circular convolutions, standardisation, exp), at the sizes where the passes'
tiling changes: lines that are not a multiple of 32, outputs split into equal
parts (64 | 65, 129), kernels longer than the period (wrapping several times),
a grid whose scratch values overlap its last elements (N=2), and a kernel too
wide for the shared-memory window (R = 480).

Tolerance: each pass adds `taps` rounded products, so g's absolute error is at
most 3 taps u sum|w||x|; against the standard deviation g is divided by, that
is 3 taps u (sum w / sqrt(sum w^2))^3 per unit of noise, and k = exp(sigma g)
carries it as a relative error.  A factor 4 covers the noise's size and the
functions' own last places.
"""
import math

import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import Dev

pytestmark = pytest.mark.gpu


def mix(x):
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def restated(n, mu, sigma, L, seed):
    with np.errstate(over="ignore"):
        c = mix(np.array([seed], np.uint64)) + np.uint64(2) * np.arange(n ** 3, dtype=np.uint64)
        u = [((mix(c + np.uint64(i)) >> np.uint64(11)).astype(np.float64) + 1.0) * 2.0 ** -53 for i in (0, 1)]
    g = (np.sqrt(-2.0 * np.log(u[0])) * np.cos(2.0 * np.pi * u[1])).reshape(n, n, n)
    s = 0.5 * L * n
    R = min(max(1, math.ceil(6.0 * s)), 2047)
    w = np.exp(-np.arange(-R, R + 1) ** 2 / (2.0 * s * s))
    for axis in (2, 1, 0):
        # the kernel folded onto the period, then a circular convolution
        fold = np.zeros(n)
        np.add.at(fold, np.arange(-R, R + 1) % n, w)
        C = fold[(np.arange(n)[None, :] - np.arange(n)[:, None]) % n]      # C[i, j]: in j -> out i
        g = np.moveaxis(np.tensordot(g, C, axes=([axis], [1])), -1, axis)
    g = (g - g.mean()) / g.std()
    tol = 4 * sigma * 3 * (2 * R + 1) * 2.0 ** -53 * (w.sum() / math.sqrt((w ** 2).sum())) ** 3 + 1e-14
    return np.exp(mu + sigma * g).ravel(), tol


@pytest.mark.parametrize("N,L", [(2, 0.5), (3, 0.9), (8, 0.25), (31, 0.2), (33, 0.1), (33, 1.5), (64, 0.1), (65, 0.1),
                                 (129, 0.05), (160, 1.0)])
def test_field_against_restatement(N, L):
    dev = Dev()
    mu, sigma, seed = 0.3, 0.8, 1234 + N
    k, r = dev.zeros(N ** 3), dev.zeros(N ** 3)
    _lib.field_lognormal(N, mu, sigma, L, seed, 2.5, k.data_ptr(), r.data_ptr())
    want, tol = restated(N, mu, sigma, L, seed)
    assert np.all(dev.get(r) == 2.5)
    assert np.max(np.abs(dev.get(k) / want - 1.0)) <= tol
