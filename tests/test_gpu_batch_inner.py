"""The batched engine's FP32 inner loop at the sizes where it can go wrong:
grids whose nodes are not a multiple of four or of the update's chunk of 8192
nodes (1, 2, 12, 13), tiles with one and with several rows of positions per
thread (13, 29, 40), several tiles per plane (40), uniform rho*c (read as one
value) and varying rho*c, checksum on and off.

Each instance's steps are compared with the oracle's FP64 PCG to 1e-13: the
outer iteration stops at a true relative residual of 1e-10, and the Jacobi-
scaled systems here have condition numbers of a few tens, so the fields agree
to 1e-8.  The instances of one batch are also run alone and must give the same bits."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import bits, random_field

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 12, 13, 29, 40]


def problem(N, uniform):
    k, r = random_field(N, 7 * N, contrast=1.0)
    if uniform:
        r = np.full_like(r, 0.75)
    return k, r


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("detect", [True, False])
def test_sizes_alone_and_mixed(oracle, uniform, detect):
    dt, steps = 2e-4, 3
    mix = _lib.Batch(rtol=1e-10, detect=detect)
    slots = {}
    for N in SIZES:
        k, r = problem(N, uniform)
        slots[N] = mix.add(N, dt, k, r, T0=_lib.gaussian_ic(N, 0.15), steps=steps)
    while mix.step()[0]:
        pass
    for N in SIZES:
        k, r = problem(N, uniform)
        T0 = _lib.gaussian_ic(N, 0.15)
        b = _lib.Batch(rtol=1e-10, detect=detect)
        s = b.add(N, dt, k, r, T0=T0, steps=steps)
        while b.step()[0]:
            pass
        T, inf = b.field(s), b.info(s)
        b.close()
        assert inf["stalls"] == 0 and inf["inner_faults"] == 0 and inf["rel_residual"] < 1e-10
        assert np.array_equal(bits(T), bits(mix.field(slots[N]))), N
        assert inf["inner_iters"] == mix.info(slots[N])["inner_iters"]
        o = oracle.Oracle(N, dt, k, r, form="wht", no_source=True, ic="gaussian", ic_sigma=0.15)
        ref = o.run_case(steps, snap_every=0, tol=1e-13)["T"]
        assert np.linalg.norm(T - ref) <= 1e-8 * np.linalg.norm(ref), N
    mix.close()
