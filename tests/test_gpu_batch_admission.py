"""What the batched engine admits: every coefficient has to be positive, wherever
the bad one sits and whether rho*c is one value or not; rho*c that differs in one
element only, the first or the last, is not taken for one value."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import random_field

pytestmark = pytest.mark.gpu

N = 9


def solve(b, k, r, dt=2e-4, steps=2):
    s = b.add(N, dt, k, r, T0=_lib.gaussian_ic(N, 0.15), steps=steps)
    while b.step()[0]:
        pass
    T, inf = b.field(s), b.info(s)
    b.remove(s)
    assert inf["rel_residual"] < 1e-10 and inf["stalls"] == 0
    return T


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("which", ["k", "rhoc"])
@pytest.mark.parametrize("at", [0, 1, N ** 3 // 2, N ** 3 - 1])
@pytest.mark.parametrize("bad", [0.0, -1.0, float("nan")])
def test_bad_coefficient_is_refused(uniform, which, at, bad):
    k, r = random_field(N, 3, contrast=1.0)
    if uniform:
        r = np.full_like(r, 0.75)
    (k if which == "k" else r)[at] = bad
    b = _lib.Batch(rtol=1e-10)
    with pytest.raises(_lib.HeatError) as e:
        b.add(N, 2e-4, k, r, T0=_lib.gaussian_ic(N, 0.15), steps=1)
    assert e.value.status == 1
    solve(b, *random_field(N, 3, contrast=1.0))         # the engine works on
    b.close()


@pytest.mark.parametrize("at", [None, 0, 1, N ** 3 - 2, N ** 3 - 1])
def test_one_different_value(oracle, at):
    """As the oracle's FP64 solution to 1e-8 (tests/test_gpu_batch_inner.py); the
    one element's factor of 40 moves the field by far more."""
    k, _ = random_field(N, 5, contrast=1.0)
    r = np.full(N ** 3, 0.75)
    if at is not None:
        r[at] = 30.0
    b = _lib.Batch(rtol=1e-10)
    T = solve(b, k, r)
    b.close()
    o = oracle.Oracle(N, 2e-4, k, r, form="wht", no_source=True, ic="gaussian", ic_sigma=0.15)
    ref = o.run_case(2, snap_every=0, tol=1e-13)["T"]
    assert np.linalg.norm(T - ref) <= 1e-8 * np.linalg.norm(ref)
