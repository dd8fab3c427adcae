"""The batched engine's inner update at the grids where its chunks' rounds change
(N = 83 | 84: one and two, 133 | 134: two and four), and where the last round of
2048 nodes is full (N = 15, 63) or not (16).

Each instance is compared with the oracle's FP64 PCG to 1e-13, as in
test_gpu_batch_inner.py (the outer iteration stops at a true relative residual of
1e-10 and the Jacobi-scaled systems have condition numbers of a few tens, so the
fields agree to 1e-8), and gives the same bits alone and among others."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import bits, random_field

pytestmark = pytest.mark.gpu

DT, STEPS = 5e-5, 2


def problem(N):
    k, r = random_field(N, 7 * N, contrast=1.0)
    return k, np.full_like(r, 0.75) if N % 2 else r


def run(sizes):
    b = _lib.Batch(rtol=1e-10)
    slots = [b.add(N, DT, *problem(N), T0=_lib.gaussian_ic(N, 0.15), steps=STEPS) for N in sizes]
    while b.step()[0]:
        pass
    out = [(b.field(s), b.info(s)) for s in slots]
    b.close()
    return out


@pytest.mark.parametrize("N", [15, 16, 63, 83, 84, 133, 134])
def test_edges(oracle, N):
    (T, inf), = run([N])
    assert inf["stalls"] == 0 and inf["inner_faults"] == 0 and inf["rel_residual"] < 1e-10
    _, (mixed, inf2), _ = run([20, N, 9])
    assert np.array_equal(bits(T), bits(mixed)) and inf["inner_iters"] == inf2["inner_iters"]
    k, r = problem(N)
    o = oracle.Oracle(N, DT, k, r, form="wht", no_source=True, ic="gaussian", ic_sigma=0.15)
    ref = o.run_case(STEPS, snap_every=0, tol=1e-13)["T"]
    assert np.linalg.norm(T - ref) <= 1e-8 * np.linalg.norm(ref)
