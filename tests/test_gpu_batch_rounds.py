"""The batched engine's inner update at the edges of its rounds per block, which
follow the rounds of 2048 nodes of all instances together (N = 105 alone: 582
rounds, one per block; 106: 599, two; 133: 1175, two; 134: 1202, four), and where
the last round is full (N = 15, 63) or not (16).

Each instance is compared with the oracle's FP64 PCG to 1e-13, as in
test_gpu_batch_inner.py (the outer iteration stops at a true relative residual of
1e-10 and the Jacobi-scaled systems have condition numbers of a few tens, so the
fields agree to 1e-8).  It gives the same bits alone, among small ones and beside a
large one, whatever rounds a block then has."""
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


@pytest.mark.parametrize("N", [15, 16, 63, 105, 106, 133, 134])
def test_edges(oracle, N):
    (T, inf), = run([N])
    assert inf["stalls"] == 0 and inf["inner_faults"] == 0 and inf["rel_residual"] < 1e-10
    for others in ([20, N, 9], [110, N], [140, N]):         # one to two, and four rounds a block
        mixed, inf2 = run(others)[1]
        assert np.array_equal(bits(T), bits(mixed)) and inf["inner_iters"] == inf2["inner_iters"], others
    k, r = problem(N)
    o = oracle.Oracle(N, DT, k, r, form="wht", no_source=True, ic="gaussian", ic_sigma=0.15)
    ref = o.run_case(STEPS, snap_every=0, tol=1e-13)["T"]
    assert np.linalg.norm(T - ref) <= 1e-8 * np.linalg.norm(ref)


def test_rounds_change_while_running():
    """Instances leave and the others go on with fewer rounds a block: same bits."""
    b = _lib.Batch(rtol=1e-10)
    small = b.add(30, DT, *problem(30), T0=_lib.gaussian_ic(30, 0.15), steps=6)
    large = b.add(140, DT, *problem(140), T0=_lib.gaussian_ic(140, 0.15), steps=6)
    b.step()
    b.step()
    b.remove(large)                                         # four rounds a block, then one
    b.step()
    mid = b.add(110, DT, *problem(110), T0=_lib.gaussian_ic(110, 0.15), steps=2)
    while b.step()[0]:                                      # two, as mid is done but stays
        pass
    T = b.field(small)
    assert b.info(mid)["steps_done"] == 2
    b.close()
    a = _lib.Batch(rtol=1e-10)
    s = a.add(30, DT, *problem(30), T0=_lib.gaussian_ic(30, 0.15), steps=6)
    while a.step()[0]:
        pass
    assert np.array_equal(bits(T), bits(a.field(s)))
    a.close()
