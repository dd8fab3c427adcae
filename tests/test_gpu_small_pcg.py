"""The cooperative PCG kernel (small grids) against the oracle, bit for bit, at
the sizes where its variants change: positions per thread (N = 13 | 14 and
19 | 20: (N+3)^2 positions of a tile plane against 256 and 512), the exchange
gate (more than 48 CTAs), runs per CTA (53 | 54: more flat blocks than CTAs
fit at once), several planes per tile (64), and the last size a run is one
flat block (88 | 89)."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import Dev, bits, field, random_field

pytestmark = pytest.mark.gpu


def pair(oracle, N, form, **kw):
    # (a one-element field has no variance to standardise)
    k, r = field(N, "lognormal", sigma=1.0, L=0.25, seed=N) if N > 1 else random_field(N, 1)
    o = oracle.Oracle(N, 5e-4, k, r, form=form, detect=True, ic="gaussian", ic_sigma=0.15, **kw)
    g = _lib.Solver(N, 5e-4, k, r, kernel=form, scatter="colored", detect=True, ic="gaussian", ic_sigma=0.15, **kw)
    return o, g


@pytest.mark.parametrize("form,N", [("wht", n) for n in (1, 4, 13, 14, 19, 20, 27, 53, 54, 64, 88, 89)] +
                         [("fast", n) for n in (13, 14, 20, 53, 54, 64)] + [("gauss", n) for n in (14, 24)])
def test_solve_and_faults_bitwise(oracle, form, N):
    """Two steps with the source, the detectors and a kept reference; then a
    flip at every place the kernel handles one, on a node of a tile face."""
    o, g = pair(oracle, N, form)
    ref = o.run_case(2, snap_every=1, keep_snaps=True)
    got = g.run_case(2, snap_every=1, keep_reference=True)
    NN = N + 1
    node = (NN // 2 * NN + NN // 2) * NN + NN // 2
    runs = [(None, got, ref)]
    if N > 1:
        for fi in ((_lib.LEVELS["R"], 1, node % N ** 3, 55, 0), (_lib.LEVELS["P"], 0, node, 52, 3),
                   (_lib.LEVELS["RV"], 1, node, 60, 2), (_lib.LEVELS["AP"], 0, node, 55, 1)):
            runs.append((fi, g.run_case(2, snap_every=1, fi=fi),
                         o.run_case(2, snap_every=1, fi=fi, ref_snaps=ref["snaps"])))
    for fi, a, b in runs:
        assert np.array_equal(bits(a["T"]), bits(b["T"])), fi
        for s, t in zip(a["steps"], b["steps"]):
            assert s["cg_iters"] == t["cg_iters"], fi
            for key in ("d1", "d2", "tmin", "tmax") + (("E", "spread") if fi else ()):
                assert np.float64(s[key]).view(np.uint64) == np.float64(t[key]).view(np.uint64), (fi, key)
    g.close()


@pytest.mark.parametrize("N", [13, 30, 54])
@pytest.mark.parametrize("cap", [0, 1, 2, 3, 500])
def test_iteration_cap_and_zero_rhs(oracle, N, cap):
    """Caps at even and odd iterations, and b = 0 from x = 0 (breakdown at the first iteration)."""
    o, g = pair(oracle, N, "wht")
    dev = Dev()
    T = o.initial_condition()
    b = o.build_rhs(T)
    bd, xd = dev.put(b), dev.put(T)
    it = g.pcg_ptr(bd.data_ptr(), xd.data_ptr(), cap, 1e-12)
    it_ref, x_ref, _ = o.pcg(b, T, cap, 1e-12)
    assert it == it_ref and np.array_equal(bits(dev.get(xd)), bits(x_ref))
    z = np.zeros(o.Nn)
    bd, xd = dev.put(z), dev.put(z)
    it = g.pcg_ptr(bd.data_ptr(), xd.data_ptr(), cap, 1e-12)
    it_ref, x_ref, _ = o.pcg(z, z, cap, 1e-12)
    assert it == it_ref and np.array_equal(bits(dev.get(xd)), bits(x_ref))
    g.close()


def test_handles_in_threads(oracle):
    """Cooperative solves of several handles from several threads, beside a
    batched engine's steps: each gives the bits it gives alone."""
    import threading

    probs = [(48, "wht"), (30, "fast"), (60, "wht")]
    solvers = [pair(oracle, N, form)[1] for N, form in probs]

    def solve(i, out):
        for _ in range(3):
            solvers[i].advance(4, from_ic=True)
        out[i] = solvers[i].get_field()

    alone, mixed = {}, {}
    for i in range(len(probs)):
        solve(i, alone)
    k, r = field(40, "lognormal", sigma=1.0, L=0.25, seed=3)
    b = _lib.Batch(rtol=1e-8)
    s = [b.add(40, 5e-4, k, r, T0=_lib.gaussian_ic(40, 0.15), steps=20) for _ in range(2)]
    th = [threading.Thread(target=solve, args=(i, mixed)) for i in range(len(probs))]
    for t in th:
        t.start()
    while b.step()[0]:
        pass
    for t in th:
        t.join()
    for i in range(len(probs)):
        assert np.array_equal(bits(alone[i]), bits(mixed[i])), probs[i]
        solvers[i].close()
    assert np.array_equal(bits(b.field(s[0])), bits(b.field(s[1])))
    b.close()
