"""A wait inside a kernel that gives up fails the call that launched it, whichever
call that is, and leaves the handle usable.  With fail_waits every wait counts as
given up (the kernels run on or return by themselves).  N = 12 is the
cooperative solve, N = 80 the loop of launches; the atomic scatter has no such
waits."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import Dev, bits, field

pytestmark = pytest.mark.gpu


def solver(N, form, scatter="colored"):
    k, r = field(N, "lognormal", sigma=1.0, L=0.25, seed=N)
    return _lib.Solver(N, 5e-4, k, r, kernel=form, scatter=scatter, detect=True, ic="gaussian", ic_sigma=0.15)


@pytest.mark.parametrize("form,N", [("wht", 12), ("wht", 80), ("fast", 12), ("fast", 80), ("gauss", 12)])
def test_every_call_reports_it(form, N):
    dev = Dev()
    g = solver(N, form)
    assert (g.coop_ctas > 0) == (N == 12)
    T0 = _lib.gaussian_ic(N, 0.15)
    x, y, b, s = dev.put(T0), dev.zeros(T0.size), dev.zeros(T0.size), dev.put(T0)

    def outputs():
        g.build_rhs_ptr(x.data_ptr(), b.data_ptr())
        g.apply_ptr(x.data_ptr(), y.data_ptr())
        s.copy_(x)
        dev.torch.cuda.synchronize()
        it = g.pcg_ptr(b.data_ptr(), s.data_ptr(), 500, 1e-8)
        res = g.run_case(2, snap_every=1)
        T, its, _ = g.solve_host(T0, 2)
        adv = g.advance(2, from_ic=True)[0]
        n, log = g.diag_cg()
        return ([dev.get(v).copy() for v in (b, y, s)] + [res["T"], T, g.get_field()],
                [it, its, adv, n, log["rel0"]] + [r["cg_iters"] for r in res["steps"]] + [r["d2"] for r in res["steps"]])

    want = outputs()
    g.fail_waits(True)
    for call in (lambda: g.build_rhs_ptr(x.data_ptr(), b.data_ptr()), lambda: g.apply_ptr(x.data_ptr(), y.data_ptr()),
                 lambda: g.apply_ptr(x.data_ptr(), y.data_ptr(), dt_eff=0.0),
                 lambda: g.pcg_ptr(b.data_ptr(), s.data_ptr(), 500, 1e-8), lambda: g.run_case(2, snap_every=1),
                 lambda: g.solve_host(T0, 2), lambda: g.advance(2, from_ic=True),
                 lambda: g.time_kernel(0, reps=2)):
        with pytest.raises(_lib.HeatError, match="gave up"):
            call()
    g.fail_waits(False)
    got = outputs()
    assert got[1] == want[1]
    for a, c in zip(got[0], want[0]):
        assert np.array_equal(bits(a), bits(c))
    g.close()


def test_atomic_scatter_has_no_waits():
    g = solver(12, "wht", scatter="atomic")
    g.fail_waits(True)
    g.run_case(1, snap_every=0)
    g.close()


@pytest.mark.parametrize("N", [12, 80])
def test_failed_log_leaves_nothing_behind(N):
    """A diag_cg that fails frees the buffer its solve logged into; later solves
    of the handle give what they gave, and a later log is whole."""
    g = solver(N, "wht")
    n, log = g.diag_cg()
    want = g.run_case(2, snap_every=0)["T"]
    g.fail_waits(True)
    with pytest.raises(_lib.HeatError, match="gave up"):
        g.diag_cg()
    g.fail_waits(False)
    assert np.array_equal(bits(g.run_case(2, snap_every=0)["T"]), bits(want))
    m, again = g.diag_cg()
    assert m == n and all(np.array_equal(bits(again[k]), bits(log[k])) for k in ("rel", "alpha", "beta"))
    g.close()
