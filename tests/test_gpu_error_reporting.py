"""An error belongs to the call that reports it: the next call of the thread,
on the same or another handle, is not failed by it."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import bits, field

pytestmark = pytest.mark.gpu


def solver(N):
    k, r = field(N, "lognormal", sigma=1.0, L=0.25, seed=N)
    return _lib.Solver(N, 5e-4, k, r, detect=True, no_source=True, ic="gaussian", ic_sigma=0.15)


def test_refused_allocation_does_not_fail_the_next_call():
    """A campaign whose kept fields do not fit the device (N = 128: 17 MB each,
    200 of them with 1 GB free) is refused; solves go on."""
    import torch

    N = 128
    r = np.ones(N ** 3)
    g = _lib.Solver(N, 5e-4, r, r, detect=True, no_source=True, ic="gaussian", ic_sigma=0.15)
    other = solver(10)
    g.advance(1, from_ic=True)
    want = g.get_field()
    torch.cuda.synchronize()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    for nxt in (lambda: g.advance(1, from_ic=True), lambda: other.advance(1, from_ic=True)):
        with pytest.raises(_lib.HeatError):
            g.campaign(200, 5, 1, 1)
        nxt()
    del rest
    torch.cuda.empty_cache()
    assert np.array_equal(bits(g.get_field()), bits(want))
    g.close()
    other.close()
