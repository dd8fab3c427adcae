"""The initial condition a handle keeps on the device is uploaded on the handle's
own stream, complete before the first step reads it: a solve neither waits for
work that the caller has on the default stream nor takes part in its order.  A
trajectory's run keeps it only where that is little memory."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import bits, field

pytestmark = pytest.mark.gpu


def solver(N):
    k, r = field(N, "lognormal", sigma=1.0, L=0.25, seed=N)
    return _lib.Solver(N, 5e-4, k, r, detect=True, no_source=True, ic="gaussian", ic_sigma=0.15)


@pytest.mark.parametrize("how", ["advance", "run_case"])
def test_upload_is_on_the_handles_stream(how):
    import torch

    N = 24

    def go(g):
        if how == "advance":
            g.advance(1, from_ic=True)
        else:
            g.run_case(1, snap_every=0, want_T=False)

    warm, g = solver(N), solver(N)
    go(warm)                                    # kernels loaded, buffers allocated once
    torch.cuda.synchronize()
    torch.cuda._sleep(1_000_000_000)            # about half a second of the default stream
    busy = torch.cuda.Event()
    busy.record()
    go(g)                                       # the first upload of this handle
    waited = busy.query()
    torch.cuda.synchronize()
    assert not waited
    assert np.array_equal(bits(g.get_field()), bits(warm.get_field()))
    warm.close()
    g.close()


@pytest.mark.parametrize("N", [20, 65, 100])
def test_first_run_equals_the_next(N):
    g = solver(N)
    g.advance(2, from_ic=True)
    first = g.get_field()
    g.advance(2, from_ic=True)
    assert np.array_equal(bits(first), bits(g.get_field()))
    g.close()
    h = solver(N)
    got = h.run_case(2, snap_every=0)["T"]
    assert np.array_equal(bits(first), bits(got))
    h.close()


def test_run_case_keeps_no_large_field():
    """Where device memory is short, a run leaves the handle with what it had
    (N = 200: 65 MB a field, 3 GB free)."""
    import torch

    N = 200
    r = np.ones(N ** 3)
    g = _lib.Solver(N, 5e-4, r, r, detect=False, no_source=True, ic="gaussian", ic_sigma=0.15)
    g.advance(1)                                # the graph and its launch are in memory
    torch.cuda.synchronize()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device="cuda")
    before = torch.cuda.mem_get_info()[0]
    T = g.run_case(1, snap_every=0)["T"]
    assert before - torch.cuda.mem_get_info()[0] < 16 << 20
    del rest
    torch.cuda.empty_cache()
    g.advance(1, from_ic=True)                  # this call keeps it, as documented
    assert np.array_equal(bits(T), bits(g.get_field()))
    g.close()
