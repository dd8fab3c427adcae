"""Every instantiation of the slab operator against the oracle, bit for bit:
uniform and varying rho*c (the uniform form reads only k), checksum on and
off, all three element forms, on grids whose tiles are one plane deep, ragged
in every direction, and above the cooperative solve's range; through the plain
apply, the right-hand side with its source, and a few PCG iterations."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import Dev, bits, random_field, random_nodes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,N", [("wht", n) for n in (1, 2, 29, 89, 97, 131)] + [("fast", 89), ("gauss", 89)])
@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("detect", [True, False])
def test_operator_and_pcg_bitwise(oracle, form, N, uniform, detect):
    k, r = random_field(N, 3 * N)
    if uniform:
        r = np.full_like(r, 1.75)
    o = oracle.Oracle(N, 3e-4, k, r, form=form, detect=detect)
    g = _lib.Solver(N, 3e-4, k, r, kernel=form, scatter="colored", detect=detect)
    dev = Dev()
    x = random_nodes(N, N)                  # boundary values too
    xd, yd = dev.put(x), dev.zeros(o.Nn)
    for dt_eff in (o.dt, 0.0):
        rel = g.apply_ptr(xd.data_ptr(), yd.data_ptr(), dt_eff=dt_eff)
        want, rel_ref = o.apply(x, dt_eff=dt_eff, project=True, d1=detect)
        assert np.array_equal(bits(dev.get(yd)), bits(want))
        if detect:
            assert np.float64(rel).view(np.uint64) == np.float64(rel_ref).view(np.uint64)
    g.build_rhs_ptr(xd.data_ptr(), yd.data_ptr())
    b = o.build_rhs(x)
    assert np.array_equal(bits(dev.get(yd)), bits(b))
    for cap in (1, 6):
        sd = dev.put(x)
        it = g.pcg_ptr(yd.data_ptr(), sd.data_ptr(), cap, 1e-14)
        it_ref, x_ref, _ = o.pcg(b, x, cap, 1e-14)
        assert it == it_ref and np.array_equal(bits(dev.get(sd)), bits(x_ref))
    g.close()
