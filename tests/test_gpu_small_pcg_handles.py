"""Several cooperative solvers alive at once.  Grids of one instantiation of the
kernel differ in shared memory (tiles of one plane at N = 53..59, of two at
60..71), and its limit is the kernel's, not a handle's: a handle created later,
of a smaller or a larger tile, leaves the earlier ones as they were."""
import numpy as np
import pytest

from mnhack8_b200 import _lib
from tests.helpers import bits
from tests.test_gpu_small_pcg import pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["wht", "fast"])
@pytest.mark.parametrize("sizes", [(65, 54), (54, 65)])
def test_handles_of_different_tiles(oracle, form, sizes):
    # one kernel, two tile depths
    assert [_lib.layout(n)["cx"] for n in sorted(sizes)] == [1, 2]
    pairs = [pair(oracle, n, form) for n in sizes]
    for o, g in pairs + pairs[::-1]:
        ref, got = o.run_case(2, snap_every=1), g.run_case(2, snap_every=1)
        assert [s["cg_iters"] for s in got["steps"]] == [s["cg_iters"] for s in ref["steps"]]
        assert np.array_equal(bits(got["T"]), bits(ref["T"]))
    for _, g in pairs:
        g.close()
