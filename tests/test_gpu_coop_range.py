"""Where the cooperative PCG solve begins and ends, and that it is what runs
there: a CTA has one run up to N = 52 and several from 53 on; the last size whose
runs are one flat block each is 71 (729 blocks of 512 nodes against 740 runs),
72 is solved by the loop of launches.  The Gauss form has one CTA per SM: at
N = 46 its 141 tiles fit with several runs each, the 288 tiles of 47 do not.
Solves and faults at these sizes against the oracle, bit for bit."""
import pytest

from mnhack8_b200 import _lib
from tests import test_gpu_small_pcg as small
from tests.helpers import field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,N,coop", [(f, n, n <= 71) for f in ("wht", "fast") for n in (52, 53, 66, 71, 72)] +
                         [("gauss", 46, True), ("gauss", 47, False)])
def test_edges(oracle, form, N, coop):
    k, r = field(N, "lognormal", sigma=1.0, L=0.25, seed=N)
    g = _lib.Solver(N, 5e-4, k, r, kernel=form, scatter="colored")
    blocks = -(-(N + 1) ** 3 // 512)
    lay = _lib.layout(N)
    NN = N + 1
    tiles = -(-NN // lay["cx"]) * -(-NN // lay["ty"]) * -(-NN // lay["tz"])
    several = blocks > (148 if form == "gauss" else 296)
    assert g.coop_ctas == (max(tiles, -(-blocks // 3) if several else blocks) if coop else 0)
    g.close()
    small.test_solve_and_faults_bitwise(oracle, form, N)


def test_other_paths_are_not_cooperative():
    k, r = field(20, "lognormal", sigma=1.0, L=0.25, seed=20)
    with_atomics = _lib.Solver(20, 5e-4, k, r, kernel="wht", scatter="atomic")
    assert with_atomics.coop_ctas == 0
    with_atomics.close()
