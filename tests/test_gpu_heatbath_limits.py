"""The heatbath where its couplings leave the ordinary range: at an infinite or huge beta every draw is the unit
quaternion (delta = 0, or too small to move x0), so that a sweep projects each link onto its staple."""
import numpy as np
import pytest

import _oracle as O
from masterarbeit_b200 import Lattice
from masterarbeit_b200.su2g import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [float("inf"), 1e300])
@pytest.mark.parametrize("dims", [(4, 6, 2, 4), (8, 8, 10, 10)])
def test_infinite_beta_projects_onto_the_staple(dims, beta):
    want = O.start(dims, "haar", 7)
    O.sweep(dims, want, "hb", beta, 7, 0)
    # some 24 roundings of the staple's 6 terms a link, divided by |A| (0.15 at the least among these Haar links),
    # once more by a neighbour's |A|: below 2^14 units of rounding
    for precision, bound in (("fp64", 2.0 ** (14 - 53)), ("fp32", 2.0 ** (14 - 24))):
        L = Lattice(dims, precision=precision, beta=beta, seed=7, start="cold")
        L.upload(O.start(dims, "haar", 7))
        L.sweep(1, 1, 0)
        assert np.max(np.abs(L.download() - want)) <= bound, precision
        B = Batch([{"dims": dims, "beta": beta, "seed": 7, "replica": 0, "start": "cold"}], precision=precision)
        B.upload(0, O.start(dims, "haar", 7))
        B.run(1, 1, 0)
        assert np.max(np.abs(B.download(0) - want)) <= bound, precision
        # all draws in the bin that ends at x0 = 1
        counts = L.kp_histogram(beta, 3, 10000, 16)
        assert counts[-1] == 10000 and counts.sum() == 10000

