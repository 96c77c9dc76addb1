"""The FP64 sampler's logarithm, squared cosine and sine/cosine work on the random words themselves: a
heatbath pass at couplings from where almost every trial is taken to where most are refused, link by
link against the oracle's general library functions on the same words."""
import numpy as np
import pytest

import _oracle as O
from masterarbeit_b200 import Lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.05, 0.7, 2.3, 3.09, 40.0])
@pytest.mark.parametrize("dims", [(8, 6, 4, 10), (2, 4, 2, 6)])
def test_heatbath_against_the_oracle(dims, beta):
    U = O.start(dims, "haar", 21)
    L = Lattice(dims, precision="fp64", beta=beta, seed=77, start="cold")
    L.upload(U)
    acc = L.sweep(1, 1, 0, acc=True)
    want = U.copy()
    ref = O.sweep(dims, want, "hb", beta, 77, 0)
    assert abs(acc - ref) <= 1e-12
    # the functions' errors are a few 2^-53 of the draw; sqrt(delta (2 - delta)) and a link's eight passes
    # magnify them: the link-by-link bound of the heatbath tests, 1e-12
    assert np.max(np.abs(L.download() - want)) <= 1e-12
