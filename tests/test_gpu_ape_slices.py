"""FP32 smearing where four time slices of the field pass the size of L2 (126 MB on B200), beyond which a step is
another kernel, and on both sides of that line."""
import numpy as np
import pytest

import _oracle as O
from masterarbeit_b200 import Lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["all", "spatial", "temporal"])
@pytest.mark.parametrize("dims", [(2, 100, 74, 74),    # 140 MB in four slices; two neighbours in t are one site
                                  (4, 96, 74, 74),     # 135 MB
                                  (4, 72, 80, 86)])    # 127 MB: 126.8e6 bytes, below 132.6e6
def test_two_steps_against_the_oracle(dims, mode):
    U = O.start(dims, "haar", 5).astype(np.float32).astype(np.float64)
    L = Lattice(dims, precision="fp32")
    L.upload(U)
    L.ape(2, 0.1, mode)
    # u = 2^-24.  One step: a staple is two products of unit quaternions, some 10 u, six of them times 0.1, the sum and its
    # norm, |v| >= 1 - 0.6: below 25 u.  The second step carries that on with (1 + 18 * 0.1) / 0.4 = 7: below 2^8 u.
    assert np.max(np.abs(L.download() - O.ape(dims, U, 2, 0.1, mode))) <= 2.0 ** (8 - 24)
