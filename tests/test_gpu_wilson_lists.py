"""su2g_wilson forms only the loops of the extents in its list: sparse and unsorted lists, consecutive ones of
every chunk length, windows of T that start late, extents longer than the lattice, more T than one window
holds, and time extents whose columns are wide, narrow or do not fit a CTA (the per-site kernel)."""
import numpy as np
import pytest

import _oracle as O
from masterarbeit_b200 import Lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dims", [(8, 4, 6, 2), (14, 4, 2, 4), (22, 2, 4, 4), (34, 2, 2, 4), (48, 2, 2, 4)])
def test_loop_lists(dims, precision):
    U = O.start(dims, "haar", 4)
    L = Lattice(dims, precision=precision)
    L.upload(U)
    last = dims[0] - 1
    grid = [(r, t) for r in range(1, 10) for t in range(1, last + 1)]
    lists = [[(1, 1), (1, 5), (5, 1), (5, 5)], [(7, last), (2, 3), (7, 3), (2, last)], [(3, last)], [(1, 2), (2, 2)],
             [(r, 4) for r in (1, 2, 3, 5)], [(r, 2) for r in range(2, 9)], grid]
    for pairs in lists:
        R, T = [p[0] for p in pairs], [p[1] for p in pairs]
        # FP64: the loop tests' 1e-12; FP32: rounding 2^-24 of the about 2 (R + T) products of unit links a term
        bound = 1e-12 if precision == "fp64" else 2 * (max(R) + max(T)) * 2.0 ** -23
        assert np.max(np.abs(L.wilson(R, T) - O.wilson(dims, U, R, T))) <= bound, pairs[:4]
