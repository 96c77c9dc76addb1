"""FP64 sweeps of lattices up to 4096 sites, which one thread-block cluster runs in one launch, against the
checkerboard passes (which a profiled handle takes): smallest lattice, a part-filled last warp, the largest
that fits, one beyond it."""
import numpy as np
import pytest

from masterarbeit_b200 import Lattice

pytestmark = pytest.mark.gpu


def _pair(dims, replica=0):
    out = []
    for passes in (False, True):
        L = Lattice(dims, precision="fp64", beta=2.4, seed=31, start="haar", replica=replica)
        L.profile(passes)
        out.append(L)
    return out


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 6, 2, 14), (6, 10, 8, 8), (8, 8, 8, 8), (4, 16, 2, 32), (8, 8, 8, 10)])
@pytest.mark.parametrize("n_hb,n_or", [(1, 0), (1, 2), (0, 1)])
def test_one_launch_equals_passes(dims, n_hb, n_or):
    c, p = _pair(dims, replica=3)
    pc, ac = c.sweep_plaquette(1, n_hb, n_or, acc=True)
    pp, ap = p.sweep_plaquette(1, n_hb, n_or, acc=True)
    # the same draws, separately compiled: last-bit differences, which at most three sweeps magnify
    assert np.max(np.abs(c.download() - p.download())) <= 1e-10
    assert abs(pc - pp) <= 1e-12 and abs(pc - c.plaquette()) <= 1e-14
    assert abs(ac - ap) <= 1e-12


def test_runs_longer_than_one_launch():
    """1100 sub-sweeps are two launches: the field of 600 + 500, and the mean of their acceptances.  (With a
    plaquette the last sub-sweep is another code, so that only runs of the same blocks are the same.)"""
    a, b = (Lattice((4, 2, 6, 4), precision="fp64", beta=2.4, seed=5, start="haar") for _ in range(2))
    acc = a.sweep(1100, 1, 0, acc=True)
    a0, a1 = b.sweep(600, 1, 0, acc=True), b.sweep(500, 1, 0, acc=True)
    assert np.array_equal(a.download(), b.download())
    assert abs(acc - (600 * a0 + 500 * a1) / 1100) <= 1e-12
    ta, _ = a.graph_run(40, 30, 1, 0)
    tb = np.array([b.sweep_plaquette(30, 1, 0) for _ in range(40)])
    assert np.array_equal(ta, tb) and np.array_equal(a.download(), b.download())
