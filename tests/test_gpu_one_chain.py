"""One FP64 chain whatever runs it: sweeps of a handle (one cluster launch up to 4096 sites, checkerboard passes beyond or
when profiled), single passes, sweeps with the plaquette, uniform and mixed batches, per pass and persistent, give the
same field to the bit; FP32 the same but for the persistent form."""
import numpy as np
import pytest

from masterarbeit_b200 import Lattice
from masterarbeit_b200.su2g import Batch

pytestmark = pytest.mark.gpu

KW = {"beta": 2.4, "seed": 31, "start": "haar"}
N_HB, N_OR, SWEEPS = 1, 2, 3


def _handle(dims, precision, run, profile=False):
    L = Lattice(dims, precision=precision, replica=3, **KW)
    L.profile(profile)
    run(L)
    return L.download()


def _passes(L):
    for s in range(SWEEPS):
        for kind in [0] * N_HB + [1] * N_OR:
            for mu in range(4):
                for par in range(2):
                    L.update_pass(kind, mu, par, s)


def _batch(dims, precision, others, form):
    B = Batch([{"dims": d, "replica": 3 + i, **KW} for i, d in enumerate([dims] + others)], precision=precision)
    B.configure(*form)
    B.run(SWEEPS, N_HB, N_OR, 1)
    return B.download(0)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dims", [(4, 4, 4, 4), (6, 4, 4, 8), (8, 8, 8, 8), (8, 8, 8, 10), (14, 10, 12, 18)])
def test_every_form_gives_the_same_field(dims, precision):
    want = _handle(dims, precision, lambda L: L.sweep(SWEEPS, N_HB, N_OR))
    forms = {"profiled": _handle(dims, precision, lambda L: L.sweep(SWEEPS, N_HB, N_OR), profile=True),
             "passes": _handle(dims, precision, _passes),
             "plaquette": _handle(dims, precision, lambda L: L.sweep_plaquette(SWEEPS, N_HB, N_OR)),
             "loop": _handle(dims, precision, lambda L: L.graph_run(SWEEPS, 1, N_HB, N_OR)),
             "uniform": _batch(dims, precision, [dims], ("graph", 256)),
             "mixed": _batch(dims, precision, [(4, 2, 4, 6)], ("graph", 64))}
    if precision == "fp64":
        forms["persistent"] = _batch(dims, precision, [(4, 2, 4, 6)], ("persistent", 128))
    for name, got in forms.items():
        assert np.array_equal(got, want), name


@pytest.mark.parametrize("dims", [(4, 4, 4, 4), (8, 8, 8, 8), (8, 8, 8, 10)])
def test_heatbath_with_and_without_the_plaquette(dims):
    a = _handle(dims, "fp64", lambda L: L.sweep(2, 1, 0))
    assert np.array_equal(a, _handle(dims, "fp64", lambda L: L.sweep_plaquette(2, 1, 0)))
    assert np.array_equal(a, _handle(dims, "fp64", lambda L: [L.sweep_plaquette(1, 1, 0) for _ in range(2)]))


@pytest.mark.parametrize("n_hb,n_or", [(1024, 0), (24, 1000), (1024, 1), (25, 1000)])
def test_long_sweeps(n_hb, n_or):
    """A sweep of as many sub-sweeps as one cluster launch may run, and one more, which goes pass by pass."""
    def run(L):
        run.out = L.sweep_plaquette(1, n_hb, n_or, acc=True)

    a = _handle((4, 2, 4, 4), "fp64", run)
    pa = run.out
    b = _handle((4, 2, 4, 4), "fp64", run, profile=True)
    assert np.array_equal(a, b)
    # the same terms in the same order: at most the last bit of a warp's sum
    assert abs(pa[0] - run.out[0]) <= 1e-14 and abs(pa[1] - run.out[1]) <= 1e-14
