"""The update passes link by link against the oracle, one lattice for each kernel the grid's size selects (kShapes), most
with a last CTA that is not full: heatbath and overrelaxation, with and without the plaquette, FP64 and FP32."""
import numpy as np
import pytest

import _oracle as O
from masterarbeit_b200 import Lattice

pytestmark = pytest.mark.gpu

BETA, SEED = 2.4, 77
# (dims, profiled): profiled small lattices take the passes instead of one cluster launch.  By CTAs of 128 links on 148 SMs:
LATTICES = [((2, 2, 2, 2), True),          # 1 CTA, 8 links
            ((8, 8, 8, 8), True),          # 16
            ((8, 8, 8, 10), False),        # 20, the smallest beyond the cluster launch
            ((14, 10, 12, 18), False),     # 119: two CTAs per SM
            ((18, 14, 18, 22), False),     # 390: three
            ((24, 14, 18, 22), False),     # 520: four
            ((18, 22, 20, 26), False),     # 805: six (FP32: one wave of eight)
            ((30, 34, 34, 34), False)]     # 4606, beyond L2 in FP64: eight


@pytest.fixture(scope="module", params=LATTICES, ids=lambda p: "x".join(map(str, p[0])))
def case(request):
    dims, profiled = request.param
    U = O.start(dims, "haar", 21).astype(np.float32).astype(np.float64)
    hb, ov = U.copy(), U.copy()
    acc = O.sweep(dims, hb, "hb", BETA, SEED, 4, 2)
    O.sweep(dims, ov, "or")
    return dims, profiled, U, {"hb": hb, "or": ov}, acc


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["hb", "or"])
def test_one_sweep_against_the_oracle(case, kind, precision):
    dims, profiled, U, want, ref_acc = case
    want, n = want[kind], (1, 0) if kind == "hb" else (0, 1)
    ref_plaq = O.plaquette(dims, want)
    L = Lattice(dims, precision=precision, beta=BETA, seed=SEED, start="cold", replica=2)
    L.profile(profiled)
    for plaq in (False, True):
        L.upload(U)
        L.set_sweep_counter(4)
        if plaq:
            p, acc = L.sweep_plaquette(1, *n, acc=True)
        else:
            p, acc = None, L.sweep(1, *n, acc=True)
        diff = np.abs(L.download() - want).max(axis=-1).ravel()
        if precision == "fp64":
            # u = 2^-53.  A staple is off by some 30 u, which enters divided by |A|, of which the smallest among 5 million
            # Haar sums is about 0.02, and once more divided by a neighbour's (0.1), in up to six of the passes
            assert diff.max() <= 1e-11, (plaq, diff.max())
            assert np.median(diff) <= 1e-14
            tol = 1e-13
        else:
            # u = 2^-24.  A few u typically.  The uniforms have 23 of the 32 bits: a small one (probability 1e-4) moves its
            # logarithm by 1e-3, and one accept test in 10^6 turns out otherwise, with all links that read that one
            assert np.median(diff) <= 3e-6, (plaq, np.median(diff))
            assert np.mean(diff > 1e-4) <= 1e-2 and np.mean(diff > 1e-2) <= 1e-3, plaq
            tol = 1e-5 + 2.0 / diff.size   # one other draw
        if kind == "hb":
            assert abs(acc - ref_acc) <= tol
        if plaq:
            assert abs(p - ref_plaq) <= tol
