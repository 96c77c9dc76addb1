"""dQ/dU of the clover charge alone (no smearing step) against the oracle's central differences, on
geometries where its line gathering can go wrong: extents shorter than the 3-link lines, unequal
extents, and site counts that do not fill a CTA."""
import numpy as np
import pytest

import _oracle as O
from masterarbeit_b200 import Lattice
from test_gpu_adjoint import EPS, perturb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 4, 6, 2), (4, 6, 2, 10), (6, 2, 8, 4), (4, 4, 6, 6)])
def test_charge_gradient_against_the_oracle(dims):
    U = O.start(dims, "haar", 5)
    L = Lattice(dims, precision="fp64")
    L.upload(U)
    q, g = L.ape_qtop_vjp(0, 0.5)
    q0, scale = O.qtop(dims, U)
    assert abs(q - q0) <= 1e-12 * scale
    rng = np.random.default_rng(11)
    for _ in range(6):
        X = rng.standard_normal((U.shape[0], 4, 3))
        up, dn = (O.qtop(dims, np.ascontiguousarray(perturb(U, X, e)))[0] for e in (EPS, -EPS))
        # central difference: O(eps^2) truncation and a rounding of 1e-16 scale / eps, against the size of the terms
        bound = 1e-6 * max(abs(up - dn) / (2 * EPS), float(np.sqrt(np.sum((g * X) ** 2))))
        assert abs((up - dn) / (2 * EPS) - float(np.sum(g * X))) <= bound
    # FP32, the same gathering in its own precision: 24 products of rounding 2^-24 a term
    L32 = Lattice(dims, precision="fp32")
    L32.upload(U)
    _, g32 = L32.ape_qtop_vjp(0, 0.5)
    assert np.linalg.norm(g32 - g) <= 24 * 2.0 ** -23 * np.linalg.norm(g)
