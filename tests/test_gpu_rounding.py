"""FP64 results are no less accurate than the same operations in plain 64-bit numpy, both against 80-bit arithmetic:
in-place smearing, and the gradient of the charge, whose terms cancel the more the field was smeared."""
import ctypes

import numpy as np
import pytest

import _oracle as O
import _reverse as X
from masterarbeit_b200 import Lattice, su2g
from test_zz_no_alloc import DeviceBuffer

pytestmark = pytest.mark.gpu

DIMS = (8, 6, 8, 10)


def _field(seed):
    """A plaquette like that of a thermalised field (0.73) and a charge (constant fluxes through two planes), in a random
    gauge."""
    rng = np.random.default_rng(seed)

    def unit(q):
        return q / np.sqrt((q * q).sum(0))
    g = unit(rng.standard_normal((4, *DIMS)))
    n = np.indices(DIMS)
    out = []
    for mu in range(4):
        u = 0.23 * rng.standard_normal((4, *DIMS))
        u[0] += 1.0
        a, b = (0, 1) if mu < 2 else (2, 3)
        if mu == b:
            angle = 2 * np.pi / (DIMS[a] * DIMS[b]) * n[a]
        else:
            angle = -2 * np.pi / DIMS[b] * n[b] * (n[a] == DIMS[a] - 1)
        u = X.qmul(unit(u), np.stack((np.cos(angle), 0 * angle, 0 * angle, np.sin(angle))))
        out.append(X.qmul(X.qmul(g, u), X.qdag(np.roll(g, -1, 1 + mu))))
    return np.ascontiguousarray(X.host(out))


def _rms(a, exact):
    return float(np.sqrt(((a - exact) ** 2).mean() / (exact ** 2).mean()))


@pytest.mark.parametrize("mode", ["all", "spatial", "temporal"])
def test_in_place_smearing(mode):
    U = _field(1)
    exact = X.smeared(U, DIMS, 10, 0.5, mode, np.longdouble)
    plain = _rms(X.smeared(U, DIMS, 10, 0.5, mode, np.float64), exact)
    lib, got = su2g.load(), np.empty_like(U)
    buf = DeviceBuffer(U.nbytes)
    assert buf.rt.cudaMemcpy(buf.ptr, U.ctypes.data, U.nbytes, 1) == 0
    assert lib.su2g_ape_inplace_noalloc(buf.ptr, (ctypes.c_int32 * 4)(*DIMS), 10, 0.5, su2g.APE[mode], None) == 0
    assert buf.rt.cudaDeviceSynchronize() == 0
    assert buf.rt.cudaMemcpy(got.ctypes.data, buf.ptr, U.nbytes, 2) == 0
    buf.free()
    # 61 thousand numbers: two such rms differ by a percent by chance; the projection takes the reciprocal of a root instead
    # of a division (one rounding more of some fifteen)
    assert _rms(got, exact) <= 1.08 * plain, plain


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("n_ape", [0, 1, 10])
def test_gradient_of_the_charge(n_ape, seed):
    U = _field(seed)
    exact = X.charge_gradient(U, DIMS, n_ape, 0.5, np.longdouble)
    plain = _rms(X.charge_gradient(U, DIMS, n_ape, 0.5, np.float64), exact)
    L = Lattice(DIMS, precision="fp64", start="cold")
    L.upload(U)
    assert _rms(L.ape_qtop_vjp(n_ape, 0.5)[1], exact) <= plain, plain
