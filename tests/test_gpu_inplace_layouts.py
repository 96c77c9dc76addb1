"""su2g_ape_inplace_noalloc keeps its intermediate levels in other layouts than the caller's field:
every number of steps around the first, second and last one, every mode, and a field that is only
16-byte aligned (which stays in its own layout), against the oracle."""
import ctypes

import numpy as np
import pytest

import _oracle as O
from masterarbeit_b200 import su2g
from test_zz_no_alloc import DeviceBuffer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 16])
@pytest.mark.parametrize("mode", ["all", "spatial", "temporal"])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (4, 6, 2, 10), (6, 4, 8, 4)])
def test_every_step_count(dims, mode, offset):
    lib = su2g.load()
    U = O.start(dims, "haar", 9)
    cdims = (ctypes.c_int32 * 4)(*dims)
    buf = DeviceBuffer(U.nbytes + 32)
    at = ctypes.c_void_p(buf.ptr.value + offset)
    got = np.empty_like(U)
    for ns in (1, 2, 3, 4, 5):
        assert buf.rt.cudaMemcpy(at, U.ctypes.data, U.nbytes, 1) == 0
        assert lib.su2g_ape_inplace_noalloc(at, cdims, ns, 0.5, su2g.APE[mode], None) == 0
        assert buf.rt.cudaDeviceSynchronize() == 0
        assert buf.rt.cudaMemcpy(got.ctypes.data, at, U.nbytes, 2) == 0
        # FP64, as the handle's smearing against the oracle: 1e-13 a link
        assert np.max(np.abs(got - O.ape(dims, U, ns, 0.5, mode))) <= 1e-13, ns
    buf.free()
