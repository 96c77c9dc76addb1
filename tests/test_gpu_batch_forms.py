"""Every form a batch runs in -- uniform or mixed extents, a captured block or launches pass by pass (more than
640 links a pass and SM), all CTA widths, the last CTA of a replica part-filled -- against handles of the same replicas."""
import numpy as np
import pytest

from masterarbeit_b200 import Lattice
from masterarbeit_b200.su2g import Batch

pytestmark = pytest.mark.gpu

U, M = (6, 10, 4, 14), (8, 6, 4, 10)   # 1680 and 960 links a pass
FORMS = {"uniform small": [U] * 5, "uniform large": [U] * 60, "mixed small": [U, M, (2, 2, 2, 2), (4, 2, 6, 4), U],
         "mixed large": [M, U] * 36 + [(2, 2, 2, 2), U, (16, 10, 12, 14)]}


@pytest.mark.parametrize("block", [64, 128, 256])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("form", FORMS)
def test_fields_and_traces(form, precision, block):
    reps = [{"dims": d, "beta": 2.2 + 0.01 * i, "seed": 50 + i, "replica": 7 * i, "start": "haar" if i % 3 else "cold"}
            for i, d in enumerate(FORMS[form])]
    B = Batch(reps, precision=precision)
    B.configure("graph", block)
    trace = np.concatenate([B.run(2, 1, 1, 1)[0], B.run(2, 2, 1, 2)[0]])
    n = len(reps)
    for i in sorted({0, 1, 2, n // 2, n - 3, n - 2, n - 1}):
        r = dict(reps[i])
        L = Lattice(r.pop("dims"), precision=precision, **r)
        want = [L.sweep(1, 1, 1) or L.plaquette() for _ in range(2)]
        L.sweep(2, 2, 1)
        want.append(L.plaquette())
        # the same kernels' arithmetic to the bit; a plaquette summed in another order
        assert np.array_equal(B.download(i), L.download()), i
        assert np.max(np.abs(trace[:, i] - want)) <= 1e-14, i
        L.close()
    B.close()
