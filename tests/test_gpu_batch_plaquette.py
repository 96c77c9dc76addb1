"""The plaquette of a batch is its sites' sum without the rounding of intermediate sums: over links whose plaquettes and
site sums are exact in 64 bits, while a sum of 16 sites is not, the trace is the exact sum rounded once, over 6V."""
from fractions import Fraction

import numpy as np
import pytest

from masterarbeit_b200.su2g import Batch

pytestmark = pytest.mark.gpu

DIMS = [(4, 2, 2, 2), (2, 6, 4, 2), (4, 4, 4, 10)]   # one partial CTA, an uneven one, more than two CTAs


def _links(dims, rng):
    """c times the unit matrix, c = 1 + k / 2^12 (upload keeps links as they come)."""
    links = np.zeros((int(np.prod(dims)), 4, 4))
    links[:, :, 0] = 1.0 + rng.integers(0, 256, links.shape[:2]) / 4096.0
    return links


def _exact(dims, links):
    c = [[int(v) for v in row] for row in (links[:, :, 0] * 4096).astype(int)]
    n = np.arange(len(c)).reshape(dims)
    up = [np.roll(n, -1, axis=mu).reshape(-1) for mu in range(4)]
    total = sum(c[x][a] * c[up[a][x]][b] * c[up[b][x]][a] * c[x][b]
                for x in range(len(c)) for a in range(4) for b in range(a + 1, 4))
    return float(Fraction(total, 4096 ** 4)) / (6.0 * len(c))


@pytest.mark.parametrize("mode,block,more", [("graph", 64, 0), ("graph", 256, 0), ("graph", 128, 6400), ("persistent", 128, 0)])
@pytest.mark.parametrize("mixed", [False, True])
def test_the_trace_is_the_exact_sum_rounded(mode, block, more, mixed):
    """`more`: cold replicas that make the batch one of those launched pass by pass."""
    rng = np.random.default_rng(3)
    for dims in DIMS:
        if more and dims == (4, 4, 4, 10):
            continue
        reps = [dims] * 24 + [dims if not mixed else (4, 4, 4, 4)] * (1 + (more * 32 // int(np.prod(dims)) if more else 0))
        B = Batch([{"dims": d, "beta": 2.5, "seed": 1, "start": "cold"} for d in reps], precision="fp64")
        B.configure(mode, block)
        want = []
        for r in range(24):
            links = _links(dims, rng)
            B.upload(r, links)
            want.append(_exact(dims, links))
        trace, _ = B.run(1, 0, 0, 1)
        assert np.array_equal(trace[0][:24], np.array(want)), dims
        B.close()
