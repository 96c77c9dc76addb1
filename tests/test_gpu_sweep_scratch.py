"""Scratch that a handle's sweeps take on the device."""
import pytest
import torch

from masterarbeit_b200 import Lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profile", [False, True])
def test_acceptance_alone_needs_no_plaquette_scratch(profile):
    """16 bytes for each warp of a pass (64 sites): 4 MB at 64^4, where plaquette and acceptance together take 16."""
    dims = (64, 64, 64, 64)
    K = Lattice(dims, precision="fp32", start="cold", beta=2.5)   # loads the kernels
    K.profile(profile)
    want = K.sweep_plaquette(1, 1, 0, acc=True)[1]
    K.sweep(1, 1, 0, acc=True)
    L = Lattice(dims, precision="fp32", start="cold", beta=2.5)
    L.profile(profile)
    before = torch.cuda.mem_get_info()[0]
    a = L.sweep(1, 1, 0, acc=True)
    assert before - torch.cuda.mem_get_info()[0] <= 8 << 20   # allocations come in pages of 2 MB
    assert a == want
