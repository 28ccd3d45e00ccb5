"""The one-pass gradient digestion where its index arithmetic is longest: g and
h shells (auxiliary blocks up to l = 6), blocks of one element, single lanes."""
import numpy as np
import pytest

from intception_b200 import jk


@pytest.mark.gpu
@pytest.mark.parametrize('shells', [((0, 1),), ((0, 2), (4, 1)), ((1, 2), (5, 1))])
def test_one_pass_digestion_equals_per_batch_launches(shells):
    """Both digest the same auxiliary blocks; they differ by the rounding of the
    sums (1e3-1e5 terms a component, 1e-16 of the largest each)."""
    sys_, xyz = jk.lattice_system(natom=2, seed=5, shells=shells, alpha=(0.2, 5.0), nocc=3, screen=1e-18)
    g = sys_.gradient(xyz).cpu().numpy()
    sys_.per_batch_digestion = True
    ref = sys_.gradient(xyz).cpu().numpy()
    assert np.abs(g - ref).max() <= 1e-11 * max(1e-3, np.abs(ref).max())
    assert np.abs(ref).max() > 0.0
