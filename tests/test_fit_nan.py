"""A fit whose descriptors are not numbers (a steeply growing exponential times
a vanishing angular factor) reports it instead of leaving the atoms out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_nan_descriptors_are_reported(gapgb_mod):
    z = np.array([14], np.int32)
    ty, al = np.array([1, 2], np.int32), np.array([0.1, -500.0])
    m = gapgb_mod.GapModel.create(z, np.ones(1), ty, al, np.full(2, 6.0), np.ones(4),
                                  np.array([[0.1] * 4, [0.3] * 4]), np.zeros(2))
    # a straight chain: 1 + cos = 0 at its middle atom
    pos = np.array([[3.0, 1.0, 1.0], [5.0, 1.0, 1.0], [7.0, 1.0, 1.0]])
    batch = [0, 3], np.full(3, 14, np.int32), np.eye(3)[None] * 40.0, pos
    assert np.isnan(m.descriptors(*batch)).any()
    before = m.arrays()[2].copy()
    with pytest.raises(gapgb_mod.GapError):
        m.fit_energies(*batch, np.array([-1.0]), sigma_e=1e-2, jitter=1e-6)
    assert np.array_equal(m.arrays()[2], before)
    m.close()
