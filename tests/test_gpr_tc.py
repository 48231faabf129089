"""Tensor-core GPR (gpr_tc.cu): numbers of sparse-point tiles (64) around its
three C1 buffers, its five-tile ring, the three slots of partial sums and an
odd or even last tile, and ragged atom rows (128), against the FP64 form.

Tolerance: the dropped product of the two low BF16 parts is below 2^-18 |x||m|
in the exponent, |x||m| < 70 in units of theta here, so each w is within 3e-4
of its value (the other roundings are smaller), and e within 3e-4 of sum |c|.
The forces' sums keep a cancellation of at most about 30: 1e-2 in the norm."""
import numpy as np
import pytest

from test_gpr64 import WS, ZS, _cells, _pack, _sf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 13])
@pytest.mark.parametrize("M", [1, 63, 64, 65, 128, 129, 192, 256, 257, 320, 384, 385, 449, 833])
def test_tile_counts_match_fp64(gapgb_mod, M, count):
    ty, al, rc, ze = _sf(12)
    args = (ZS, WS, ty, al, rc)
    probe = gapgb_mod.GapModel.create(*args, np.ones(24), np.zeros((1, 24)), np.zeros(1), sf_zeta=ze)
    X = probe.descriptors(*_pack(_cells(14)))
    probe.close()
    rng = np.random.default_rng(M)
    mm = X[rng.choice(len(X), size=M, replace=len(X) < M)]
    sd = X.std(0)
    theta = np.where(sd > 0, sd, 1.0)
    c = rng.uniform(0.5, 1.5, M)
    m = gapgb_mod.GapModel.create(*args, theta, mm, c, sf_zeta=ze)
    off, sp, la, po = _pack(_cells(count))
    want = m.eval_batch(off, sp, la, po, atom_energy=True)
    m.set_precision("tc")
    got = m.eval_batch(off, sp, la, po, atom_energy=True)
    again = m.eval_batch(off, sp, la, po, atom_energy=True)
    m.close()
    assert np.abs(got[3] - want[3]).max() <= 3e-4 * c.sum()
    assert np.linalg.norm(got[1] - want[1]) <= 1e-2 * np.linalg.norm(want[1])
    np.testing.assert_array_equal(got[3], again[3])
