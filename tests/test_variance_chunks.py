"""K image of the tensor-core variance (variance.cu): blocks of two and three
chunks of points (the last one short), components below and beyond the 64 that
stay staged.  A cell's covf is the same bits in a large batch as alone, where a
block takes one chunk."""
import numpy as np
import pytest

import gapgb.synth as S
from test_gpr64 import WS, ZS, _sf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsf,prec", [(12, "tc"), (36, "fp32")])
@pytest.mark.parametrize("ncells", [20, 30])
def test_cells_in_a_batch_and_alone(gapgb_mod, ncells, nsf, prec):
    ty, al, rc, ze = _sf(nsf)
    D, M = 2 * nsf, 1000
    cells = [S.alloy512(seed=s) for s in range(ncells)]
    args = (ZS, WS, ty, al, rc)
    probe = gapgb_mod.GapModel.create(*args, np.ones(D), np.zeros((1, D)), np.zeros(1), sf_zeta=ze)
    X = probe.descriptors(*S.pack(cells[:4]))
    probe.close()
    rng = np.random.default_rng(ncells)
    sd = X.std(0)
    theta = np.where(sd > 0, sd, 1.0)
    m = gapgb_mod.GapModel.create(*args, theta, X[rng.choice(len(X), M, replace=False)],
                                  np.ones(M), sf_zeta=ze)
    m.set_precision(prec)
    A = rng.normal(0.0, 0.03, (M, M))
    m.set_qmm(A @ A.T / M)
    off, sp, lat, pos = S.pack(cells)
    covf, var = m.variance(off, sp, lat, pos)
    for s in (0, ncells // 2, ncells - 1):
        c1, v1 = m.variance(*S.pack([cells[s]]))
        np.testing.assert_array_equal(c1, covf[off[s]:off[s + 1]])
        np.testing.assert_array_equal(v1, var[s:s + 1])
    m.close()
