"""Fixed-point geometry and exponentials of the FP64 descriptor kernels
(wacsf64.cu): exponents from nothing to past the underflow and of either sign,
cutoffs that are powers of two or far apart, and a lattice with pairs exactly
at the cutoffs.  Tolerances are those of the kernels' other comparisons: a few
hundred roundings of 1.1e-16 on sums of at most 2000 terms of one sign."""
import numpy as np
import pytest

from helpers import three_species_cell, write_model_file

pytestmark = pytest.mark.gpu


def _lattice():
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2.0
    return np.eye(3) * 8.0, g, np.array([13, 28, 40], np.int32)[np.arange(64) % 3]


@pytest.mark.parametrize("alpha", [1e-12, 1e-5, 0.004, 0.25, 6.0, 40.0, -0.002])
@pytest.mark.parametrize("cutoffs", [(6.0, 4.0), (8.0,), (5.3, 1.9), (2.0,)])
def test_exponents_and_cutoffs_match_the_oracle(alpha, cutoffs, tmp_path, gapgb_mod, oracle_mod):
    ty, al, rc, ze = [1, 3], [abs(alpha), 1.7], [cutoffs[0]] * 2, [1.0, 1.0]
    for c in cutoffs:
        for t in (2, 4):
            ty.append(t), al.append(alpha), rc.append(c), ze.append(2.0)
    zs, ws = np.array([13, 28, 40], np.int32), np.array([1.3, -0.8, 2.0])
    rng = np.random.default_rng(5)
    D, M = 2 * len(ty), 24
    path = write_model_file(str(tmp_path / "gap_parameters"), zs, ws, np.array(ty, np.int32),
                            np.array(al), np.array(rc), rng.uniform(20.0, 60.0, D),
                            rng.normal(0.0, 10.0, (M, D)), rng.normal(0.0, 0.1, M), np.array(ze))
    m, om = gapgb_mod.GapModel.load(path), oracle_mod.Model(path)
    for lat, pos, z in (three_species_cell(1), _lattice()):
        E, F, S, _ = m.eval(z, lat, pos)
        oE, oF, oS, _, ex = oracle_mod.gap_calc(om, z, lat, pos, 6.0, True, extras=True)
        X = m.descriptors([0, len(z)], z, lat[None], pos)
        assert np.abs(X - ex["xx"]).max() <= 1e-13 * max(1.0, np.abs(ex["xx"]).max())
        assert abs(E - oE) <= 1e-11 * max(1.0, abs(oE))
        assert np.abs(F - oF).max() <= 1e-11 * max(1.0, np.abs(oF).max())
        assert np.abs(S - oS).max() <= 1e-10 * max(1.0, np.abs(oS).max())
    m.close()
