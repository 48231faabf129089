"""Neighbour lists of cells narrower than twice the cutoff (several images per
candidate) whose atoms lie on the FP32 screen's bound, rcut + 2.5e-4 sum|L| +
1e-3, to a few units in the last place of the squared distance: candidates there
are no neighbours, and nothing else may be taken for one."""
import numpy as np
import pytest

from helpers import write_model_file

pytestmark = pytest.mark.gpu


def _cells(count):
    rng = np.random.default_rng(4)
    out = []
    for _ in range(count):
        lat = np.diag([7.3, 8.1, 29.0]) + rng.normal(0.0, 0.4, (3, 3))
        bound = 6.0 + 2.5e-4 * np.abs(lat).sum() + 1e-3
        u = np.array([0.0, 0.0, 1.0]) + rng.normal(0.0, 0.15, 3)
        u /= np.linalg.norm(u)
        a = np.array([0.3, 0.2, 4.0]) + rng.random(3)
        # a third atom makes a real neighbour; the fourth is on the bound again
        pos = np.stack([a, a + u * (bound + rng.uniform(-6e-6, 6e-6)), a + [1.9, 0.3, 0.4],
                        a - u * (bound + rng.uniform(-6e-6, 6e-6))])
        out.append((lat, pos, np.array([14, 14, 32, 32], np.int32)))
    return out


@pytest.mark.parametrize("precision", ["fp64", "tc"])
def test_candidates_on_the_screens_bound(precision, tmp_path, gapgb_mod, oracle_mod):
    import gapgb.synth as S
    ty, al, rc, ze = [1, 1, 2, 4], [0.02, 0.3, 0.01, 0.01], [6.0] * 4, [1.0] * 4
    rng = np.random.default_rng(1)
    path = write_model_file(str(tmp_path / "gap_parameters"), np.array([14, 32], np.int32),
                            np.array([1.0, 2.0]), np.array(ty, np.int32), np.array(al), np.array(rc),
                            np.full(8, 5.0), rng.normal(3.0, 2.0, (6, 8)), rng.normal(0.0, 1.0, 6),
                            np.array(ze))
    m, om = gapgb_mod.GapModel.load(path), oracle_mod.Model(path)
    m.set_precision(precision)
    cells = _cells(3000)
    E, F, _ = m.eval_batch(*S.pack(cells))
    tol = 1e-11 if precision == "fp64" else 1e-4
    for s, (lat, pos, z) in enumerate(cells):
        oE, oF = oracle_mod.gap_calc(om, z, lat, pos, 6.0, True)[:2]
        assert abs(E[s] - oE) <= tol * max(1.0, abs(oE))
        assert np.abs(F[4 * s:4 * s + 4] - oF).max() <= 10 * tol * max(1.0, np.abs(oF).max())
    m.close()
