"""Precision of the FP64 descriptor kernels (wacsf64.cu) where their fixed-point
units are coarse: clusters of atoms much closer than the longest cutoff, a
cutoff far below the longest, steep exponents.  Descriptors against the oracle
to a few roundings of 1.1e-16 of each function's largest value (arguments of
the exponentials are at most about 5 here), forces to the cancellation of
their 1/r^2 terms."""
import numpy as np
import pytest

from helpers import write_model_file

pytestmark = pytest.mark.gpu

ZS, WS = np.array([13, 28, 40], np.int32), np.array([1.3, 0.8, 2.0])
# atoms, closest distance, box (A); steepest exponents
CLUSTERS = {"0.3": (20, 0.3, 1.5, 1.0), "0.1": (20, 0.1, 0.5, 10.0), "0.03": (16, 0.03, 0.14, 160.0),
            "0.005": (12, 0.005, 0.02, 4000.0)}


def _cluster(n, dmin, box, seed):
    rng, p = np.random.default_rng(seed), []
    while len(p) < n:
        x = rng.random(3) * box
        if all(np.linalg.norm(x - y) >= dmin for y in p):
            p.append(x)
    return np.eye(3) * 60.0, np.array(p) + 17.0, ZS[np.arange(n) % 3]


@pytest.mark.parametrize("rcut", [6.0, 12.0])
@pytest.mark.parametrize("which", sorted(CLUSTERS))
def test_close_atoms(which, rcut, tmp_path, gapgb_mod, oracle_mod):
    n, dmin, box, steep = CLUSTERS[which]
    ty, al, rc, ze = [1, 1, 3], [0.1, steep, 1.0], [rcut, rcut, rcut], [1.0] * 3
    for c, a in ((rcut, 0.01), (rcut, steep), (2.5 * box, 0.01)):
        for t, z in ((2, 1.0), (4, 1.0), (2, 2.0), (4, 4.0)):
            ty.append(t), al.append(a), rc.append(c), ze.append(z)
    D = 2 * len(ty)
    args = (ZS, WS, np.array(ty, np.int32), np.array(al), np.array(rc))
    cells = [_cluster(n, dmin, box, s) for s in range(3)]
    X = []
    path = write_model_file(str(tmp_path / "probe"), *args, np.ones(D), np.zeros((1, D)),
                            np.zeros(1), np.array(ze))
    m, om = gapgb_mod.GapModel.load(path, rcut), oracle_mod.Model(path)
    for lat, pos, z in cells:
        ex = oracle_mod.gap_calc(om, z, lat, pos, rcut, False, extras=True)[-1]
        x = m.descriptors([0, n], z, lat[None], pos)
        X.append(ex["xx"])
        assert (np.abs(x - ex["xx"]).max(0) <= 2e-15 * np.abs(ex["xx"]).max(0)).all()
    m.close()
    X = np.concatenate(X)
    theta = np.where(X.std(0) > 0, 3.0 * X.std(0), 1.0)
    path = write_model_file(str(tmp_path / "gap_parameters"), *args, theta, X[:8],
                            np.linspace(-1.0, 1.0, 8), np.array(ze))
    m, om = gapgb_mod.GapModel.load(path, rcut), oracle_mod.Model(path)
    for lat, pos, z in cells:
        E, F, S, _ = m.eval(z, lat, pos)
        oE, oF, oS, _ = oracle_mod.gap_calc(om, z, lat, pos, rcut, True)
        assert abs(E - oE) <= 1e-12 * len(z)
        assert np.abs(F - oF).max() <= 1e-11 * np.abs(oF).max()
        assert np.abs(S - oS).max() <= 1e-11 * np.abs(oS).max()
    m.close()
