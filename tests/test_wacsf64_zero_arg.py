"""FP64 descriptor kernels (wacsf64.cu) where an exponential's argument is zero
or next to it: functions of exponent 0 (types 1, 2, 4), and type 3 with
neighbours at R_s, exactly (a lattice, a dimer) and a few nanoangstroms off.
Tolerances are those of the kernels' other comparisons."""
import numpy as np
import pytest

from helpers import three_species_cell, write_model_file

pytestmark = pytest.mark.gpu

ZS, WS = np.array([13, 28, 40], np.int32), np.array([1.3, -0.8, 2.0])
TYPES = [1, 2, 4, 2, 1, 3, 3]
ALPHAS = [0.0, 0.0, 0.0, 0.01, 0.3, 2.0, 1.0]
ZETAS = [1.0, 1.0, 2.0, 2.0, 1.0, 1.0, 1.0]


def _cells():
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2.0
    yield np.eye(3) * 8.0, g, ZS[np.arange(64) % 3]
    yield three_species_cell(2)
    for d in (0.0, 1e-9, -1e-9, 3e-9, -3e-9, 5e-9, 1e-8, -1e-8):
        yield (np.eye(3) * 30.0, np.array([[1.0, 2.0, 3.0], [3.0 + d, 2.0, 3.0]]),
               np.array([28, 40], np.int32))


def _arrays(M):
    rng = np.random.default_rng(5)
    D = 2 * len(TYPES)
    return (ZS, WS, np.array(TYPES, np.int32), np.array(ALPHAS), np.full(len(TYPES), 6.0),
            rng.uniform(20.0, 60.0, D), rng.normal(0.0, 10.0, (M, D)), rng.normal(0.0, 0.1, M),
            np.array(ZETAS))


def test_zero_arguments_match_the_oracle(tmp_path, gapgb_mod, oracle_mod):
    path = write_model_file(str(tmp_path / "gap_parameters"), *_arrays(24))
    m, om = gapgb_mod.GapModel.load(path), oracle_mod.Model(path)
    for lat, pos, z in _cells():
        E, F, S, _ = m.eval(z, lat, pos)
        oE, oF, oS, _, ex = oracle_mod.gap_calc(om, z, lat, pos, 6.0, True, extras=True)
        X = m.descriptors([0, len(z)], z, lat[None], pos)
        assert np.abs(X - ex["xx"]).max() <= 1e-13 * max(1.0, np.abs(ex["xx"]).max())
        assert abs(E - oE) <= 1e-11 * max(1.0, abs(oE))
        assert np.abs(F - oF).max() <= 1e-11 * max(1.0, np.abs(oF).max())
        assert np.abs(S - oS).max() <= 1e-10 * max(1.0, np.abs(oS).max())
    m.close()


def test_force_rows_of_the_fit(gapgb_mod, oracle_mod, tmp_path):
    """The fit's Jacobians: its coefficients against normal equations whose
    rows are the oracle's energies and forces with unit coefficients."""
    import gapgb.synth as S
    M, se, sf, jit = 5, 2e-2, 0.1, 1e-6
    zs, ws, ty, al, rc, theta, mm, _, ze = _arrays(M)
    structs = [three_species_cell(2), list(_cells())[0]]
    batch = S.pack(structs)
    off, N = batch[0], int(batch[0][-1])
    phi, pf = np.zeros((2, M)), np.zeros((3 * N, M))
    for k in range(M):
        path = write_model_file(str(tmp_path / ("unit%d" % k)), zs, ws, ty, al, rc, theta, mm,
                                np.eye(M)[k], ze)
        om = oracle_mod.Model(path)
        for s, (lat, pos, z) in enumerate(structs):
            phi[s, k], f = oracle_mod.gap_calc(om, z, lat, pos, 6.0, True)[:2]
            pf[3 * off[s]:3 * off[s + 1], k] = f.reshape(-1)
    m = gapgb_mod.GapModel.create(zs, ws, ty, al, rc, theta, mm, np.zeros(M), sf_zeta=ze)
    rng = np.random.default_rng(1)
    E, F = rng.normal(-3.0, 0.1, 2), rng.normal(0.0, 0.5, (N, 3))
    x = (mm[:, None, :] - mm[None, :, :]) / theta
    w = 1.0 / (se ** 2 * np.diff(off))
    A = (np.exp(-0.5 * (x ** 2).sum(-1)) + jit * np.eye(M) + (phi * w[:, None]).T @ phi +
         pf.T @ pf / sf ** 2)
    b = (phi * w[:, None]).T @ E + pf.T @ F.reshape(-1) / sf ** 2
    c = m.fit(*batch, E, forces=F, sigma_e=se, sigma_f=sf, jitter=jit)
    # rounding of the rows themselves (1e-13 of the largest) bounds the residual
    res = np.linalg.norm(A @ c - b) / (np.linalg.norm(A) * np.linalg.norm(c) + np.linalg.norm(b))
    assert res <= 1e-11
    m.close()
