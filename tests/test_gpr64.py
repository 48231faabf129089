"""FP64 GPR on the tensor cores (gpr64_tc.cu): edges of its tiles (rows of 128
atoms, 32 sparse points, 128 points between drains, components 64 / 80),
coefficients of every size and sign, points and atoms far out, and the models
it leaves to the CUDA-core kernel (D > 80; scaled points beyond 2^6)."""
import numpy as np
import pytest

from helpers import three_species_cell, write_model_file

pytestmark = pytest.mark.gpu


def _sf(nsf):
    """nsf symmetry functions: radial ones, the last few angular."""
    nang = 0 if nsf < 4 else 4
    ty = [1] * (nsf - nang) + [2, 4, 2, 4][:nang]
    al = list(np.geomspace(0.004, 1.0, nsf - nang)) + [0.005, 0.005, 0.05, 0.05][:nang]
    return (np.array(ty, np.int32), np.array(al), np.full(nsf, 6.0),
            np.array([1.0] * (nsf - nang) + [1.0, 1.0, 2.0, 4.0][:nang]))


ZS, WS = np.array([13, 28, 40], np.int32), np.array([13.0, 28.0, 40.0])


def _cells(count):
    return [three_species_cell(s) for s in range(count)]


def _pack(cells):
    off = np.cumsum([0] + [len(z) for _, _, z in cells]).astype(np.int32)
    return (off, np.concatenate([z for _, _, z in cells]), np.stack([l for l, _, _ in cells]),
            np.concatenate([p for _, p, _ in cells]))


def _model(tmp_path, gapgb_mod, nsf, M, scale=1.0, stretch=1.0, seed=0):
    ty, al, rc, ze = _sf(nsf)
    D = 2 * nsf
    probe = gapgb_mod.GapModel.create(ZS, WS, ty, al, rc, np.ones(D), np.zeros((1, D)), np.zeros(1),
                                      sf_zeta=ze)
    X = probe.descriptors(*_pack(_cells(10)))
    probe.close()
    rng = np.random.default_rng(seed)
    mm = X[rng.choice(len(X), size=M, replace=len(X) < M)].copy()
    sd = X.std(0)
    theta = np.where(sd > 0, scale * sd, 1.0)
    theta[0] /= stretch
    if M > 2:
        mm[1] += 30.0 * theta  # a point far from every atom
    # from 1e-8 to 1e2, both signs, and zeros
    c = rng.choice([-1.0, 1.0], M) * 10.0 ** rng.uniform(-8, 2, M)
    c[rng.random(M) < 0.1] = 0.0
    c[0] = 1.0
    path = write_model_file(str(tmp_path / "gap_parameters"), ZS, WS, ty, al, rc, theta, mm, c, ze)
    return path, gapgb_mod.GapModel.load(path), np.abs(c).sum()


def _check(path, m, csum, oracle_mod, count, mixed):
    om = oracle_mod.Model(path)
    cells = _cells(count)
    lat, pos, z = cells[0]
    pos = pos.copy()
    pos[0] = pos[1] + np.array([1.1, 0.1, 0.0])  # an atom outside the points' range
    cells[0] = (lat, pos, z)
    if mixed:
        m.set_precision("mixed")
    off, sp, la, po = _pack(cells)
    E, F, S, e = m.eval_batch(off, sp, la, po, atom_energy=True)
    te, tf = (1e-12, 1e-10) if not mixed else (1e-4, 1e-3)
    for s, (lat, pos, z) in enumerate(cells):
        oE, oF, oS, _, ex = oracle_mod.gap_calc(om, z, lat, pos, 6.0, True, extras=True)
        a, b = off[s], off[s + 1]
        assert np.abs(e[a:b] - ex["e"]).max() <= te * csum
        assert abs(E[s] - oE) <= te * csum * len(z)
        assert np.abs(F[a:b] - oF).max() <= tf * csum * max(1.0, np.abs(oF).max() / csum)


@pytest.mark.parametrize("nsf,M,cells", [(1, 1, 1), (8, 31, 4), (32, 32, 4), (32, 33, 5),
                                         (33, 127, 4), (32, 129, 9), (40, 300, 4), (40, 161, 12),
                                         (41, 130, 3)])
@pytest.mark.parametrize("mixed", [False, True])
def test_tiles_match_the_oracle(nsf, M, cells, mixed, tmp_path, gapgb_mod, oracle_mod):
    path, m, csum = _model(tmp_path, gapgb_mod, nsf, M)
    _check(path, m, csum, oracle_mod, cells, mixed)
    m.close()


def test_wide_points_and_new_coefficients(tmp_path, gapgb_mod, oracle_mod):
    """A component whose scaled spread passes 2^6 (the CUDA-core kernel), and
    coefficients replaced on a model that has its images."""
    path, m, csum = _model(tmp_path, gapgb_mod, 32, 140, stretch=500.0)
    _check(path, m, csum, oracle_mod, 2, False)
    m.close()
    path, m, csum = _model(tmp_path, gapgb_mod, 32, 140)
    m.eval(*[v[0] if k == 1 else v for k, v in enumerate(_pack(_cells(1))[1:])])
    c = np.random.default_rng(9).normal(0.0, 1.0, 140)
    m.set_coeff(c)
    m.save(str(tmp_path / "again"))
    _check(str(tmp_path / "again"), m, np.abs(c).sum(), oracle_mod, 2, False)
    m.close()


def test_energies_do_not_depend_on_the_batch(tmp_path, gapgb_mod):
    """The split over sparse points follows the batch size; sums are integers."""
    _, m, _ = _model(tmp_path, gapgb_mod, 32, 300)
    cells = _cells(60)
    off, sp, la, po = _pack(cells)
    E, F, S, e = m.eval_batch(off, sp, la, po, atom_energy=True)
    E1, F1, S1, e1 = m.eval_batch(off[:2], sp[:off[1]], la[:1], po[:off[1]], atom_energy=True)
    assert np.array_equal(e1, e[:off[1]]) and np.array_equal(F1, F[:off[1]])
    m.close()
