"""FP64 descriptor kernels (wacsf64.cu): every template size, several cutoffs,
remainders of the pair units, atoms without neighbours or with one, and the
same bits alone (atoms split over blocks) as inside a large batch."""
import numpy as np
import pytest

from helpers import three_species_cell, write_model_file

pytestmark = pytest.mark.gpu


def _sf(nal, zetas, cutoffs, types=(2, 4)):
    ty, al, rc, ze = [1, 1, 3], [0.01, 0.7, 2.5], [max(cutoffs), 4.5, max(cutoffs)], [1.0] * 3
    for c in cutoffs:
        for a in np.geomspace(0.004, 0.3, nal):
            for z in zetas:
                for t in types:
                    ty.append(t), al.append(float(a)), rc.append(c), ze.append(float(z))
    return np.array(ty, np.int32), np.array(al), np.array(rc), np.array(ze)


# (alphas, zetas, cutoffs): template sizes 1/2/4 x degree 1/2/4, one to three
# cutoffs; the last two sets keep the generic kernels (zeta 5; five alphas)
SETS = [(1, (1,), (6.0,)), (2, (1,), (6.0, 3.0, 1.5)), (4, (1,), (5.0,)),
        (1, (1, 2), (6.0,)), (2, (2,), (6.0, 4.0)), (3, (1, 2), (5.5,)),
        (1, (1, 3), (6.0,)), (2, (1, 2, 4), (6.0, 3.5)), (4, (1, 2, 3, 4), (6.0,)),
        (1, (1, 5), (6.0,)), (5, (1,), (6.0,))]


def _cells():
    rng = np.random.default_rng(3)
    lone = (np.eye(3) * 30.0, np.array([[1.0, 2.0, 3.0]]), np.array([13], np.int32))
    pair = (np.eye(3) * 30.0, np.array([[1.0, 2.0, 3.0], [3.1, 2.2, 3.0]]), np.array([28, 40], np.int32))
    dense = rng.random((20, 3))
    dense = (np.diag([7.1, 6.6, 5.2]) + rng.normal(0, 0.3, (3, 3)),
             None, np.array([13, 28, 40], np.int32)[np.arange(20) % 3])
    grid = np.stack(np.meshgrid(np.arange(3), np.arange(3), np.arange(3), indexing="ij"), -1)
    frac = (grid.reshape(-1, 3)[:20] + 0.5 + rng.normal(0, 0.05, (20, 3))) / 3.0
    dense = (dense[0], frac @ dense[0], dense[2])
    return [lone, pair, three_species_cell(1), dense]


def _model(tmp_path, gapgb_mod, sf, seed=0):
    ty, al, rc, ze = sf
    rng = np.random.default_rng(seed)
    D, M = 2 * len(ty), 24
    if D > 128:
        raise AssertionError("test set too long")
    zs, ws = np.array([13, 28, 40], np.int32), np.array([1.3, -0.8, 2.0])
    theta = rng.uniform(20.0, 60.0, D)
    mm = rng.normal(0.0, 10.0, (M, D))
    path = write_model_file(str(tmp_path / "gap_parameters"), zs, ws, ty, al, rc, theta, mm,
                            rng.normal(0.0, 0.1, M), ze)
    return path, gapgb_mod.GapModel.load(path)


@pytest.mark.parametrize("k", range(len(SETS)))
def test_sets_match_the_oracle(k, tmp_path, gapgb_mod, oracle_mod):
    path, m = _model(tmp_path, gapgb_mod, _sf(*SETS[k]))
    om = oracle_mod.Model(path)
    for lat, pos, z in _cells():
        E, F, S, _ = m.eval(z, lat, pos)
        oE, oF, oS, _, ex = oracle_mod.gap_calc(om, z, lat, pos, 6.0, True, extras=True)
        X = m.descriptors([0, len(z)], z, lat[None], pos)
        scale = max(1.0, np.abs(ex["xx"]).max())
        assert np.abs(X - ex["xx"]).max() <= 1e-13 * scale
        assert abs(E - oE) <= 1e-11 * max(1.0, abs(oE))
        assert np.abs(F - oF).max() <= 1e-11 * max(1.0, np.abs(oF).max())
        assert np.abs(S - oS).max() <= 1e-10 * max(1.0, np.abs(oS).max())
    m.close()


@pytest.mark.parametrize("k", [1, 7])
def test_alone_and_in_a_batch_bit_for_bit(k, tmp_path, gapgb_mod):
    """A cell alone is split over blocks, one of 1600 atoms of cells is not."""
    _, m = _model(tmp_path, gapgb_mod, _sf(*SETS[k]))
    cells = [three_species_cell(s) for s in range(50)]
    off = np.cumsum([0] + [len(z) for _, _, z in cells]).astype(np.int32)
    E, F, S = m.eval_batch(off, np.concatenate([z for _, _, z in cells]),
                           np.stack([l for l, _, _ in cells]),
                           np.concatenate([p for _, p, _ in cells]))
    for s in (0, 17, 49):
        lat, pos, z = cells[s]
        e, f, st, _ = m.eval(z, lat, pos)
        # (24 sparse points: one tile of the GPR, so it too adds in one order)
        Xa = m.descriptors([0, len(z)], z, lat[None], pos)
        Xb = m.descriptors(off, np.concatenate([c[2] for c in cells]),
                           np.stack([c[0] for c in cells]), np.concatenate([c[1] for c in cells]))
        assert np.array_equal(Xa, Xb[off[s]:off[s + 1]])
        assert np.array_equal(f, F[off[s]:off[s + 1]])
        assert np.array_equal(st, S[s]) and e == E[s]
    m.close()
