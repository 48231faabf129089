"""Energy and stress of a cell do not depend on the batch it is in, bit for
bit, around the sizes at which a structure's sums are split into parts (512
atoms each)."""
import numpy as np
import pytest

from helpers import synth_model_file, three_species_cell

pytestmark = pytest.mark.gpu


def _fcc(reps, seed):
    rng = np.random.default_rng(seed)
    basis = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
    g = np.stack(np.meshgrid(*[np.arange(r) for r in reps], indexing="ij"), -1).reshape(-1, 1, 3)
    frac = (g + basis[None]).reshape(-1, 3)
    lat = np.diag(3.9 * np.array(reps)) + rng.normal(0.0, 0.05, (3, 3))
    pos = (frac / np.array(reps)) @ lat + rng.normal(0.0, 0.08, (len(frac), 3))
    return lat, pos, np.array([13, 28, 40], np.int32)[np.arange(len(frac)) % 3]


@pytest.mark.parametrize("reps", [(4, 4, 8), (5, 5, 10), (4, 8, 8), (5, 7, 8), (7, 8, 10)])
@pytest.mark.parametrize("precision", ["fp64", "tc"])
def test_alone_and_among_small_cells(reps, precision, tmp_path, gapgb_mod, oracle_mod):
    import gapgb.synth as S
    path = synth_model_file(str(tmp_path / "gap_parameters"), oracle_mod, [three_species_cell(0)],
                            M=30, coeff_std=0.1)
    m = gapgb_mod.GapModel.load(path)
    m.set_precision(precision)
    cells = [_fcc(reps, 3)] + [three_species_cell(s) for s in range(60)] + [_fcc(reps, 4)]
    off, sp, lat, pos = S.pack(cells)
    E, _, St = m.eval_batch(off, sp, lat, pos)
    for s in (0, 30, 61):
        l, p, z = cells[s]
        e, _, st, _ = m.eval(z, l, p)
        assert e == E[s] and np.array_equal(st, St[s])
    m.close()
