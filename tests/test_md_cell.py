"""A caller that strains the cell between MD steps (d_lat and d_pos are its own
buffers): a step that refreshes the list takes the cell as it is now."""
import numpy as np
import pytest

from helpers import synth_model_file

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "tc"])
def test_refreshed_step_after_a_strain(precision, tmp_path, gapgb_mod, oracle_mod):
    import gapgb.synth as S
    from gapgb.md import MD, masses_of, maxwell_boltzmann
    path = synth_model_file(str(tmp_path / "gap_parameters"), oracle_mod,
                            [S.si64(seed=s) for s in range(2)], M=100, coeff_std=0.05, seed=2)
    off, sp, lat, pos = S.pack([S.si64(seed=20 + s, jitter=0.05) for s in range(2)])
    m = masses_of(sp)
    model, fresh = gapgb_mod.GapModel.load(path), gapgb_mod.GapModel.load(path)
    model.set_precision(precision)
    fresh.set_precision(precision)
    md = MD(model, off, sp, lat, pos, maxwell_boltzmann(off, m, 300.0, seed=1), m, dt=1.0,
            skin=0.8, rebuild_every=50)
    md.run(2)
    md.t["lat"].mul_(1.004)
    md.t["pos"].mul_(1.004)
    md.run(1)
    E, F, St, _ = md.outputs()
    E0, F0, S0 = fresh.eval_batch(off, sp, 1.004 * lat, md.positions())
    # FP64: summation order; TC: the extra slots of the skin round differently
    tol = (1e-11, 1e-10, 1e-9) if precision == "fp64" else (1e-6, 1e-3, 1e-2)
    assert np.abs(E - E0).max() <= tol[0] * len(sp)
    assert np.abs(F - F0).max() <= tol[1] * max(1.0, np.abs(F0).max())
    assert np.abs(St - S0).max() <= tol[2] * max(1.0, np.abs(S0).max())
    md.close()
    model.close()
    fresh.close()
