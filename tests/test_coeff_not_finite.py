"""A model file with coefficients that are not finite: the FP64 and mixed forms
return what the sum over the sparse points gives, and take finite coefficients
afterwards."""
import numpy as np
import pytest

from helpers import synth_model_file, three_species_cell

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_not_finite_coefficients_show(bad, precision, tmp_path, gapgb_mod, oracle_mod):
    path = synth_model_file(str(tmp_path / "gap_parameters"), oracle_mod, [three_species_cell(0)],
                            M=30, coeff_std=1.0)
    m0 = gapgb_mod.GapModel.load(path)
    c0 = m0.arrays()[2].copy()
    m0.close()
    lines = open(path).read().split("\n")
    at = max(k for k, l in enumerate(lines) if l.strip())
    c = lines[at].split()
    c[7] = str(bad)
    lines[at] = " ".join(c)
    open(path, "w").write("\n".join(lines))
    m = gapgb_mod.GapModel.load(path)
    m.set_precision(precision)
    lat, pos, z = three_species_cell(1)
    E, F, _, _ = m.eval(z, lat, pos, lgrad=False)
    # one term of the sum over the points is not finite and decides it
    assert np.isnan(E) if np.isnan(bad) else E == bad
    m.set_coeff(c0)
    good = str(tmp_path / "good")
    m.save(good)
    oE = oracle_mod.gap_calc(oracle_mod.Model(good), z, lat, pos, 6.0, False)[0]
    E = m.eval(z, lat, pos, lgrad=False)[0]
    assert abs(E - oE) <= (1e-11 if precision == "fp64" else 1e-3) * max(1.0, abs(oE))
    m.close()
