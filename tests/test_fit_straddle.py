"""The energy fit's kernel-value sums of a structure that lies in two chunks of
row tiles (152 x 128 = 19456 rows on a GB300: a 32-atom cell and 38 cells of
512 atoms), against normal equations of the library's own energies with unit
coefficients."""
import numpy as np
import pytest

from helpers import three_species_cell

pytestmark = pytest.mark.gpu


def test_structure_across_a_chunk(gapgb_mod):
    import torch
    import gapgb.synth as S
    ty, al, rc, ze = S.sf_table()
    zs = np.array([13, 28, 40], np.int32)
    rows = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    structs = [three_species_cell(0)] + [S.alloy512(seed=s) for s in range(rows // 512 + 1)]
    batch = S.pack(structs)
    off = batch[0]
    assert off[-1] > rows and rows not in off
    M, D = 20, 2 * len(ty)
    probe = gapgb_mod.GapModel.create(zs, zs.astype(float), ty, al, rc, np.ones(D), np.zeros((1, D)),
                                      np.zeros(1), sf_zeta=ze)
    X = probe.descriptors(*batch)
    probe.close()
    mm = X[np.random.default_rng(3).choice(len(X), M, replace=False)]
    theta = X.std(0)
    m = gapgb_mod.GapModel.create(zs, zs.astype(float), ty, al, rc, theta, mm, np.zeros(M), sf_zeta=ze)
    phi = np.zeros((len(structs), M))
    for k in range(M):
        m.set_coeff(np.eye(M)[k])
        phi[:, k] = m.eval_batch(*batch, lgrad=False)[0]
    E = np.random.default_rng(1).normal(-3.0, 0.1, len(structs)) * np.diff(off)
    c = m.fit_energies(*batch, E, sigma_e=2e-2, jitter=1e-6)
    x = (mm[:, None, :] - mm[None, :, :]) / theta
    w = 1.0 / (2e-2 ** 2 * np.diff(off))
    A = np.exp(-0.5 * (x ** 2).sum(-1)) + 1e-6 * np.eye(M) + (phi * w[:, None]).T @ phi
    b = (phi * w[:, None]).T @ E
    # rounding of the rows themselves (1e-13 of the largest) bounds the residual
    res = np.linalg.norm(A @ c - b) / (np.linalg.norm(A) * np.linalg.norm(c) + np.linalg.norm(b))
    assert res <= 1e-11
    m.close()
