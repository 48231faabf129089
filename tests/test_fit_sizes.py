"""Fits at the edges of the Cholesky blocks (64 columns, 16-column sub-blocks),
of the row slices of the normal matrix and of the Jacobian product's tiles (32
points, 48 rows): the device coefficients against normal equations whose rows
are the library's own FP64 evaluations with unit coefficients."""
import numpy as np
import pytest

from helpers import three_species_cell

pytestmark = pytest.mark.gpu

ZS = np.array([13, 28, 40], np.int32)


@pytest.mark.parametrize("M,cells,forces", [(1, 1, True), (31, 2, True), (63, 1, True),
                                            (64, 2, False), (65, 3, True), (129, 2, True),
                                            (200, 70, False)])
def test_backward_error(M, cells, forces, gapgb_mod):
    import gapgb.synth as S
    ty, al, rc, ze = S.sf_table()
    structs = [three_species_cell(s) for s in range(cells)]
    batch = S.pack(structs)
    off = batch[0]
    D = 2 * len(ty)
    probe = gapgb_mod.GapModel.create(ZS, ZS.astype(float), ty, al, rc, np.ones(D), np.zeros((1, D)),
                                      np.zeros(1), sf_zeta=ze)
    X = probe.descriptors(*batch)
    probe.close()
    theta, mm, _ = S.model_arrays(X, M, theta_scale=1.0, seed=3)
    theta = np.where(X.std(0) > 0, X.std(0), 1.0)
    m = gapgb_mod.GapModel.create(ZS, ZS.astype(float), ty, al, rc, theta, mm, np.zeros(M), sf_zeta=ze)
    N, ns = int(off[-1]), cells
    phi, pf, ps = np.zeros((ns, M)), np.zeros((3 * N, M)), np.zeros((6 * ns, M))
    for k in range(M):
        c = np.zeros(M)
        c[k] = 1.0
        m.set_coeff(c)
        E, F, St = m.eval_batch(*batch)
        phi[:, k], pf[:, k], ps[:, k] = E, F.reshape(-1), St.reshape(-1)
    rng = np.random.default_rng(1)
    E, F, St = rng.normal(-3.0, 0.1, ns), rng.normal(0.0, 0.5, (N, 3)), rng.normal(0.0, 1.0, (ns, 6))
    se, sf, ss, jit = 2e-2, 0.1, 0.2, 1e-6
    x = (mm[:, None, :] - mm[None, :, :]) / theta
    w = 1.0 / (se ** 2 * np.diff(off))
    A = np.exp(-0.5 * (x ** 2).sum(-1)) + jit * np.eye(M) + (phi * w[:, None]).T @ phi
    b = (phi * w[:, None]).T @ E
    if forces:
        c = m.fit(*batch, E, forces=F, stress=St, sigma_e=se, sigma_f=sf, sigma_s=ss, jitter=jit)
        A += pf.T @ pf / sf ** 2 + ps.T @ ps / ss ** 2
        b += pf.T @ F.reshape(-1) / sf ** 2 + ps.T @ St.reshape(-1) / ss ** 2
    else:
        c = m.fit_energies(*batch, E, sigma_e=se, jitter=jit)
    # rounding of the rows themselves (1e-13 of the largest) bounds the residual
    res = np.linalg.norm(A @ c - b) / (np.linalg.norm(A) * np.linalg.norm(c) + np.linalg.norm(b))
    assert res <= 1e-11
    m.close()
