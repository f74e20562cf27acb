"""The large eigensolver on matrices with equal eigenvalues."""
import numpy as np
import pytest
import torch

import qspectra_gb300 as qg
from qspectra_gb300 import _native
from qspectra_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# one CTA, clusters of two to eight, more columns than lanes; batches on either
# side of a full chip; matrices that are diagonal, decoupled, tiny and large
@pytest.mark.parametrize('n,B', [(1, 3), (2, 2), (3, 5), (6, 1), (31, 4), (63, 2), (64, 1),
                                 (129, 2), (170, 40), (276, 3), (276, 33), (301, 160), (465, 2),
                                 (600, 1)])
@pytest.mark.parametrize('kind', ['dense', 'band', 'decoupled', 'tiny', 'huge'])
def test_eigenpairs(n, B, kind):
    rng = np.random.RandomState(n + B)
    A = rng.randn(B, n, n)
    A = A + A.transpose(0, 2, 1)
    if kind == 'band':
        A = np.array([np.diag(100 * rng.randn(n)) + np.eye(n, k=1) + np.eye(n, k=-1)
                      for _ in range(B)])
    elif kind == 'decoupled':
        A[:, : n // 2, n // 2:] = 0
        A[:, n // 2:, : n // 2] = 0
        A[:, n // 2:, n // 2:] = np.eye(n - n // 2)
    elif kind in ('tiny', 'huge'):
        A *= 1e-60 if kind == 'tiny' else 1e60
    E, U = _native.eigh_large(torch.as_tensor(A).cuda())
    E, U = E.cpu().numpy(), U.cpu().numpy()
    ref = np.linalg.eigvalsh(A)
    scale = np.abs(A).sum(-1).max()
    # backward stable: n ulp of the norm; vectors of clusters by one sweep of
    # Gram-Schmidt
    assert np.abs(E - ref).max() < 4 * n * 2.3e-16 * scale
    eye = np.eye(n)
    assert np.abs(U.transpose(0, 2, 1) @ U - eye).max() < 1e-10
    assert np.abs(A @ U - U * E[:, None, :]).max() < 1e-11 * scale


@pytest.mark.parametrize('H', [np.zeros((1, 1)), np.zeros((3, 3)), np.diag([0.0, 0.0, 5.0]),
                               1e-30 * np.ones((2, 2))])
def test_eigensolver_takes_zero_matrices(H):
    E, U = _native.eigh_large(torch.as_tensor(H)[None].cuda())
    E, U = E[0].cpu().numpy(), U[0].cpu().numpy()
    assert np.abs(U.T @ U - np.eye(len(H))).max() < 1e-12
    assert np.abs(U @ np.diag(E) @ U.T - H).max() <= 1e-12 * max(np.abs(H).max(), 1e-300)


def test_dimer_spectra_in_the_mean_rotating_frame():
    """A dimer's two-exciton energy is zero in its mean rotating frame."""
    H = np.array([[12000.0, 50.0], [50.0, 12500.0]])
    ham = qg.ElectronicHamiltonian(H, bath=qg.DebyeBath(qg.CM_K * 77, 35, 106),
                                   dipoles=[[1, 0, 0]] * 2,
                                   energy_spread_extra=wl.energy_spread_for_dt(H, 2.0))
    m = qg.RedfieldModel(ham, unit_convert=qg.CM_FS, secular=False)
    _, R = qg.third_order_response(m, 40 * m.time_step, population_times=[0.0])
    assert np.isfinite(R).all()
