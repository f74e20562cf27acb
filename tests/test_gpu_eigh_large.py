"""The large eigensolver on matrices with equal eigenvalues."""
import numpy as np
import pytest
import torch

import qspectra_gb300 as qg
from qspectra_gb300 import _native
from qspectra_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


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
