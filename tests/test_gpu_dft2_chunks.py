"""The two-dimensional transform at the sizes where its frequency chunk changes."""
import numpy as np
import pytest
import torch

from conftest import rel_err
from qspectra_gb300 import _native

pytestmark = pytest.mark.gpu


# on 152 SMs chunks of 2, 4, 8; 2, 4 (a tie with 2), 2, 8 (a tie with both); and a
# last chunk that is not full
@pytest.mark.parametrize('n1,waits,n3', [(30, 1, 30), (64, 3, 64), (60, 3, 200), (64, 5, 64),
                                         (100, 3, 100), (100, 4, 100), (50, 6, 100), (7, 2, 33)])
def test_matches_numpy(n1, waits, n3):
    rng = np.random.RandomState(n1 + waits)
    x = rng.randn(n1, waits, n3) + 1j * rng.randn(n1, waits, n3)
    f1, f3 = np.linspace(-300, 300, 2 * n1 - 1), np.linspace(-250, 300, 2 * n3 - 1)
    uc, dt = 2 * np.pi * 2.99792458e-5, 2.0
    X = _native.dft2(torch.as_tensor(x).cuda(), 0.0, dt, torch.as_tensor(f1).cuda(), -1, 1.0, dt,
                     torch.as_tensor(f3).cuda(), 1, 10.0, uc).cpu().numpy()
    a = np.exp(-1j * np.outer(f1 - 10.0, np.arange(n1) * dt) * uc)
    b = np.exp(1j * np.outer(f3 - 10.0, 1.0 + np.arange(n3) * dt) * uc)
    # sums of 200 terms and 200 rows of them
    assert rel_err(X, dt * dt * np.einsum('kn,nbm,lm->kbl', a, x, b)) < 1e-13
