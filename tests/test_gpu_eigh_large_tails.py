"""The large eigensolver where the elements of a column differ by many orders."""
import numpy as np
import pytest
import torch

from qspectra_gb300 import _native

pytestmark = pytest.mark.gpu


# a cluster per matrix (one CTA, two, eight) and one CTA on a copy
@pytest.mark.parametrize('n', [5, 40, 129, 276, 600])
@pytest.mark.parametrize('tail', [5e-9, 1e-8, 3e-7, 1e-12])
@pytest.mark.parametrize('scale', [1.0, 1e-130, 1e150])
def test_small_elements_below_a_large_one(n, tail, scale):
    """Columns (1, tail, .., tail): tail^2 is lost beside 1^2, tail is not beside 1."""
    A = np.diag(np.linspace(-1.0, 1.0, n)) + np.eye(n, k=1) + np.eye(n, k=-1)
    A += tail * (np.ones((n, n)) - np.eye(n))
    A = scale * A
    E, U = _native.eigh_large(torch.as_tensor(A)[None].cuda())
    E, U = E[0].cpu().numpy() / scale, U[0].cpu().numpy()
    A /= scale
    norm = np.abs(A).sum(-1).max()
    # backward stable: n ulp of the norm, and the vectors to the same residual
    # as any other matrix
    assert np.abs(E - np.linalg.eigvalsh(A)).max() < 4 * n * 2.3e-16 * norm
    assert np.abs(A @ U - U * E).max() < 1e-11 * norm
    assert np.abs(U.T @ U - np.eye(n)).max() < 1e-10


@pytest.mark.parametrize('n', [40, 600])
@pytest.mark.parametrize('where', [(0, 0), (3, 1), (30, 2)])
@pytest.mark.parametrize('value', [float('nan'), float('inf')])
def test_a_non_finite_element_is_reported(n, where, value):
    A = np.eye(n) + np.eye(n, k=1) + np.eye(n, k=-1)
    A[where] = A[where[::-1]] = value
    with pytest.raises(_native.QsxError):
        _native.eigh_large(torch.as_tensor(A)[None].cuda())
