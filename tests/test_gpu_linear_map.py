"""A linear map's host and GPU sides: the same values, types and matrix."""
import numpy as np
import pytest
import torch

from qspectra_gb300.dynamics.liouville_space import LinearMap

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('scalar', [False, True])
def test_vector_and_rows_agree(scalar):
    rng = np.random.RandomState(0)
    m = rng.randn(1 if scalar else 5, 9) + 1j * rng.randn(1 if scalar else 5, 9)
    x = rng.randn(9) + 0j
    f = LinearMap(m, scalar=scalar)
    for a, b in ((f(x), f(x[None])[0]), (f(list(x)), f(torch.as_tensor(x)).cpu().numpy())):
        assert isinstance(a, np.ndarray) and a.shape == b.shape
        np.testing.assert_allclose(a, b, rtol=1e-14)
    assert f.shape == m.shape


def test_the_matrix_may_be_changed():
    rng = np.random.RandomState(1)
    m, x = rng.randn(5, 9) + 0j, rng.randn(9) + 0j
    f = LinearMap(m)
    np.testing.assert_allclose(f(x), m @ x, rtol=1e-14)
    f.matrix *= 2
    np.testing.assert_allclose(f(x), 2 * m @ x, rtol=1e-14)
    g = LinearMap(m)
    g.matrix[0] = 0
    assert g(x)[0] == 0
    g.matrix = torch.as_tensor(m[:2]).cuda()
    assert g.shape == (2, 9)
    np.testing.assert_allclose(g(x), m[:2] @ x, rtol=1e-14)
