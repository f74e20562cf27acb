"""Real blocked matrices on the tensor cores at the edges of their tiles."""
import numpy as np
import pytest
import torch

from conftest import rel_err
from qspectra_gb300 import _native

pytestmark = pytest.mark.gpu


# every padded size, odd sizes (one bulk copy a sample) and even ones, powers of
# two and one more, rows in the first and the second 32 rows of the operand,
# fewer and more samples than CTAs.  A product's error is below 2^-21 of the
# sum of its terms' sizes, and ten products of about that size add up below 4e-6
@pytest.mark.parametrize('m,K,nsel,batch', [
    (1, 2, 1, 3), (4, 17, 4, 5), (9, 33, 2, 700), (16, 4, 16, 7), (17, 16, 4, 2),
    (25, 9, 8, 305), (31, 3, 31, 3), (32, 5, 16, 9), (33, 17, 4, 4), (36, 9, 6, 1),
    (49, 17, 7, 311), (49, 64, 1, 3), (50, 8, 16, 2), (57, 2, 50, 5), (63, 33, 4, 2),
    (64, 16, 8, 6)])
def test_powers_and_rows(m, K, nsel, batch):
    assert _native.load().qsx_rk4_block_matrix_real_tc_supported(m, K, nsel)
    rng = np.random.RandomState(m + K)
    D = (0.02 / np.sqrt(m) * rng.randn(batch, m, m) - 0.01 * np.eye(m)).astype(np.float32)
    sel = list(rng.permutation(m)[:nsel])
    out = _native.rk4_block_matrix_real_tc(torch.as_tensor(D).cuda(), K, sel)[0].cpu().numpy()
    P = D.astype(np.float64) + np.eye(m)
    Pk = P.copy()
    for k in range(1, K):
        assert rel_err(out[:, m + (k - 1) * nsel:m + k * nsel], (Pk - np.eye(m))[:, sel]) < 4e-6
        Pk = Pk @ P
    assert rel_err(out[:, :m], Pk - np.eye(m)) < 4e-6
