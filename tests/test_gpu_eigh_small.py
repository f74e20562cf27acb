"""FP64 eigenpairs of small blocks (a warp or a CTA per matrix, a thread in large batches) against LAPACK's."""
import numpy as np
import pytest
import torch

from qspectra_gb300 import _native

pytestmark = pytest.mark.gpu


def matrices(kind, n, batch):
    rng = np.random.RandomState(n + batch)
    A = rng.randn(batch, n, n)
    A = A + A.transpose(0, 2, 1)
    if kind == 'graded':
        d = 10.0 ** -np.arange(n)
        A = A * d[:, None] * d
    elif kind == 'near':         # gaps of 1e-3 down to nothing around a common level
        A = A * 10.0 ** -rng.randint(3, 17, (batch, 1, 1)) + 3 * np.eye(n)
    elif kind == 'decoupled':    # even and odd states do not meet
        A = A * (np.arange(n)[:, None] % 2 == np.arange(n) % 2)
    elif kind == 'ring':         # exactly degenerate pairs
        A = np.repeat((np.roll(np.eye(n), 1, 0) + np.roll(np.eye(n), -1, 0))[None], batch, 0)
    elif kind == 'zero':
        A = A * 0
    return A


# each step of the kernel rounds by a few units: the basis loses at most 2 eps
# a rotation round (three sweeps of seven) and n eps in each product, below 2e-14
@pytest.mark.parametrize('kind', ['random', 'graded', 'near', 'decoupled', 'ring', 'zero'])
@pytest.mark.parametrize('scale', [1.0, 1e-190, 1e200])
@pytest.mark.parametrize('blocks,batch', [([0, 3], 1), ([0, 4], 5), ([0, 5], 3), ([0, 6], 301),
                                          ([0, 7], 64), ([0, 8], 7), ([0, 1, 8, 12, 14], 33),
                                          ([0, 3], 600), ([0, 2, 6], 2000),
                                          ([0, 9], 3), ([0, 1, 16], 5), ([0, 1, 8, 29], 40),
                                          ([0, 32], 2)])
def test_eigenpairs(kind, scale, blocks, batch):
    n = blocks[-1]
    A = np.zeros((batch, n, n))
    for a, b in zip(blocks[:-1], blocks[1:]):
        A[:, a:b, a:b] = matrices(kind, b - a, batch)
    lower = A * scale + np.tril(np.ones((n, n)), -1)     # the upper triangle is what counts
    E, U = (x.cpu().numpy() for x in _native.eigh(torch.as_tensor(lower).cuda(), blocks))
    E = E / scale
    ref = np.zeros((batch, n))
    for a, b in zip(blocks[:-1], blocks[1:]):
        ref[:, a:b] = np.linalg.eigvalsh(A[:, a:b, a:b])
        assert np.all(np.diff(E[:, a:b]) >= 0)
        outside = np.ones(n, bool)
        outside[a:b] = False
        assert np.all(U[:, a:b][:, :, outside] == 0)
    norm = max(np.abs(A).max(), 1e-300) * n
    assert np.abs(E - ref).max() <= 2e-14 * norm
    assert np.abs(U.transpose(0, 2, 1) @ U - np.eye(n)).max() <= 2e-14
    assert np.abs(A @ U - U * E[:, None]).max() <= 4e-14 * norm
    if kind == 'decoupled' and len(blocks) == 2:
        for u in U:                                       # exact zeros stay
            even = np.abs(u[::2]).max(0) > 0
            assert np.all(even != (np.abs(u[1::2]).max(0) > 0))
