"""Disorder draws on the GPU against the streams they stand for."""
import numpy as np
import pytest

import qspectra_gb300 as qg
from qspectra_gb300 import _native
from qspectra_gb300.simulate.ensemble import disorder_offsets

pytestmark = pytest.mark.gpu


# one sample, a ragged warp, several CTAs; odd and even counts; enough normals
# to draw past the words that need no twisted neighbour (227) and past the
# first 624; seeds of zero to several words, the largest index
@pytest.mark.parametrize('size,n,start', [(1, 1, 0), (33, 2, 5), (97, 7, 0), (5, 31, 1000),
                                          (3, 240, 0), (2, 1001, (1 << 32) - 2)])
@pytest.mark.parametrize('seed', [[], [0], [1234], [7, 0, 4294967295]])
def test_draws_match_the_host_streams(size, n, start, seed):
    out = _native.disorder_draws(seed, start, size, n, 33.5).cpu().numpy()
    ref = np.array([33.5 * np.random.RandomState(seed + [k]).randn(n)
                    for k in range(start, start + size)])
    # a logarithm's last bit, halved by the root, and the products after it
    assert np.abs(out - ref).max() <= 4 * np.finfo(float).eps * np.abs(ref).max()


@pytest.mark.parametrize('disorder,seed', [(50.0, 3), (50.0, [1, 2]), (0.0, 3), (None, 0),
                                           (lambda rs: np.diag(rs.rand(3)), 4),
                                           (50.0, list(range(20))), (50, 3)])
def test_offsets_match_the_host_for_every_kind_of_disorder(disorder, seed):
    ham = qg.ElectronicHamiltonian(np.diag([1.0, 2.0, 3.0]), disorder=disorder,
                                   random_seed=seed).in_rotating_frame(2.0)
    out = disorder_offsets(ham, 5, 2)
    out = out if isinstance(out, np.ndarray) else out.cpu().numpy()
    ref = ham.disorder_offsets(5, 2)
    assert np.abs(out - ref).max() <= 4 * np.finfo(float).eps * max(np.abs(ref).max(), 1e-300)


@pytest.mark.parametrize('seed', [-1, 1 << 32, 1.5])
def test_bad_seeds_are_refused_as_before(seed):
    ham = qg.ElectronicHamiltonian(np.eye(2), disorder=1.0, random_seed=seed)
    with pytest.raises((ValueError, TypeError)):
        disorder_offsets(ham, 2)
