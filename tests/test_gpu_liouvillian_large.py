"""Dense generator blocks that give a thread eight elements, against the small
ones sample by sample."""
import numpy as np
import pytest
import torch

from qspectra_gb300 import _native

pytestmark = pytest.mark.gpu


# sites that occupy no, one and several states, more than 64 of them (no masks),
# a bad index, both orders: the same sums in the same order
@pytest.mark.parametrize('n,n_sites,batch', [(12, 11, 150), (25, 24, 6), (13, 70, 80)])
@pytest.mark.parametrize('transpose', [False, True])
def test_batches_equal_their_samples(n, n_sites, batch, transpose):
    rng = np.random.RandomState(n)
    occ = (rng.rand(n_sites, n) < 0.2) * rng.randn(n_sites, n)
    c = lambda *s: torch.as_tensor(rng.randn(*s) + 1j * rng.randn(*s)).cuda()  # noqa: E731
    H = torch.as_tensor(rng.randn(batch, n, n)).cuda()
    G, M = c(batch, n, n), c(batch, n_sites, n, n)
    idx = rng.permutation(n * n).astype(np.int32)
    idx[7] = n * n                     # out of range: its row and column are NaN
    run = lambda s: _native.redfield_liouvillian(  # noqa: E731
        H[s].contiguous(), G[s].contiguous(), M[s].contiguous(), torch.as_tensor(idx).cuda(), 0.3,
        occ=torch.as_tensor(occ).cuda(), transpose=transpose)
    whole = run(slice(None))
    assert batch * len(idx) ** 2 >= 8 * 256 * 1024
    for s in (0, batch // 2, batch - 1):
        assert torch.equal(torch.nan_to_num(whole[s], nan=1e300),
                           torch.nan_to_num(run(slice(s, s + 1))[0], nan=1e300))
