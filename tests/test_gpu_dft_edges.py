"""Direct transforms against their definition where the blocks of 32 samples,
the slices and the chunks of frequencies end."""
import numpy as np
import pytest
import torch

from qspectra_gb300 import _native

pytestmark = pytest.mark.gpu


# a phase's argument is rounded to half a unit of at most 2000 rad, and a block
# adds 32 roundings: below 1e-12 of the sum of the samples' sizes
@pytest.mark.parametrize('nt', [1, 15, 16, 17, 31, 32, 33, 512, 513, 1000])
@pytest.mark.parametrize('nf,batch', [(1, 1), (8, 3), (9, 2)])
def test_one_axis(nt, nf, batch):
    rng = np.random.RandomState(nt + nf)
    x = rng.randn(batch, nt) + 1j * rng.randn(batch, nt)
    f = rng.randn(nf) * 2
    X = _native.dft(torch.as_tensor(x).cuda(), 0.3, 0.7, torch.as_tensor(f), 0.5, 1.1, -1)
    t = 0.3 + 0.7 * np.arange(nt)
    ref = 0.7 * x @ np.exp(-1j * np.outer(t, (f - 0.5) * 1.1))
    assert np.abs(X.cpu().numpy() - ref).max() <= 1e-12 * 0.7 * np.abs(x).sum(1).max()


# F3 = 2, 4 and 8 frequencies a CTA, samples across blocks
@pytest.mark.parametrize('n1,n3,nf1,nf3,batch', [(1, 1, 1, 1, 1), (33, 31, 5, 3, 2),
                                                 (20, 64, 40, 300, 2), (40, 33, 21, 700, 1),
                                                 (7, 65, 300, 9, 170)])
def test_two_axes(n1, n3, nf1, nf3, batch):
    rng = np.random.RandomState(n1 + nf3)
    x = rng.randn(n3, batch, n1) + 1j * rng.randn(n3, batch, n1)
    f1, f3 = rng.randn(nf1), rng.randn(nf3)
    xt = torch.as_tensor(x).cuda().permute(2, 1, 0).contiguous()
    X = _native.dft2(xt, 0.2, 0.5, f1, -1, -0.1, 0.4, f3, 1, 0.1, 1.3).cpu().numpy()
    e1 = np.exp(-1j * np.outer(f1 - 0.1, 1.3 * (0.2 + 0.5 * np.arange(n1))))
    e3 = np.exp(1j * np.outer(f3 - 0.1, 1.3 * (-0.1 + 0.4 * np.arange(n3))))
    ref = np.einsum('kn,mbn,lm->kbl', e1, x, e3, optimize=True) * 0.2
    assert np.abs(X - ref).max() <= 1e-12 * 0.2 * np.abs(x).sum((0, 2)).max()
