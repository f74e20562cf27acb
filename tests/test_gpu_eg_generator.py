"""The fit's generator and RK4 step kernels, forward and backward, against the
torch forms that autograd differentiates."""
import numpy as np
import pytest
import torch

import oracle as orc
from conftest import rel_err
from qspectra_gb300 import _native
from qspectra_gb300.simulate import adjoint as adj

pytestmark = pytest.mark.gpu


# direct terms alone, just past them, the usual count; a and y on both sides of
# the series' range (4 K puts y at 70), x = 0
@pytest.mark.parametrize('K', [1, 2, 24, 25, 26, 1000])
@pytest.mark.parametrize('T,gam', [(53.5, 106.0), (208.5, 40.0), (2.8, 106.0), (2.0, 500.0)])
def test_debye_unit_matches_the_direct_sum(K, T, gam):
    bath = orc.DebyeBathSpec(T, 1.0, gam)
    x = np.array([-1900.0, -700.3, -2 * np.pi * T * 6, -40.0, -1e-3, 0.0, 1e-9, 33.0, 80.5,
                  2 * np.pi * T * 6.01, 900.0])
    val, der = _native.debye_unit(torch.as_tensor(x).cuda(), T, gam, K)
    ref = np.array([bath.corr_complex(v, K) for v in x])
    hval, hder = adj._debye_unit(torch.as_tensor(x), T, gam, K)
    # as exact as the direct sum itself
    assert rel_err(val.cpu().numpy(), ref) < 1e-14
    assert rel_err(val.cpu().numpy(), hval.numpy()) < 1e-14
    assert rel_err(der.cpu().numpy(), hder.numpy()) < 1e-14


@pytest.mark.parametrize('N,S', [(1, 1), (2, 5), (7, 33), (8, 4), (15, 3), (16, 2), (17, 2)])
def test_generator_and_gradient_match_torch(N, S):
    rng = np.random.RandomState(N)
    H0 = rng.randn(S, N, N) * 60
    H0 = H0 + H0.transpose(0, 2, 1) + 12300 * np.eye(N)
    w = torch.as_tensor(rng.randn(S, N, N) + 1j * rng.randn(S, N, N)).cuda()
    args = (53.5, 106.0, 12300.0, 2e-4)
    grads, Ls = [], []
    for eigh in (None, torch.linalg.eigh):
        H = torch.as_tensor(H0).cuda().requires_grad_(True)
        lam = torch.tensor(35.0, dtype=torch.float64, device='cuda', requires_grad=True)
        L = adj.eg_heisenberg_generator(H, lam, *args, eigh=eigh)
        (L * w).real.sum().backward()
        Ls.append(L.detach().cpu().numpy())
        grads.append((H.grad.cpu().numpy(), lam.grad.cpu().numpy()))
    assert rel_err(Ls[0], Ls[1]) < 1e-12
    sym = [0.5 * (g[0] + g[0].transpose(0, 2, 1)) for g in grads]
    # eigenvector derivatives over gaps down to a hundredth of the spread
    assert rel_err(sym[0], sym[1]) < 1e-10
    assert rel_err(grads[0][1], grads[1][1]) < 1e-12


@pytest.mark.parametrize('N,S', [(1, 3), (7, 9), (8, 4), (16, 3), (17, 2)])
def test_rk4_step_and_gradient_match_torch(N, S):
    rng = np.random.RandomState(N)
    L0 = 0.2 * (rng.randn(S, N, N) + 1j * rng.randn(S, N, N))
    w = torch.as_tensor(rng.randn(S, N, N) + 1j * rng.randn(S, N, N)).cuda()
    out = []
    for f in (lambda L: adj.rk4_step_minus_identity(L, 0.7),
              lambda L: (0.7 * L) + 0.5 * (0.7 * L) @ (0.7 * L) + (0.7 * L) @ (0.7 * L)
              @ ((0.7 * L) / 6 + (0.7 * L) @ (0.7 * L) / 24)):
        L = torch.as_tensor(L0).cuda().transpose(1, 2).requires_grad_(True)
        D = f(L)
        (D * w).real.sum().backward()
        out.append((D.detach().cpu().numpy(), L.grad.cpu().numpy()))
    assert rel_err(out[0][0], out[1][0]) < 1e-13
    assert rel_err(out[0][1], out[1][1]) < 1e-13
