"""The transposed 'fe' RK4 loop against NumPy, at the sizes where its forms meet
and its tiles end."""
import numpy as np
import pytest
import torch

from conftest import rel_err
from qspectra_gb300 import _native
from qspectra_gb300.simulate.third_order import pair_tables

pytestmark = pytest.mark.gpu


def reference(Q, Ae, Me, pairs, y0, nsteps, h):
    S, P, N, _ = Q.shape
    R = np.conj(Me[:, pairs[:, 0]] + Me[:, pairs[:, 1]] - Ae[:, None])      # (S, P, c, b)

    def rhs(X):   # X (S, P, N)
        return np.einsum('sqbr,sqb->srb', Q, X) + np.einsum('spc,spcb->spb', X, R)

    X = np.broadcast_to(y0, (S, P * N)).reshape(S, N, P).transpose(0, 2, 1).astype(complex)
    out = [X]
    for _ in range(nsteps):
        k1 = rhs(X)
        k2 = rhs(X + h / 2 * k1)
        k3 = rhs(X + h / 2 * k2)
        k4 = rhs(X + h * k3)
        X = X + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        out.append(X)
    return np.stack(out, 1).transpose(0, 1, 3, 2).reshape(S, nsteps + 1, N * P)


# 1 to 28 pairs fit a CTA in FP64, 45 in FP32 (450 of 512 elements); 55 pairs
# past that, odd (8-byte loads); 66 and 78 even with a ragged second tile
@pytest.mark.parametrize('N', [2, 3, 4, 6, 8, 10, 11, 12, 13])
@pytest.mark.parametrize('S', [1, 3])
@pytest.mark.parametrize('prec', ['fp64', 'fp32'])
@pytest.mark.parametrize('per_sample', [False, True])
def test_loop_matches_numpy(N, S, prec, per_sample):
    pairs, _ = pair_tables(N)
    P = len(pairs)
    rng = np.random.RandomState(N)

    def rand(*shape):
        return (rng.randn(*shape) + 1j * rng.randn(*shape)) * 0.1 / np.sqrt(P)

    Q, Ae, Me = rand(S, P, N, P), rand(S, N, N), rand(S, N, N, N)
    y0 = rng.randn(*((S,) if per_sample else ()), P * N) + 0j
    cdt = torch.complex64 if prec == 'fp32' else torch.complex128
    precision = _native.QSX_FP32 if prec == 'fp32' else _native.QSX_FP64
    out = _native.fe_heisenberg_rk4(
        torch.as_tensor(Q).to(cdt).cuda(), torch.as_tensor(Ae).to(cdt).cuda(),
        torch.as_tensor(Me).to(cdt).cuda(), torch.as_tensor(pairs).cuda(),
        torch.as_tensor(y0).cuda(), 7, 0.8, precision).cpu().numpy()
    ref = reference(Q, Ae, Me, pairs, y0, 7, 0.8)
    assert rel_err(out, ref) < (1e-5 if prec == 'fp32' else 1e-13)


def test_a_non_finite_state_is_reported():
    pairs, _ = pair_tables(4)
    z = lambda *s: torch.zeros(s, dtype=torch.complex128, device='cuda')  # noqa: E731
    Q = z(1, 6, 4, 6)
    Q[0, 2, 1, 3] = float('inf')
    with pytest.raises(_native.IntegratorError):
        _native.fe_heisenberg_rk4(Q, z(1, 4, 4), z(1, 4, 4, 4), torch.as_tensor(pairs).cuda(),
                                  torch.ones(24, dtype=torch.complex128, device='cuda'), 3, 1.0)


# past one CTA a sample: teams of CTAs with Q on chip (rows in shared memory and
# in registers, odd and even pair counts, elements of two columns in a CTA, more
# samples than teams), and the loop over the L2 where no team holds a sample.
# 32-bit sums of up to 300 terms of that size stay below 1e-5
@pytest.mark.parametrize('N,S,prec', [(14, 1, 'fp32'), (14, 70, 'fp32'), (16, 20, 'fp32'),
                                      (17, 5, 'fp32'), (20, 9, 'fp32'), (22, 8, 'fp32'),
                                      (24, 4, 'fp32'), (26, 1, 'fp32'), (14, 6, 'fp64'),
                                      (17, 2, 'fp64'), (20, 1, 'fp64'), (22, 1, 'fp64'),
                                      (24, 1, 'fp64')])
def test_large_loops_match_numpy(N, S, prec):
    test_loop_matches_numpy(N, S, prec, True)
