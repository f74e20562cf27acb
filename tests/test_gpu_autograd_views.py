"""The fit's differentiable pieces where autograd hands over conjugate views, asks
for second derivatives, or a transform watches the operations."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

from conftest import rel_err
from qspectra_gb300.simulate import adjoint as adj

pytestmark = pytest.mark.gpu

ARGS = (53.5, 106.0, 12300.0, 2e-4)


def draw(*shape, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(shape, dtype=torch.complex128, generator=g).cuda()


def hamiltonians(N, S):
    H = 60 * draw(S, N, N, seed=N).real
    return H + H.transpose(1, 2) + 12300 * torch.eye(N, dtype=torch.float64, device='cuda')


def err(a, b):
    return rel_err(a.detach().cpu().numpy(), b.detach().cpu().numpy())


LOSSES = {
    'plain': lambda D, w: (D * w).real.sum(),
    'conjugate': lambda D, w: (D.conj() * w).real.sum(),
    'adjoint': lambda D, w: (D.mH @ w).real.sum(),
    'einsum': lambda D, w: torch.einsum('sij,sij->', D.conj(), w).real,
}


@pytest.mark.parametrize('loss', LOSSES)
@pytest.mark.parametrize('view', [False, True])
def test_step_gradient_of_conjugate_views(loss, view):
    L0, w, out = 0.2 * draw(5, 7, 7), draw(5, 7, 7, seed=1), []
    for f in (adj.rk4_step_minus_identity, adj._rk4_step_arrays):
        L = L0.clone().requires_grad_(True)
        D = f(L.conj() if view else L, 0.7)
        LOSSES[loss](D, w).backward()
        out.append((D, L.grad))
    assert err(out[0][0], out[1][0]) < 1e-14
    assert err(out[0][1], out[1][1]) < 1e-13


@pytest.mark.parametrize('loss', LOSSES)
def test_generator_gradient_of_conjugate_views(loss):
    w, out = draw(5, 7, 7, seed=1), []
    for eigh in (None, torch.linalg.eigh):
        H = hamiltonians(7, 5).requires_grad_(True)
        lam = torch.tensor(35.0, dtype=torch.float64, device='cuda', requires_grad=True)
        LOSSES[loss](adj.eg_heisenberg_generator(H, lam, *ARGS, eigh=eigh), w).backward()
        out.append((0.5 * (H.grad + H.grad.transpose(1, 2)), lam.grad))
    # eigenvector derivatives over gaps down to a hundredth of the spread
    assert err(out[0][0], out[1][0]) < 1e-10
    assert err(out[0][1], out[1][1]) < 1e-12


def test_second_derivative_of_the_step():
    w, v, out = draw(3, 7, 7, seed=1), draw(3, 7, 7, seed=2), []
    for f in (adj.rk4_step_minus_identity, adj._rk4_step_arrays):
        L = (0.2 * draw(3, 7, 7)).requires_grad_(True)
        (g,) = torch.autograd.grad((f(L, 0.7) * w).real.sum(), L, create_graph=True)
        out.append(torch.autograd.grad((g * v).real.sum(), L)[0])
    assert err(*out) < 1e-13


def test_second_derivative_of_the_generator():
    """Along one direction against central differences of the first derivative."""
    w = draw(2, 4, 4, seed=1)
    H0, dH = hamiltonians(4, 2), 60 * draw(2, 4, 4, seed=3).real
    dH = dH + dH.transpose(1, 2)
    lam0 = torch.tensor(35.0, dtype=torch.float64, device='cuda')

    def first(H, lam, **kw):
        L = adj.eg_heisenberg_generator(H, lam, *ARGS)
        return torch.autograd.grad((L * w).abs().square().sum(), (H, lam), **kw)

    H, lam = H0.clone().requires_grad_(True), lam0.clone().requires_grad_(True)
    gH, glam = first(H, lam, create_graph=True)
    dot = (gH * dH).sum() + 0.3 * glam
    second = torch.autograd.grad(dot, (H, lam))
    h = 1e-4
    ends = []
    for s in (h, -h):
        ends.append(first((H0 + s * dH).requires_grad_(True),
                          (lam0 + 0.3 * s).requires_grad_(True)))
    # 1e-4 of a direction of 1e2 moves the eigenvalues by 1e-4 of their spread:
    # its square, and 1e-15 / 1e-4 of rounding
    sym = lambda x: 0.5 * (x + x.transpose(1, 2))  # noqa: E731
    assert err(sym(second[0]), sym((ends[0][0] - ends[1][0]) / (2 * h))) < 1e-6
    assert err(second[1], (ends[0][1] - ends[1][1]) / (2 * h)) < 1e-6


def test_transforms_of_the_step():
    L, t = 0.2 * draw(3, 7, 7), draw(3, 7, 7, seed=2)
    f = lambda x: adj.rk4_step_minus_identity(x, 0.7)  # noqa: E731
    many = torch.stack([L, 2 * L])
    assert err(torch.func.vmap(f)(many), adj._rk4_step_arrays(many, 0.7)) < 1e-14
    want = torch.func.jvp(lambda x: adj._rk4_step_arrays(x, 0.7), (L,), (t,))[1]
    assert err(torch.func.jvp(f, (L,), (t,))[1], want) < 1e-14
    with fwd.dual_level():
        assert err(fwd.unpack_dual(f(fwd.make_dual(L, t))).tangent, want) < 1e-14


@pytest.mark.parametrize('shape', [(0, 7, 7), (3, 0, 0), (3, 1, 1)])
def test_empty_batches_and_blocks_of_the_step(shape):
    L = draw(*shape).requires_grad_(True)
    D = adj.rk4_step_minus_identity(L, 0.7)
    assert D.shape == shape
    assert torch.autograd.grad(D.real.sum(), L)[0].shape == shape
