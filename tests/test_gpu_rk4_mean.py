"""Ensemble means of one projection in blocks of steps, and their adjoint,
against the stepped loops (themselves checked against the oracle)."""
import numpy as np
import pytest
import torch

from conftest import rel_err
from qspectra_gb300 import _native
from test_gpu_rk4 import random_generators

pytestmark = pytest.mark.gpu


def inputs(S, m, seed, prec=_native.QSX_FP64, per_sample=False):
    rng = np.random.RandomState(seed)
    D = _native.rk4_propagator(torch.as_tensor(random_generators(S, m, seed)).cuda(), 1.0, prec)
    lead = (S,) if per_sample else ()
    def vec(*shape):
        return torch.as_tensor(rng.randn(*shape) + 1j * rng.randn(*shape)).cuda()
    return D, vec(*lead, m), vec(*lead, 1, m), vec


# the first and last supported lengths and the stepped ones beside them, block
# counts on either side of 32 and 64; row counts to 16 and past; samples below,
# at and above the persistent grid
@pytest.mark.parametrize('m,S,nsteps', [
    (7, 3, 62), (7, 3, 63), (7, 5, 64), (1, 2, 95), (8, 305, 1023), (7, 40, 1024),
    (16, 3, 2047), (7, 700, 2047), (15, 2, 2048), (2, 3, 4095), (3, 2, 4096), (17, 3, 100)])
@pytest.mark.parametrize('per_sample', [False, True])
def test_mean_matches_the_stepped_loop(m, S, nsteps, per_sample):
    D, y0, c, _ = inputs(S, m, m + nsteps, per_sample=per_sample)
    kw = dict(proj=c, per_sample=False, mean=True)
    out = _native.rk4(D, y0, nsteps, 1, **kw)['mean'].cpu().numpy()
    ref = _native.rk4(D, y0, nsteps, 1, variant=1, **kw)['mean'].cpu().numpy()
    assert rel_err(out, ref) < 1e-10   # an ulp a step and term, 4096 x 16 of them


@pytest.mark.parametrize('m,S,nsteps', [(9, 3, 63), (12, 400, 500), (16, 2, 800)])
def test_single_precision_mean(m, S, nsteps):
    D, y0, c, _ = inputs(S, m, m, _native.QSX_FP32)
    kw = dict(proj=c, per_sample=False, mean=True)
    out = _native.rk4(D, y0, nsteps, 1, **kw)['mean'].cpu().numpy()
    ref = _native.rk4(D, y0, nsteps, 1, variant=1, **kw)['mean'].cpu().numpy()
    exact = _native.rk4(D.to(torch.complex128), y0, nsteps, 1, variant=1, **kw)['mean']
    assert rel_err(ref, exact.cpu().numpy()) < 1e-4
    assert rel_err(out, exact.cpu().numpy()) < 1e-10


@pytest.mark.parametrize('m,S,nsteps,ck', [
    (7, 3, 1, 1), (7, 3, 62, 64), (7, 3, 63, 64), (7, 5, 64, 5), (1, 2, 95, 16), (8, 305, 1023, 64),
    (16, 3, 2047, 64), (7, 200, 2047, 100), (15, 2, 2048, 64), (2, 3, 4095, 64),
    (3, 2, 4096, 64), (17, 3, 100, 10)])
@pytest.mark.parametrize('per_sample', [False, True])
def test_adjoint_matches_the_stepped_adjoint(m, S, nsteps, ck, per_sample):
    D, y0, c, vec = inputs(S, m, m + nsteps, per_sample=per_sample)
    c = c.reshape(-1, m)[0]
    g = vec(nsteps + 1)
    nck = max(1, -(-nsteps // ck))
    states = _native.rk4(D, y0, (nck - 1) * ck, ck, state=True, variant=1)['state']
    ref = _native.rk4_adjoint(D, states, ck, nsteps, c, g, 0.25).cpu().numpy()
    out = _native.rk4_mean_adjoint(D, y0, ck, nsteps, c, g, 0.25).cpu().numpy()
    # both sum nsteps outer products in another order: as above, per product
    assert rel_err(out, ref) < 1e-9


def test_an_unexcited_unstable_mode_runs_the_stepped_loops():
    m, S, nsteps = 5, 3, 600
    L = random_generators(S, m, seed=5)
    L[:, -1, :] = L[:, :, -1] = 0
    L[:, -1, -1] = 30.0
    D = _native.rk4_propagator(torch.as_tensor(L).cuda(), 1.0)
    y0 = torch.ones(m, dtype=torch.complex128, device='cuda')
    y0[-1] = 0
    kw = dict(proj=y0[None], per_sample=False, mean=True)
    out = _native.rk4(D, y0, nsteps, 1, **kw)['mean']
    assert torch.isfinite(out.abs()).all()
    assert torch.equal(out, _native.rk4(D, y0, nsteps, 1, variant=1, **kw)['mean'])
    g = torch.ones(nsteps + 1, dtype=torch.complex128, device='cuda')
    states = _native.rk4(D, y0, nsteps - 100, 100, state=True, variant=1)['state']
    assert torch.equal(_native.rk4_mean_adjoint(D, y0, 100, nsteps, y0, g, 0.5),
                       _native.rk4_adjoint(D, states, 100, nsteps, y0, g, 0.5))
    L[0, 0, 0] = np.nan
    D = _native.rk4_propagator(torch.as_tensor(L).cuda(), 1.0)
    with pytest.raises(_native.IntegratorError):
        _native.rk4(D, y0, nsteps, 1, **kw)
