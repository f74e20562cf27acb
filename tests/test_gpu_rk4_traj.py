"""The doubling form of the RK4 loop (few samples, every state saved) against
the oracle's stage-form RK4 and against the stepped loop."""
import numpy as np
import pytest
import torch

import oracle as orc
from conftest import rel_err
from qspectra_gb300 import _native
from test_gpu_rk4 import random_generators

pytestmark = pytest.mark.gpu


def run(L, y0, nsteps, every, prec, shared=False, **kw):
    precision = _native.QSX_FP32 if prec == 'fp32' else _native.QSX_FP64
    D = _native.rk4_propagator(torch.as_tensor(L).cuda(), 1.0, precision)
    return _native.rk4(D[0] if shared else D, torch.as_tensor(y0).cuda(), nsteps, every,
                       state=True, **kw)['state'].cpu().numpy()


# one CTA per sample and spread over the chip; block sizes that end on, before
# and after a power of two; steps between saves with one, two and three bits
@pytest.mark.parametrize('m,B,nsteps,every', [
    (1, 1, 7, 1), (2, 3, 8, 1), (4, 1, 119, 1), (7, 1, 2047, 1), (8, 5, 64, 1),
    (16, 1, 255, 1), (33, 2, 256, 1), (49, 1, 1000, 1), (49, 3, 257, 1), (64, 1, 130, 1),
    (64, 2, 63, 1), (7, 2, 99, 3), (49, 1, 160, 4), (64, 1, 77, 7)])
@pytest.mark.parametrize('prec', ['fp64', 'fp32'])
@pytest.mark.parametrize('shared', [False, True])
def test_states_match_the_oracle(m, B, nsteps, every, prec, shared):
    L = random_generators(B, m, seed=m + nsteps)
    if shared:
        L = np.broadcast_to(L[:1], L.shape).copy()
    rng = np.random.RandomState(m)
    y0 = rng.randn(B, m) + 1j * rng.randn(B, m)
    t = np.arange(0, nsteps + 1, every) * 1.0
    ref = np.array([orc.rk4_integrate(L[b], y0[b], t, h=1.0) for b in range(B)])
    if prec == 'fp32' and np.abs(ref).max() > np.finfo(np.float32).max:
        with pytest.raises(_native.IntegratorError):   # as the FP32 stepped loop does
            run(L, y0, nsteps, every, prec, shared)
        return
    out = run(L, y0, nsteps, every, prec, shared)
    # FP64: an ulp a step and term; FP32: the rounded propagator's contract
    assert rel_err(out, ref) < (1e-4 if prec == 'fp32' else 1e-11)
    stepped = run(L, y0, nsteps, every, prec, shared, variant=1)
    assert rel_err(out, stepped) < (1e-4 if prec == 'fp32' else 1e-11)


@pytest.mark.parametrize('m,nsteps', [(4, 400), (49, 1000)])
def test_an_unexcited_unstable_mode_runs_the_stepped_loop(m, nsteps):
    """Powers of the growing mode overflow; its amplitude is exactly zero, so
    the stepped loop's states stay finite and the result is that loop's."""
    L = random_generators(1, m, seed=5)
    L[0, -1, :] = L[0, :, -1] = 0
    L[0, -1, -1] = 30.0
    y0 = np.ones((1, m), complex)
    y0[0, -1] = 0
    out = run(L, y0, nsteps, 1, 'fp64')
    assert np.isfinite(out).all()
    assert np.array_equal(out, run(L, y0, nsteps, 1, 'fp64', variant=1))


def test_a_blow_up_is_reported():
    L = np.full((1, 5, 5), 30.0 + 0j)
    with pytest.raises(_native.IntegratorError):
        run(L, np.ones((1, 5), complex), 900, 1, 'fp64')
