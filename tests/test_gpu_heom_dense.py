"""Small hierarchies through their dense propagator against the stepped loop,
and large propagators in the doubling loop."""
import numpy as np
import pytest
import torch

import oracle as orc
import qspectra_gb300 as qg
from conftest import rel_err
from qspectra_gb300 import _native
from qspectra_gb300 import workloads as wl
from qspectra_gb300.simulate import utils
from test_gpu_rk4 import random_generators

pytestmark = pytest.mark.gpu


# below, at and above the number of steps and the size that take it
@pytest.mark.parametrize('n,K,level,sub,block,points', [
    (2, 0, 2, 'e', 'ee', 65), (2, 1, 4, 'e', 'ee', 64), (3, 1, 3, 'e', 'ee', 200),
    (3, 1, 3, 'ge', 'eg', 90), (2, 1, 3, 'gef', 'fe', 70), (4, 0, 3, 'e', 'ee', 130),
    (4, 0, 4, 'e', 'ee', 80)])
@pytest.mark.parametrize('kw', [{}, dict(low_temp_corr=False), dict(aki_temp_corr=True),
                                dict(modified_HEOM=True)])
@pytest.mark.parametrize('prec', ['fp64', 'fp32'])
@pytest.mark.parametrize('heisenberg', [False, True])
def test_dense_form_matches_the_stepped_loop(n, K, level, sub, block, points, kw, prec, heisenberg,
                                             monkeypatch):
    ham = qg.ElectronicHamiltonian(wl.fmo7_hamiltonian(n, seed=n),
                                   bath=qg.DebyeBath(qg.CM_K * 300, 35, 106))
    m = qg.HEOMModel(ham, hilbert_subspace=sub, unit_convert=qg.CM_FS, K=K, level_cutoff=level, **kw)
    f = m.equation_of_motion(block, heisenberg)
    rng = np.random.RandomState(n)
    y0 = rng.randn(f.dim) + 1j * rng.randn(f.dim)
    t = np.arange(points) * 2.0
    out, calls = [], []
    real = utils._heom_propagator
    monkeypatch.setattr(utils, '_heom_propagator', lambda *a: calls.append(1) or real(*a))
    for most in (utils.HEOM_DENSE_MAX, 0):
        monkeypatch.setattr(utils, 'HEOM_DENSE_MAX', most)
        out.append([qg.integrate(f, y0, t, precision=prec, step=1.0, heom_nodes=nodes)
                    for nodes in (None, 1)])
        assert (len(calls) > 0) == (f.dim <= 400 and 2 * (points - 1) >= 64) or most == 0
    for a, b in zip(*out):
        assert a.shape == b.shape
        assert rel_err(a, b) < (1e-11 if prec == 'fp64' else 1e-5)


@pytest.mark.parametrize('m,nsteps,every', [(65, 200, 1), (128, 37, 1), (129, 300, 3),
                                            (252, 500, 1), (512, 80, 1)])
def test_large_propagators_by_doubling(m, nsteps, every):
    """Few squares, then blocks: against the oracle through an exact D."""
    L = random_generators(1, m, seed=m)
    nsteps = nsteps // every * every
    A = L[0]
    D = A + A @ A / 2 + A @ A @ (A / 6 + A @ A / 24)
    rng = np.random.RandomState(m)
    y0 = rng.randn(m) + 1j * rng.randn(m)
    ref = orc.rk4_integrate(A, y0, np.arange(0, nsteps + 1, every) * 1.0, h=1.0)
    out = _native.rk4(torch.as_tensor(D)[None].cuda(), torch.as_tensor(y0).cuda(), nsteps, every,
                      state=True)['state'][0].cpu().numpy()
    assert rel_err(out, ref) < 1e-11


def test_a_growing_hierarchy_is_reported():
    ham = qg.ElectronicHamiltonian(wl.fmo7_hamiltonian(2), bath=qg.DebyeBath(qg.CM_K * 300, 35, 106))
    m = qg.HEOMModel(ham, hilbert_subspace='e', unit_convert=qg.CM_FS, K=0, level_cutoff=2)
    f = m.equation_of_motion('ee')
    with pytest.raises(_native.IntegratorError):
        qg.integrate(f, np.ones(f.dim, complex), np.arange(0, 200) * 500.0)
