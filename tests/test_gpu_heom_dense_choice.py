"""What the dense form of small hierarchies must leave to the loop, and keep."""
import numpy as np
import pytest
import torch

import qspectra_gb300 as qg
from conftest import rel_err
from qspectra_gb300 import _native
from qspectra_gb300 import workloads as wl
from qspectra_gb300.simulate import utils

pytestmark = pytest.mark.gpu


def equation(n, K, level):
    ham = qg.ElectronicHamiltonian(wl.fmo7_hamiltonian(n, seed=n),
                                   bath=qg.DebyeBath(qg.CM_K * 300, 35, 106))
    m = qg.HEOMModel(ham, hilbert_subspace='e', unit_convert=qg.CM_FS, K=K, level_cutoff=level)
    f = m.equation_of_motion('ee')
    rng = np.random.RandomState(n)
    return f, rng.randn(f.dim) + 1j * rng.randn(f.dim)


@pytest.fixture
def dense_calls(monkeypatch):
    calls, real = [], utils._heom_propagator
    monkeypatch.setattr(utils, '_heom_propagator', lambda *a: calls.append(1) or real(*a))
    return calls


@pytest.mark.parametrize('nodes', [0, -1, 1000])
@pytest.mark.parametrize('points', [20, 200])
def test_node_counts_out_of_range_are_refused(nodes, points):
    f, y0 = equation(2, 0, 2)
    with pytest.raises((_native.QsxError, RuntimeError)):
        qg.integrate(f, y0, np.arange(points) * 1.0, heom_nodes=nodes)


# seven outputs are stepped, eight doubled; 252 elements in FP32 pay from about
# 150 steps on, 392 with a power of 8 steps never below 256
@pytest.mark.parametrize('n,K,level,points,every,prec,dense', [
    (3, 1, 3, 7, 100, 'fp64', False), (3, 1, 3, 8, 100, 'fp64', True),
    (3, 0, 2, 3, 500, 'fp32', False), (2, 0, 2, 65, 1, 'fp64', True),
    (6, 0, 2, 65, 1, 'fp32', False), (6, 0, 2, 301, 1, 'fp32', True),
    (7, 0, 2, 33, 8, 'fp32', False), (7, 0, 2, 65, 1, 'fp64', True)])
def test_choice(n, K, level, points, every, prec, dense, dense_calls):
    f, y0 = equation(n, K, level)
    t = np.arange(points) * 0.5 * every
    out = qg.integrate(f, y0, t, precision=prec, step=0.5, heom_nodes=1)
    assert bool(dense_calls) == dense
    assert _native.rk4_doubles(f.dim, points - 1, every) == (points >= 8)
    ref = qg.integrate(f, torch.as_tensor(np.array([y0, y0])), t, step=0.5, heom_nodes=1)
    assert rel_err(out, ref[0].cpu().numpy()) < (1e-11 if prec == 'fp64' else 1e-5)


@pytest.mark.parametrize('nodes', [1, None])
def test_blocks_of_outputs(nodes, dense_calls, monkeypatch):
    """Equal blocks, each from the last state of the one before."""
    f, y0 = equation(2, 1, 3)
    t = np.arange(131) * 1.0
    whole = qg.integrate(f, y0, t, step=0.5, heom_nodes=nodes)
    monkeypatch.setattr(utils, 'HEOM_DENSE_BLOCK', 32 * f.dim)
    parts = qg.integrate(f, y0, t, step=0.5, heom_nodes=nodes)
    assert len(dense_calls) == 2
    assert parts.shape == whole.shape
    assert rel_err(parts, whole) < 1e-13
