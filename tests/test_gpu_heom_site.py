"""The on-chip FP32 hierarchy loop against the per-stage kernels and FP64."""
import numpy as np
import pytest
import torch

import qspectra_gb300 as qg
from conftest import rel_err
from qspectra_gb300 import _native
from qspectra_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def tables(n, level, K=0, block='ee', sub='e', heisenberg=False, **kw):
    ham = qg.ElectronicHamiltonian(wl.ring_hamiltonian(n, seed=n),
                                   bath=qg.DebyeBath(qg.CM_K * 300, 35, 106))
    m = qg.HEOMModel(ham, hilbert_subspace=sub, unit_convert=qg.CM_FS, K=K, level_cutoff=level, **kw)
    return m, m.tables(block, heisenberg)


# every padded block size, hierarchies in one CTA to eight, more samples than
# clusters fit at once, several nodes kept, steps between saves
@pytest.mark.parametrize('n,level,S,every,keep', [
    (3, 2, 1, 1, 1), (3, 5, 7, 2, 35), (4, 5, 3, 1, 5), (5, 4, 200, 4, 1), (6, 5, 2, 1, 2),
    (7, 4, 33, 1, 120), (8, 2, 5, 3, 9), (8, 5, 70, 6, 1), (8, 5, 1, 1, 495), (8, 6, 2, 4, 3)])
@pytest.mark.parametrize('kw', [{}, dict(low_temp_corr=False), dict(modified_HEOM=True),
                                dict(heisenberg=True)])
def test_matches_the_per_stage_kernels(n, level, S, every, keep, kw):
    m, tb = tables(n, level, **kw)
    rng = np.random.RandomState(n + S)
    base = m.hamiltonian.H('e')
    H = torch.as_tensor(np.array([base + np.diag(rng.randn(n) * 50) for _ in range(S)])).cuda()
    y0 = torch.as_tensor(rng.randn(S, tb.nnodes * n * n) + 1j * rng.randn(S, tb.nnodes * n * n)).cuda()
    run = lambda prec, v: _native.heom_rk4(tb, H, H, y0, 12, 0.5, qg.CM_FS, batch=S,  # noqa: E731
                                           save_every=every, save_nodes=keep, precision=prec,
                                           mean=True, variant=v)
    a, b, c = run(_native.QSX_FP32, 0), run(_native.QSX_FP32, 1), run(_native.QSX_FP64, 1)
    for key in ('state', 'mean'):
        x, y, z = (r[key].cpu().numpy() for r in (a, b, c))
        assert rel_err(y, z) < 1e-5
        assert rel_err(x, z) < 1e-5


# two bath modes (two "up" terms a site), states on two sites (whole term
# lists), a shared initial state and Hamiltonian
@pytest.mark.parametrize('n,level,K,block,sub', [(3, 2, 1, 'ee', 'e'), (8, 2, 1, 'ee', 'ge'),
                                                 (3, 4, 0, 'ff', 'gef')])
def test_other_term_lists(n, level, K, block, sub):
    m, tb = tables(n, level, K, block, sub)
    Hx, Hy = m.block_hamiltonians(block)
    rng = np.random.RandomState(n)
    E = tb.nx * tb.ny
    y0 = torch.as_tensor(rng.randn(tb.nnodes * E) + 1j * rng.randn(tb.nnodes * E)).cuda()
    run = lambda prec, v: _native.heom_rk4(tb, Hx, Hy, y0, 10, 0.5, qg.CM_FS, batch=3,  # noqa: E731
                                           save_nodes=tb.nnodes, precision=prec,
                                           variant=v)['state'].cpu().numpy()
    ref = run(_native.QSX_FP64, 1)
    assert rel_err(run(_native.QSX_FP32, 0), ref) < 1e-5


def test_a_non_finite_sample_is_reported():
    m, tb = tables(8, 3)
    H = torch.as_tensor(m.hamiltonian.H('e')).cuda().repeat(4, 1, 1)
    H[2, 3, 3] = float('nan')
    y0 = torch.ones(tb.nnodes * 64, dtype=torch.complex128, device='cuda')
    with pytest.raises(_native.IntegratorError):
        _native.heom_rk4(tb, H, H, y0, 4, 0.5, qg.CM_FS, batch=4, precision=_native.QSX_FP32)
