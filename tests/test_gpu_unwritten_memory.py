"""Shared memory that a kernel has not written: calls on good input right after one
that left NaN all over every SM's."""
import numpy as np
import pytest
import torch

import qspectra_gb300 as qg
from conftest import rel_err
from qspectra_gb300 import _native
from test_gpu_fe_heisenberg import test_loop_matches_numpy as compare_fe_loop
from test_gpu_heom_site import tables

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def fill_with_nan():
    """495 nodes of 8 x 8 elements, 64 samples: 190 KB a CTA, 256 CTAs, all NaN."""
    _, tb = tables(8, 5)
    H = torch.full((64, 8, 8), float('nan'), dtype=torch.float64, device='cuda')
    y = torch.ones(tb.nnodes * 64, dtype=torch.complex128, device='cuda')
    return lambda: _native.heom_rk4(tb, H, H, y, 2, 0.5, qg.CM_FS, batch=64,
                                    precision=_native.QSX_FP32, check_finite=False)


# 3, 5 and 7 sites are padded to 4, 6 and 8; the nodes do not divide evenly over
# the CTAs of a cluster, at the cluster sizes of few and of many samples
@pytest.mark.parametrize('n,level', [(3, 4), (5, 5), (5, 6), (5, 7), (7, 4), (7, 5)])
@pytest.mark.parametrize('S', [1, 3, 64])
def test_hierarchy_on_chip(n, level, S, fill_with_nan):
    m, tb = tables(n, level)
    rng = np.random.RandomState(n + S)
    base = m.hamiltonian.H('e')
    H = torch.as_tensor(np.array([base + np.diag(rng.randn(n) * 50) for _ in range(S)])).cuda()
    y0 = torch.as_tensor(rng.randn(S, tb.nnodes * n * n)
                         + 1j * rng.randn(S, tb.nnodes * n * n)).cuda()
    run = lambda prec, v: _native.heom_rk4(tb, H, H, y0, 6, 0.5, qg.CM_FS, batch=S,  # noqa: E731
                                           save_nodes=tb.nnodes, precision=prec,
                                           variant=v)['state'].cpu().numpy()
    fill_with_nan()
    x = run(_native.QSX_FP32, 0)
    assert rel_err(x, run(_native.QSX_FP64, 1)) < 1e-5


# teams of CTAs whose last rows end at unwritten columns of X or at the sums, by
# the plan on 152 SMs: P = 28 to 55 of the 128 terms that the lanes take
@pytest.mark.parametrize('N,S,prec', [(8, 4, 'fp64'), (8, 5, 'fp64'), (8, 10, 'fp64'),
                                      (8, 15, 'fp64'), (9, 3, 'fp64'), (9, 7, 'fp64'),
                                      (10, 8, 'fp64'), (11, 2, 'fp64'), (11, 4, 'fp64'),
                                      (11, 2, 'fp32'), (11, 4, 'fp32')])
def test_two_exciton_team(N, S, prec, fill_with_nan):
    fill_with_nan()
    compare_fe_loop(N, S, prec, True)
