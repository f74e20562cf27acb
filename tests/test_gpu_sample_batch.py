"""The Hamiltonians of disorder samples: what the offsets may be, and streams."""
import numpy as np
import pytest
import torch

import qspectra_gb300 as qg
from qspectra_gb300 import _native
from qspectra_gb300 import workloads as wl
from qspectra_gb300.simulate.ensemble import SampleBatch

pytestmark = pytest.mark.gpu


def model(n=4, **kw):
    ham = qg.ElectronicHamiltonian(wl.fmo7_hamiltonian(n), bath=qg.DebyeBath(qg.CM_K * 77, 35, 106),
                                   dipoles=np.eye(n, 3), **kw)
    return qg.RedfieldModel(ham, hilbert_subspace='gef', unit_convert=qg.CM_FS, secular=False)


def expected(m, off, subspace):
    H = np.repeat(m.hamiltonian.H(subspace)[None], len(off), 0)
    n = off.shape[1]
    pairs = [(i, j) for i in range(n) for j in range(i + 1, n)]
    shift = {'g': np.zeros((len(off), 1)), 'e': off,
             'f': np.array([[o[i] + o[j] for i, j in pairs] for o in off])}
    d = np.concatenate([shift[x] for x in 'gef' if x in subspace], 1)
    i = np.arange(H.shape[1])
    H[:, i, i] += d
    return H


@pytest.mark.parametrize('subspace', ['e', 'ge', 'f', 'ef', 'gef'])
@pytest.mark.parametrize('form', ['plain', 'shared', 'strided', 'negative view', 'gradient'])
def test_every_form_of_offsets(subspace, form):
    m, rng = model(), np.random.RandomState(0)
    off = rng.randn(5, 4) * 50
    t = torch.as_tensor(off).cuda()
    if form == 'shared':
        off = np.repeat(off[:1], 5, 0)
        t = t[:1]
    elif form == 'strided':
        t = t.T.contiguous().T
    elif form == 'negative view':
        off = -off
        t = torch.complex(torch.zeros_like(t), t).conj().imag
        assert t.is_neg()
    elif form == 'gradient':
        t.requires_grad_(True)
    H = SampleBatch(m, 5, offsets=t).H(subspace)
    np.testing.assert_array_equal(H.detach().cpu().numpy(), expected(m, off, subspace))
    if form == 'gradient':
        w = torch.as_tensor(rng.randn(*H.shape)).cuda()
        (H * w).sum().backward()
        want = [[(expected(m, np.eye(4)[[i]], subspace) - expected(m, np.zeros((1, 4)), subspace))[0]
                 for i in range(4)]]
        want = np.einsum('sab,niab->si', w.cpu().numpy(), np.array(want))
        np.testing.assert_allclose(t.grad.cpu().numpy(), want, rtol=1e-13, atol=1e-13)


def test_objects_made_on_a_busy_stream_serve_another():
    m = model(disorder=100.0, random_seed=3)
    off = m.hamiltonian.disorder_offsets(64)
    dense = np.random.RandomState(1).randn(40, 30) + 0j
    x = torch.ones(3, 30, dtype=torch.complex128, device='cuda')
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for busy in (False, True):      # once to have the memory, which waits for the GPU
        with torch.cuda.stream(a):
            if busy:
                torch.cuda._sleep(400_000_000)      # about 0.2 s
            batch, table = SampleBatch(m, 64), _native.CsrMap(dense)
        with torch.cuda.stream(b):
            H, y = batch.H('e'), table(x)
            H, y = H.cpu().numpy(), y.cpu().numpy()
        if not busy:
            batch.offsets.zero_()
            table.vals.zero_()
            del batch, table
            torch.cuda.synchronize()
    np.testing.assert_allclose(H, expected(m, off, 'e'), rtol=1e-13)
    np.testing.assert_allclose(y, np.repeat(dense.sum(1)[None], 3, 0), rtol=1e-13)
