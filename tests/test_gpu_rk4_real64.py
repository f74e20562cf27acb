"""FP64 real (Hermitian) ensemble loop against a NumPy recurrence and the
complex loop."""
import numpy as np
import pytest
import torch

import qspectra_gb300 as qg
from conftest import rel_err
from qspectra_gb300 import _native
from qspectra_gb300 import workloads as wl
from qspectra_gb300.simulate import ensemble as ens

pytestmark = pytest.mark.gpu


# every block size; samples that fill no CTA, some CTAs unevenly, one per SM
# and more than one group a CTA; no step, one and several
@pytest.mark.parametrize('nb', [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize('S,nsteps', [(1, 0), (1, 37), (3, 1), (153, 2), (307, 12), (1700, 5)])
def test_real_mean_matches_numpy(nb, S, nsteps):
    m = nb * nb
    rng = np.random.RandomState(m + S)
    D = 0.05 * rng.randn(S, m, m) - 0.05 * np.eye(m)
    x0 = rng.randn(m)
    for sel in (list(range(m)), [m - 1, 0]):
        out, status = _native.rk4_real_mean_f64(torch.as_tensor(D).cuda(),
                                                torch.as_tensor(x0), nsteps, sel)
        x = np.repeat(x0[None], S, 0)
        ref = [x.mean(0)[sel]]
        for _ in range(nsteps):
            x = x + np.einsum('sij,sj->si', D, x)
            ref.append(x.mean(0)[sel])
        # m products and S samples a value, 37 steps
        assert rel_err(out.cpu().numpy(), np.array(ref)) < 1e-13
        assert int(status.item()) == 0


def test_a_non_finite_sample_is_reported():
    D = torch.zeros((5, 9, 9), dtype=torch.float64, device='cuda')
    D[3, 2, 2] = float('nan')
    _, status = _native.rk4_real_mean_f64(D, torch.ones(9), 3, [0])
    assert int(status.item()) & _native.QSX_ERR_NONFINITE


def model(n, secular=False, basis='site', sub='ge'):
    H = wl.fmo7_hamiltonian(n_sites=n, seed=n)
    ham = qg.ElectronicHamiltonian(H, bath=qg.DebyeBath(qg.CM_K * 77, 35, 106),
                                   dipoles=[[1, 0, 0]] * n, disorder=wl.fwhm_for_sd(80.0),
                                   random_seed=1)
    return qg.RedfieldModel(ham, hilbert_subspace=sub, unit_convert=qg.CM_FS, secular=secular,
                            evolve_basis=basis)


@pytest.mark.parametrize('n', [2, 3, 7, 8, 9])
@pytest.mark.parametrize('kind', ['pure', 'complex', 'mixed', 'not hermitian'])
@pytest.mark.parametrize('form', [(False, 'site', 'ge'), (False, 'site', 'gef'),
                                  (True, 'site', 'ge'), (True, 'eigen', 'ge')])
def test_driver_matches_the_complex_loop(n, kind, form):
    if form[2] == 'gef' and n > 7:
        pytest.skip('more than 32 states')
    m = model(n, *form)
    rng = np.random.RandomState(n)
    psi = rng.randn(n) + 1j * rng.randn(n) * (kind != 'pure')
    rho = psi / np.linalg.norm(psi)
    if kind in ('mixed', 'not hermitian'):
        rho = np.outer(rho.conj(), rho) * 0.5 + np.eye(n) / (2 * n)
    if kind == 'not hermitian':
        rho[0, 1] += 1e-13
    out = []
    for on in (True, False):
        ens.set_hermitian_form(on)
        if n == 9:   # 81 rows: past the batched propagator, refused either way
            with pytest.raises(_native.QsxError):
                qg.simulate_dynamics(m, rho, duration=60 * m.time_step, ensemble_size=5)
            ens.set_hermitian_form(True)
            continue
        try:
            _, r = qg.simulate_dynamics(m, rho, duration=60 * m.time_step, ensemble_size=5,
                                        precision='fp64')
        finally:
            ens.set_hermitian_form(True)
        out.append(r)
    assert n == 9 or rel_err(out[0], out[1]) < 1e-13
