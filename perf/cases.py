"""Timed cases: what programs ask of this package, from one dimer trajectory to
a 16384-sample disorder ensemble, each through a public entry point.

Every case is a dict of plain values.  ``prepare`` makes the model (or plan)
and inputs that a program holds before the call, ``run`` makes the call,
``work`` counts what the result cannot do without, and ``exact`` evaluates the
same fixed-step RK4 result in 64-bit torch from the formulas alone.

Results of single-precision propagation are returned in single precision: the
drivers hand them back in float64 containers, but a program that asks for
``precision='fp32'`` has seven digits and keeps them as such.
"""
import itertools
import math

import numpy as np
import torch

import qspectra_gb300 as qg
from qspectra_gb300 import workloads as wl
from qspectra_gb300.dynamics.heom import HEOMEquationOfMotion
from qspectra_gb300.simulate.adjoint import AbsorptionFit
from qspectra_gb300.simulate.ensemble import RedfieldEnsembleWorkload
from qspectra_gb300.simulate.third_order import ThirdOrderEngine

UC = 2 * math.pi * 2.99792458e-5            # cm^-1 to rad / fs
KB = 0.69503476                             # cm^-1 / K
RW_FIT = 12300.0                            # rotating frame of the fit


def listed():
    return [
        # the smallest call: one dimer trajectory, as in a notebook or a scan
        dict(name='dynamics_dimer', kind='dynamics', sites=2, points=120,
             precision='fp64', secular=False),
        # one 7-site trajectory of 1 ps, the plain form at its default precision
        dict(name='dynamics_site7', kind='dynamics', sites=7, points=1000,
             precision='fp64', secular=False),
        # one 7-site absorption spectrum, 2048 samples of 1 fs
        dict(name='absorption_site7', kind='absorption', sites=7, points=2048,
             precision='fp64', secular=False),
        # disorder averages through the drivers, at the default precision ...
        dict(name='dynamics_ensemble_fp64', kind='dynamics_ensemble', sites=7, points=500,
             samples=300, precision='fp64'),
        dict(name='absorption_ensemble_fp64', kind='absorption_ensemble', sites=7,
             points=1024, samples=600, precision='fp64'),
        # ... and in single precision, odd sizes
        dict(name='dynamics_ensemble_fp32', kind='dynamics_ensemble', sites=5, points=777,
             samples=2001, precision='fp32'),
        # the production step: spectrum and populations of 16384 samples
        dict(name='workload_fp32', kind='workload', sites=7, points=2048, dynamics=1000,
             samples=16384, precision='fp32', build='fp32'),
        # one step of fitting a Hamiltonian to a spectrum: misfit and gradient
        dict(name='fit_gradient', kind='fit', sites=7, points=2048, samples=1024,
             freqs=1024),
        # a small 2D spectrum, three population times
        dict(name='spectra_2d', kind='spectra_2d', sites=4, points=100, waits=3,
             precision='fp64'),
        # third-order response of a 24-site chain, 276 two-exciton states
        dict(name='third_order_chain24', kind='third_order', sites=24, points=128,
             samples=32, precision='fp32'),
        # hierarchical equations: one trimer trajectory, one ring ensemble
        dict(name='heom_trimer', kind='heom', sites=3, K=1, level=3, points=500,
             precision='fp64'),
        dict(name='heom_ring8', kind='heom_ensemble', sites=8, level=5, points=301,
             samples=64, precision='fp32'),
    ]


def draw(rng):
    def span(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(['dynamics', 'absorption', 'dynamics_ensemble', 'absorption_ensemble',
                       'workload', 'fit', 'spectra_2d', 'third_order', 'heom',
                       'heom_ensemble'])
    prec = rng.choice(['fp64', 'fp32'])
    c = dict(kind=kind)
    if kind == 'dynamics':
        c.update(sites=rng.randint(2, 8), points=span(40, 1000), precision=prec,
                 secular=rng.random() < 0.3)
    elif kind == 'absorption':
        c.update(sites=rng.randint(2, 16), points=span(128, 2048), precision=prec,
                 secular=rng.random() < 0.3)
    elif kind == 'dynamics_ensemble':
        c.update(sites=rng.randint(2, 8), points=span(60, 1000),
                 samples=span(16, 300 if prec == 'fp64' else 4096), precision=prec)
    elif kind == 'absorption_ensemble':
        c.update(sites=rng.randint(2, 12), points=span(128, 2048),
                 samples=span(16, 600 if prec == 'fp64' else 8192), precision=prec)
    elif kind == 'workload':
        c.update(sites=rng.randint(3, 8), points=span(256, 2048), dynamics=span(128, 1000),
                 samples=span(512, 12000) if prec == 'fp32' else span(32, 400),
                 precision=prec,
                 build='fp64' if prec == 'fp64' else rng.choice(['fp32', 'fp64']))
    elif kind == 'fit':
        c.update(sites=rng.randint(2, 8), points=span(256, 2048), samples=span(32, 1024),
                 freqs=span(128, 1024))
    elif kind == 'spectra_2d':
        c.update(sites=rng.randint(2, 6), points=span(30, 128), waits=rng.randint(1, 5),
                 precision=prec)
    elif kind == 'third_order':
        c.update(sites=rng.randint(6, 24), points=span(32, 128), samples=span(4, 32),
                 precision='fp32')
    elif kind == 'heom':
        c.update(sites=rng.randint(2, 4), K=rng.randint(0, 1), level=rng.randint(2, 4),
                 points=span(60, 500), precision=prec)
    else:
        c.update(sites=rng.randint(3, 8), level=rng.randint(2, 5), points=span(40, 301),
                 samples=span(4, 64 if prec == 'fp32' else 12), precision=prec)
    return c


# ------------------------------------------------------------------ inputs
def system(case, seed):
    """The numbers a case is made of: one-exciton Hamiltonian (cm^-1), dipoles,
    bath (kelvin, reorganisation energy, cutoff), disorder SD and RK4 step."""
    n, kind = case['sites'], case['kind']
    rs = np.random.RandomState([seed % (1 << 31), n])
    if kind == 'third_order':               # nearest and next-nearest couplings
        H = np.diag(rs.normal(12300.0, 100.0, n))
        H += -80.0 * (np.eye(n, k=1) + np.eye(n, k=-1)) + 15.0 * (np.eye(n, k=2) + np.eye(n, k=-2))
        bath, sd, dt = (300.0, 40.0, 100.0), 60.0, 2.0
    elif kind == 'heom_ensemble':           # a ring
        H = np.diag(rs.normal(12400.0, 80.0, n))
        for i in range(n):
            H[i, (i + 1) % n] = H[(i + 1) % n, i] = -100.0
        bath, sd, dt = (300.0, 35.0, 106.0), 50.0, 0.5
    else:                                   # a light-harvesting complex
        J = np.triu(rs.normal(0.0, 50.0, (n, n)), 1)
        H = J + J.T + np.diag(rs.uniform(12000.0, 12600.0, n))
        bath = (300.0 if kind == 'heom' else 77.0, 35.0, 106.0)
        sd, dt = 80.0, 2.0 if kind == 'spectra_2d' else 1.0
    dip = rs.randn(n, 3)
    dip /= np.linalg.norm(dip, axis=1, keepdims=True)
    return H, dip, bath, sd, dt


def shifts(case, seed, sd):
    """Site-energy shifts (samples, sites) of a case that is handed its draws."""
    rs = np.random.RandomState([seed % (1 << 31), 77, case['sites']])
    return sd * rs.randn(case['samples'], case['sites'])


def waits(case, dt):
    return np.array([0.0, 20.0, 60.0, 100.0, 160.0])[:case['waits']] * dt


def target(case, H):
    """A smooth band spectrum on the fit's frequency grid: the shape measured data have."""
    f = np.linspace(11800.0, 13000.0, case['freqs'])
    E, U = np.linalg.eigh(H)
    mu = U.sum(0) ** 2
    g = np.exp(-0.5 * ((f[:, None] - E[None, :] - 15.0) / 90.0) ** 2) / (90.0 * math.sqrt(2 * math.pi))
    return f, (math.pi / UC) * (g @ mu)


def prepare(case, seed):
    H, dip, (T, lam, gam), sd, dt = system(case, seed)
    n, kind = case['sites'], case['kind']
    bath = qg.DebyeBath(KB * T, lam, gam)
    s = dict(case=case, dt=dt)
    if kind == 'fit':
        f, y = target(case, H)
        s['fit'] = AbsorptionFit(n, shifts(case, seed, sd), f, dipoles=dip, temperature_K=T,
                                 cutoff_freq=gam, rw_freq=RW_FIT, dt=dt,
                                 nsteps=case['points'] - 1)
        s['target'] = torch.as_tensor(y).cuda()
        # away from the parameters that made the target, as in mid-fit
        s['theta'] = s['fit'].pack(H + np.diag(np.linspace(-9.0, 9.0, n)), 1.1 * lam)
        return s
    extra = wl.energy_spread_for_dt(H, dt, qg.CM_FS)
    ham = qg.ElectronicHamiltonian(H, bath=bath, dipoles=dip, disorder=wl.fwhm_for_sd(sd),
                                   random_seed=seed % (1 << 31), energy_spread_extra=extra)
    psi = np.zeros(n)
    psi[0] = 1.0
    s['psi'] = psi
    if kind == 'heom':
        s['model'] = qg.HEOMModel(ham, hilbert_subspace='e', unit_convert=qg.CM_FS,
                                  K=case['K'], level_cutoff=case['level'])
    elif kind == 'heom_ensemble':
        m = qg.HEOMModel(ham, hilbert_subspace='e', unit_convert=qg.CM_FS, K=0,
                         level_cutoff=case['level'])
        Hs = (torch.as_tensor(m.hamiltonian.H('e')).cuda()[None]
              + torch.diag_embed(torch.as_tensor(shifts(case, seed, sd)).cuda()))
        Hx, Hy = m.block_hamiltonians('ee', Hs)
        s['eom'] = HEOMEquationOfMotion(m, m.tables('ee'), Hx, Hy, 'ee', False)
        y0 = m.density_matrix_to_state_vector(np.outer(psi, psi), 'ee')
        s['y0'] = torch.as_tensor(y0).cuda().expand(case['samples'], -1).contiguous()
    else:
        sub = 'gef' if kind in ('spectra_2d', 'third_order') else 'ge'
        s['model'] = qg.RedfieldModel(ham, hilbert_subspace=sub, unit_convert=qg.CM_FS,
                                      secular=case.get('secular', False))
    if kind == 'workload':
        s['work'] = RedfieldEnsembleWorkload(s['model'], case['points'] * dt,
                                             case['dynamics'] * dt, psi)
        s['offsets'] = torch.as_tensor(shifts(case, seed, sd)).cuda()
    elif kind == 'third_order':
        s['engine'] = ThirdOrderEngine(s['model'], case['points'] * dt, [0.0, 200.0, 500.0],
                                       precision=case['precision'])
        s['offsets'] = torch.as_tensor(shifts(case, seed, sd)).cuda()
    return s


# -------------------------------------------------------------------- run
def kept(x, precision):
    if precision == 'fp64':
        return x
    if isinstance(x, torch.Tensor):
        return x.to(torch.complex64 if x.is_complex() else torch.float32)
    return x.astype(np.complex64 if np.iscomplexobj(x) else np.float32)


def run(s):
    c, dt = s['case'], s['dt']
    kind, prec, duration = c['kind'], c.get('precision'), c['points'] * s['dt']
    if kind in ('dynamics', 'heom'):
        t, rho = qg.simulate_dynamics(s['model'], s['psi'], duration=duration, precision=prec)
        return kept(rho, prec)
    if kind == 'absorption':
        f, X = qg.absorption_spectra(s['model'], duration, precision=prec)
        return f, kept(X, prec)
    if kind == 'dynamics_ensemble':
        t, rho = qg.simulate_dynamics(s['model'], s['psi'], duration=duration,
                                      ensemble_size=c['samples'], precision=prec)
        return kept(rho, prec)
    if kind == 'absorption_ensemble':
        f, X = qg.absorption_spectra(s['model'], duration, ensemble_size=c['samples'],
                                     precision=prec)
        return f, kept(X, prec)
    if kind == 'workload':
        X, pops, status = s['work'].run(s['offsets'], prec, build_precision=c['build'])
        return kept(X, prec), kept(pops, prec), status
    if kind == 'fit':
        theta = s['theta'].clone().requires_grad_(True)
        loss = s['fit'].misfit(theta, s['target'])
        loss.backward()
        return loss.detach(), theta.grad
    if kind == 'spectra_2d':
        (f1, t2, f3), X = qg.two_dimensional_spectra(
            s['model'], duration, population_times=waits(c, dt), precision=prec)
        return f1, f3, kept(X, prec)
    if kind == 'third_order':
        R = s['engine'].run(s['offsets'])
        return {g: kept(v, prec) for g, v in R.items()}
    t = np.arange(0, duration, dt)
    return kept(qg.integrate(s['eom'], s['y0'], t, precision=prec, heom_nodes=1), prec)


# ------------------------------------------------------------------- work
def work(case):
    """Inputs and outputs once; one application of the step's linear map per
    sample and step (a real map of n^2 coordinates for a density matrix, a
    complex one of n for a coherence), the generator's own terms for HEOM."""
    n, T, S = case['sites'], case['points'], case.get('samples', 1)
    kind, B = case['kind'], 8 if case.get('precision') == 'fp32' else 16
    ee, eg = 2.0 * n ** 4, 8.0 * n ** 2
    ins = 8.0 * (n * n + S * n)
    if kind in ('dynamics', 'dynamics_ensemble'):
        return dict(bytes=ins + B * T * n * n, flops=S * T * ee)
    if kind in ('absorption', 'absorption_ensemble'):
        return dict(bytes=ins + 8.0 * T, flops=S * T * eg + 16.0 * T * math.log2(2 * T))
    if kind == 'workload':
        return dict(bytes=ins + B / 2 * (2 * T + n * case['dynamics']),
                    flops=S * (T * eg + case['dynamics'] * ee))
    if kind == 'fit':
        return dict(bytes=ins + 8.0 * (case['freqs'] + n * n), flops=S * T * 3 * eg)
    if kind == 'spectra_2d':
        p = n * (n - 1) // 2
        fe = 16.0 * (n * p * p + p * n * n)
        return dict(bytes=ins + 16.0 * case['waits'] * 4 * T * T,
                    flops=T * 4 * fe + case['waits'] * T * T * 8.0 * n * n)
    if kind == 'third_order':
        p = n * (n - 1) // 2
        fe = 8.0 * (n * p * p + p * n * n)
        return dict(bytes=ins + 2 * 3 * B * T * T,
                    flops=S * (T * 4 * fe + 2 * 3 * T * T * 8.0 * n * n))
    nodes = math.comb(n * (case.get('K', 0) + 1) + case['level'] - 1, case['level'] - 1)
    rhs = nodes * (16.0 * n ** 3 + 8.0 * n * n * 2 * n)
    return dict(bytes=ins + B * S * T * n * n, flops=S * T * 4 * rhs)


# ------------------------------------------------------------------ exact
def f64(x, dtype=torch.float64):
    return torch.as_tensor(np.asarray(x), dtype=dtype).cuda()


def pairs(n):
    return list(itertools.combinations(range(n), 2))


def lift(H1):
    """Two-exciton matrices (S, P, P) of one-exciton ones."""
    p = pairs(H1.shape[-1])
    i, j = f64([a for a, _ in p], torch.long), f64([b for _, b in p], torch.long)
    def same(a, b):
        return (a[:, None] == b[None, :]).double()
    def el(a, b):
        return H1[:, a][:, :, b]
    return (el(j, j) * same(i, i) + el(j, i) * same(i, j)
            + el(i, j) * same(j, i) + el(i, i) * same(j, j))


def debye(x, bath, lam=None):
    """One-sided correlation function, 999 Matsubara terms."""
    T, gam = KB * bath[0], bath[2]
    lam = bath[1] if lam is None else lam
    nu = 2 * math.pi * T * torch.arange(1, 1000, dtype=torch.float64, device=x.device)
    w = nu / (nu ** 2 - gam ** 2)
    flat = x.reshape(-1)
    step = len(flat) if flat.requires_grad else 1 << 15
    tail = torch.cat([(w / (nu - 1j * v[:, None])).sum(1) for v in flat.split(step)])
    head = (1 / math.tan(gam / (2 * T)) - 1j) / (gam - 1j * flat)
    c = lam * gam * (head + 4 * T * tail)
    return torch.where(flat == 0, lam * (2 * T / gam - 1j), c).reshape(x.shape)


class Exact:
    """Redfield generator of a batch, per manifold, in the site basis:
    d rho = -(A_X rho + rho A_Y^H) + sum_i (M_i^X rho K_i^Y + K_i^X rho M_i^Y^H),
    M_i = U (K_i o C) U^T, A = sum_i K_i M_i + i H."""

    def __init__(self, case, seed, offsets=None, sub='ge'):
        H, self.dip, self.bath, sd, self.dt = system(case, seed)
        self.n = n = case['sites']
        self.rw = np.trace(H) / n
        off = np.zeros((1, n)) if offsets is None else offsets
        self.H1 = f64(H - self.rw * np.eye(n))[None] + torch.diag_embed(f64(off))
        self.S = len(off)
        self.man = {}
        for x in sub:
            h = dict(g=lambda: torch.zeros_like(self.H1[:, :1, :1]), e=lambda: self.H1,
                     f=lambda: lift(self.H1))[x]()
            sites = dict(g=[()], e=[(i,) for i in range(n)], f=pairs(n))[x]
            occ = f64([[float(i in st) for st in sites] for i in range(n)])
            E, U = torch.linalg.eigh(h)
            C = debye(E[:, None, :] - E[:, :, None], self.bath)       # C[b, c] = C(E_c - E_b)
            M = []
            for i in range(n):
                Ki = U.transpose(1, 2) @ (occ[i][:, None] * U)
                M.append(U.to(C.dtype) @ (Ki * C) @ U.transpose(1, 2).to(C.dtype))
            M = torch.stack(M, 1)
            A = torch.einsum('ia,siab->sab', occ.to(M.dtype), M) + 1j * h
            self.man[x] = (h, U, occ, M, A)

    def maps(self, block):
        (_, _, ox, Mx, Ax), (_, _, oy, My, Ay) = (self.man[x] for x in block)
        Qx = torch.einsum('ib,siac->sbac', oy.to(Mx.dtype), Mx) - Ax[:, None]
        Qy = torch.einsum('ia,sibd->sabd', ox.to(My.dtype), My) - Ay[:, None]
        return UC * Qx, UC * Qy

    def dense(self, block, secular=False):
        """(S, m, m) generator, m = nx ny, on column-stacked elements a + nx b."""
        Qx, Qy = self.maps(block)
        nx, ny = Qx.shape[-1], Qy.shape[-1]
        L = torch.zeros(self.S, ny, nx, ny, nx, dtype=Qx.dtype, device=Qx.device)
        for b in range(ny):
            L[:, b, :, b, :] += Qx[:, b]
        for a in range(nx):
            L[:, :, a, :, a] += Qy[:, a].conj()
        L = L.reshape(self.S, nx * ny, nx * ny)
        if secular:
            W = torch.einsum('sbd,sac->sbadc', self.man[block[1]][1], self.man[block[0]][1])
            W = W.reshape(self.S, nx * ny, nx * ny).to(L.dtype)
            k = torch.arange(nx * ny, device=L.device)
            a, b = k % nx, k // nx
            pop = (a == b) & (block[0] == block[1])
            keep = (pop[:, None] & pop[None, :]) | torch.eye(nx * ny, dtype=bool, device=L.device)
            L = W @ ((W.transpose(1, 2) @ L @ W) * keep) @ W.transpose(1, 2)
        return L

    def step(self, block, secular=False):
        A = self.dt * self.dense(block, secular)
        A2 = A @ A
        return A + A2 / 2 + A2 @ (A / 6 + A2 / 24)


def steps(D, y, count, save):
    """save(y_n), n = 0 .. count, for y_{n+1} = y_n + D y_n; y (S, m, k)."""
    out = [save(y)]
    for _ in range(count):
        y = y + D @ y
        out.append(save(y))
    return torch.stack(out)


def transform(x, dt, sign):
    """(grid minus rw, transform) along the first axis on the padded FFT grid."""
    n = len(x)
    f = np.fft.fftshift(np.fft.fftfreq(2 * n - 1, dt * UC / (2 * math.pi)))
    f = -f[::-1] if sign == 1 else f
    ph = torch.exp(1j * sign * UC * dt * f64(f)[:, None] * torch.arange(n, device=x.device).double())
    return f, dt * torch.tensordot(ph, x.to(torch.complex128), 1)


def drawn_shifts(case, seed, sd):
    """The disorder draws of an ensemble driver: one seeded stream per sample."""
    return sd * np.array([np.random.RandomState([seed % (1 << 31), k]).randn(case['sites'])
                          for k in range(case['samples'])])


def exact(case, seed):
    kind, n = case['kind'], case['sites']
    with torch.no_grad():
        if kind == 'fit':
            return exact_fit(case, seed)
        if kind in ('heom', 'heom_ensemble'):
            return exact_heom(case, seed)
        if kind in ('spectra_2d', 'third_order'):
            return exact_third(case, seed)
        sd = system(case, seed)[3]
        off = (shifts(case, seed, sd) if kind == 'workload'
               else drawn_shifts(case, seed, sd) if 'samples' in case else None)
        ex = Exact(case, seed, off)
        secular = case.get('secular', False)
        pops = X = None
        if 'dynamics' in kind or kind == 'workload':
            y = torch.zeros(ex.S, n * n, 1, dtype=torch.complex128, device='cuda')
            y[:, 0] = 1.0
            count = case['dynamics' if kind == 'workload' else 'points'] - 1
            r = steps(ex.step('ee', secular), y, count, lambda v: v[:, :, 0].mean(0))
            pops = r.reshape(-1, n, n).transpose(1, 2)
        if 'absorption' in kind or kind == 'workload':
            mu = f64(ex.dip[:, 0], torch.complex128)
            sig = steps(ex.step('eg', secular), mu.expand(ex.S, n)[:, :, None],
                        case['points'] - 1, lambda v: (v[:, :, 0] @ mu).mean())
            f, X = transform(sig, ex.dt, 1)
        if kind == 'workload':
            return X.real, torch.diagonal(pops, dim1=1, dim2=2).real, None
        return pops if X is None else (f + ex.rw, X.real)


def exact_fit(case, seed):
    H, dip, bath, sd, dt = system(case, seed)
    n = case['sites']
    f, y = target(case, H)
    iu = torch.triu_indices(n, n, 1, device='cuda')
    H0 = H + np.diag(np.linspace(-9.0, 9.0, n))
    theta = f64(np.concatenate([np.diag(H0), H0[np.triu_indices(n, 1)], [1.1 * bath[1]]]))
    with torch.enable_grad():
        theta.requires_grad_(True)
        J = torch.zeros(n, n, dtype=torch.float64, device='cuda').index_put((iu[0], iu[1]), theta[n:-1])
        h = J + J.T + torch.diag(theta[:n]) + torch.diag_embed(f64(shifts(case, seed, sd)))
        h = h - RW_FIT * torch.eye(n, device='cuda')
        E, U = torch.linalg.eigh(h)
        C = debye(E[:, None, :] - E[:, :, None], bath, theta[-1])
        Uc = U.to(C.dtype)
        G = (((U * U).to(C.dtype) @ C) * Uc) @ Uc.transpose(1, 2)
        A = -dt * UC * (G + 1j * h)
        A2 = A @ A
        D = A + A2 / 2 + A2 @ (A / 6 + A2 / 24)
        mu = f64(dip[:, 0], torch.complex128)
        sig = steps(D, mu.expand(len(h), n)[:, :, None], case['points'] - 1,
                    lambda v: (v[:, :, 0] @ mu).mean())
        k = torch.arange(case['points'], device='cuda').double()
        spec = (dt * torch.exp(1j * UC * dt * (f64(f) - RW_FIT)[:, None] * k) @ sig).real
        loss = ((spec - f64(y)) ** 2).sum() / (f64(y) ** 2).sum()
        loss.backward()
    return loss.detach(), theta.grad


def exact_third(case, seed):
    H, dip, bath, sd, dt = system(case, seed)
    n, T = case['sites'], case['points']
    single = case['kind'] == 'spectra_2d'
    ex = Exact(case, seed, None if single else shifts(case, seed, sd), 'gef')
    t2 = waits(case, dt) if single else np.array([0.0, 200.0, 500.0])
    S, p = ex.S, pairs(n)
    c16 = dict(dtype=torch.complex128, device='cuda')
    mu = f64(dip[:, 0], torch.complex128)
    up = torch.zeros(len(p), n, **c16)           # dipole e -> f
    for q, (k, l) in enumerate(p):
        up[q, k], up[q, l] = mu[l], mu[k]
    # t3 in the Heisenberg picture: rows w(t3) with w . rho the signal
    Deg, Dee = ex.step('eg'), ex.step('ee')
    w_eg = steps(Deg.transpose(1, 2), mu.expand(S, n)[:, :, None], T - 1, lambda v: v[:, :, 0])
    Qx, Qy = ex.maps('fe')

    def back(w):                                 # transpose of the 'fe' generator
        return (torch.einsum('sbac,sab->scb', Qx, w)
                + torch.einsum('sabd,sab->sad', Qy.conj(), w))

    w, w_fe = up.expand(S, -1, -1), []
    for k in range(T):
        w_fe.append(torch.einsum('sfe,fk->ske', w, up))          # V2 from the left, then tr
        if k < T - 1:
            k1 = back(w); k2 = back(w + dt / 2 * k1); k3 = back(w + dt / 2 * k2)
            k4 = back(w + dt * k3)
            w = w + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    w_fe = torch.stack(w_fe)                     # (T, S, e, e'): coefficient of rho[e, e']
    # V2 '+' on 'ee' towards 'eg': minus the right product rho mu
    W = w_fe - torch.einsum('tsa,b->tsab', w_eg, mu)
    g3 = torch.einsum('tsa,a->ts', w_eg, mu)     # V2 '+' on 'gg' towards 'eg'
    out = {}
    for geo in ('-++',) if single else ('-++', '+-+'):
        if geo == '-++':                         # 'ge': V0 '-' gives -rho0 mu, V1 '+' from the left
            s1 = steps(ex.step('ge'), -mu.expand(S, n)[:, :, None], T - 1, lambda v: v[:, :, 0])
            r = torch.einsum('tsb,a->tsab', s1, mu)
            rg = -torch.einsum('tsb,b->ts', s1, mu)
        else:                                    # 'eg': V0 '+' from the left, V1 '-' on either side
            s1 = steps(Deg, mu.expand(S, n)[:, :, None], T - 1, lambda v: v[:, :, 0])
            r = -torch.einsum('tsa,b->tsab', s1, mu)
            rg = torch.einsum('tsa,a->ts', s1, mu)
        y = r.permute(1, 3, 2, 0).reshape(S, n * n, T)           # column-stacked
        cols, at = [], 0
        for k in np.rint(t2 / dt).astype(int):
            for _ in range(k - at):
                y = y + Dee @ y
            at = k
            z = y.reshape(S, n, n, T)                            # [s, b, a, t1]
            R = torch.einsum('sbat,usab->tu', z, W) + torch.einsum('ts,us->tu', rg, g3)
            cols.append(R)
        out[geo] = torch.stack(cols, 1)          # (T1, T2, T3)
    if not single:
        return out
    f1, X = transform(out['-++'], dt, -1)
    f3, X = transform(X.permute(2, 1, 0), dt, 1)
    return f1 + ex.rw, f3 + ex.rw, X.permute(2, 1, 0)


def exact_heom(case, seed):
    H, dip, (Tk, lam, gam), sd, dt = system(case, seed)
    n, K, T = case['sites'], case.get('K', 0), KB * Tk
    off = shifts(case, seed, sd) if 'samples' in case else np.zeros((1, n))
    h = (f64(H - np.trace(H) / n * np.eye(n))[None] + torch.diag_embed(f64(off)))
    h = h.to(torch.complex128)[:, None]
    S, modes = len(off), n * (K + 1)
    nu = 2 * math.pi * T * np.arange(K + 5001)
    nu[0] = gam
    c = np.empty(K + 5001, complex)
    c[0] = lam * gam * (1 / math.tan(gam / (2 * T)) - 1j)
    c[1:] = 4 * lam * gam * T * nu[1:] / (nu[1:] ** 2 - gam ** 2)
    rest = float(np.sum(c[K + 1:] / nu[K + 1:]).real)
    nodes = [v for total in range(case['level'])
             for v in itertools.combinations_with_replacement(range(modes), total)]
    occ = np.zeros((len(nodes), modes), int)
    for i, v in enumerate(nodes):
        for m in v:
            occ[i, m] += 1
    where = {tuple(v): i for i, v in enumerate(occ)}
    none = len(nodes)                            # a node of zeros
    eye = torch.eye(n, device='cuda')
    damp = f64(occ @ np.tile(nu[:K + 1], n))[:, None, None] + 2 * rest * (1 - eye.double())
    up, down, num = [], [], []
    for m in range(modes):
        e = np.eye(modes, dtype=int)[m]
        up.append(f64([where.get(tuple(v + e), none) for v in occ], torch.long))
        down.append(f64([where.get(tuple(v - e), none) for v in occ], torch.long))
        num.append(f64(occ[:, m])[:, None, None])
    rho = torch.zeros(S, len(nodes) + 1, n, n, dtype=torch.complex128, device='cuda')
    rho[:, 0, 0, 0] = 1.0

    def rhs(r):
        x = r[:, :-1]
        d = -1j * (h @ x - x @ h) - damp * x
        for m in range(modes):
            j, ck = m // (K + 1), c[m % (K + 1)]
            u, v = r[:, up[m]], num[m] * r[:, down[m]]
            d[:, :, j, :] += -1j * (u + ck * v)[:, :, j, :]
            d[:, :, :, j] += 1j * (u + np.conj(ck) * v)[:, :, :, j]
        return torch.cat([UC * d, torch.zeros_like(r[:, -1:])], 1)

    out = [rho[:, 0]]
    for _ in range(case['points'] - 1):
        k1 = rhs(rho); k2 = rhs(rho + dt / 2 * k1); k3 = rhs(rho + dt / 2 * k2)
        k4 = rhs(rho + dt * k3)
        rho = rho + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        out.append(rho[:, 0])
    out = torch.stack(out, 1)                    # (S, T, n, n)
    if 'samples' in case:
        return out.transpose(2, 3).reshape(S, case['points'], n * n)
    return out[0]
