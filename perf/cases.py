"""The work that users of the propagators have them do, as cases to be timed.

Every case advances a state through a public entry point: ``propagate`` of the
complex128 classes (Wigner2D with Caldeira-Leggett, ODM or no damping,
Fokker-Planck, Gross-Pitaevskii, Dirac2D, Dirac3D), ``Run`` with its frames,
``WignerBatch.run`` (both precisions) and ``WignerControl.propagate`` with its
backward sweep.  Sizes and parameters are those of this repository's benchmark
and tests (double well 0.05 x^4 - x^2, Caldeira-Leggett gamma = 0.1, dt = 0.005;
Coulomb packets for the spinors; the 64-instance mixed-grid batch; the 512^2
control problem); the grids are the powers of two that the propagators take,
square and not.  The seed moves the initial packet and the potential's
coefficients (the ``cf[]`` slots of the expression strings).
"""
import math

import numpy as np
import torch

DEV = 'cuda'
POT = 'cf[0]*pow(x,4) + cf[1]*pow(x,2) + cf[2]*x'
DPOT = '4.*cf[0]*pow(x,3) + 2.*cf[1]*x + cf[2]'
POT_T = POT + ' + 0.2*x*sin(3.*t)'
DPOT_T = DPOT + ' + 0.2*sin(3.*t)'
COULOMB2 = '-1./sqrt(x*x+y*y+0.5)'
COULOMB3 = '-1./sqrt(x*x+y*y+z*z+0.5)'
FIELDS2 = (COULOMB2, '-0.5*y', '0.5*x', '0.')
FIELDS3 = (COULOMB3, '-0.5*y', '0.5*x', '0.')
C_LIGHT = 137.036


def _wigner(name, n_x, n_p, steps, **more):
    case = dict(name=name, kind='wigner', n_x=n_x, n_p=n_p, steps=steps, amp=10., dt=0.005, hbar=1., mass=1.,
                gamma=0.1, d_lambda=0., damping='CaldeiraLeggett', timedep=False, form='lie')
    case.update(more)
    return case


def listed():
    return [
        # a first look at a system: small grid, undamped coherent state, many short steps
        _wigner('wigner_256_undamped', 256, 256, 200, gamma=0., dt=0.01),
        # a whole Run() of a small damped system: host state in, frames and observables out
        _wigner('run_128x64_frames', 128, 64, 60, form='run', damping='CaldeiraLeggett', skip=10),
        # the reference's main workload: a fine grid with Caldeira-Leggett damping
        _wigner('wigner_1024_damped', 1024, 1024, 20, amp=12.),
        # a wide, flat grid, driven potential, hbar and mass not 1, diffusion in lambda
        _wigner('wigner_2048x256_driven', 2048, 256, 20, hbar=0.8, mass=1.7, d_lambda=0.002, timedep=True),
        # Lindblad (ODM) damping of a harmonic-like well
        _wigner('wigner_512_odm', 512, 512, 10, amp=12., gamma=0.0175, damping='ODM'),
        # a condensate: Strang steps with the mean-field term
        _wigner('gpitaevskii_512', 512, 512, 10, form='gp'),
        # a parameter scan: 64 instances of uneven grids together, both precisions
        dict(name='batch_64_mixed', kind='batch', precision='mixed', count=64, low=128, high=1024, pick=0, steps=10),
        dict(name='batch_64_f32', kind='batch', precision='f32', count=64, low=128, high=1024, pick=0, steps=10),
        # relativistic packets in two and three dimensions
        dict(name='dirac2d_512', kind='dirac2', n_x=512, n_y=512, steps=20, dt=1e-4),
        dict(name='dirac3d_128', kind='dirac3', n_x=128, n_y=128, n_z=128, steps=4, dt=1e-4),
        # gradients of a control problem, damped in complex128 and a quick undamped one in complex64
        dict(name='control_512_c128', kind='control', n_x=512, n_p=512, precision='c128', gamma=0.1, steps=60,
             checkpoint=20),
        dict(name='control_256_c64', kind='control', n_x=256, n_p=256, precision='c64', gamma=0., steps=60,
             checkpoint=20),
    ]


def draw(rng):
    """One more case: axes spread over their logarithms, steps so that the work stays below the listed cases'."""
    def axis(low, high):
        return 1 << rng.randint(int(math.log2(low)), int(math.log2(high)))

    kind = rng.choice(['wigner', 'wigner', 'wigner', 'run', 'gp', 'batch', 'dirac2', 'dirac3', 'control'])
    if kind in ('wigner', 'run', 'gp'):
        n_x, n_p = axis(32, 2048 if kind == 'wigner' else 512), axis(32, 1024 if kind == 'wigner' else 512)
        damping, gamma, form = 'CaldeiraLeggett', rng.uniform(0.02, 0.2), {'wigner': 'lie'}.get(kind, kind)
        cap = 16 << 20
        if kind == 'wigner':
            form = rng.choice(['lie', 'lie', 'kvn'])
            if form == 'lie' and rng.random() < 0.3:
                damping, cap = 'ODM', 2 << 20
        elif kind == 'gp':
            cap = 2 << 20
        elif kind == 'run':
            cap = 1 << 20
        if rng.random() < 0.25:
            gamma = 0.
        if damping == 'ODM' and gamma != 0.:
            gamma *= 0.1
        case = _wigner('', n_x, n_p, max(1, min(rng.randint(5, 97), cap // (n_x * n_p))), form=form,
                       amp=rng.uniform(8., 12.), hbar=rng.choice([1., 0.8]), mass=rng.choice([1., 1.7]),
                       gamma=gamma, d_lambda=rng.choice([0., 0.002]), damping=damping, timedep=rng.random() < 0.4)
        if form == 'run':
            case['skip'] = rng.randint(3, 20)
    elif kind == 'batch':
        low = axis(64, 512)
        high = min(1024, low * rng.choice([1, 2, 4, 8]))
        case = dict(kind='batch', precision=rng.choice(['mixed', 'mixed', 'f32']), count=rng.randint(1, 40), low=low,
                    high=high, pick=rng.randint(1, 1 << 20), steps=rng.randint(2, 9))
    elif kind == 'dirac2':
        n_x, n_y = axis(64, 1024), axis(64, 512)
        case = dict(kind='dirac2', n_x=n_x, n_y=n_y, dt=1e-4, steps=max(1, min(rng.randint(3, 41), (5 << 20) // (n_x * n_y))))
    elif kind == 'dirac3':
        n_x, n_y, n_z = axis(32, 128), axis(32, 128), axis(32, 128)
        case = dict(kind='dirac3', n_x=n_x, n_y=n_y, n_z=n_z, dt=1e-4, steps=rng.randint(1, 4))
    else:
        n_x, n_p = axis(64, 512), axis(64, 512)
        case = dict(kind='control', n_x=n_x, n_p=n_p, precision=rng.choice(['c128', 'c128', 'c64']),
                    gamma=rng.choice([0., rng.uniform(0.02, 0.2)]), steps=rng.randint(9, 60),
                    checkpoint=rng.randint(4, 25))
    case.pop('name', None)
    return case


# ---------------------------------------------------------------- inputs
def _index(n, dev):
    """FFT-shifted signed index of each array position."""
    k = torch.arange(n, dtype=torch.float64, device=dev)
    return torch.where(k < n / 2, k, k - n)


def _draws(seed, n):
    return np.random.default_rng([seed, 77]).uniform(0., 1., n)


def _cat(n_x, n_p, amp, x0, p0, dev):
    """Two packets at +-x0 with their interference (a Wigner function with negative parts)."""
    x = (2. * amp / n_x * _index(n_x, dev))[None, :]
    p = (2. * amp / n_p * _index(n_p, dev))[:, None]
    q = p - p0
    return (torch.exp(-(x - x0) ** 2 - q * q) + torch.exp(-(x + x0) ** 2 - q * q) +
            2. * torch.exp(-x * x - q * q) * torch.cos(2. * x0 * q))


def _wigner_inputs(case, seed, dev):
    u = _draws(seed, 4)
    coef = (0.04 + 0.02 * u[0], -1. + 0.2 * u[1], 0.1 * u[2])
    W0 = _cat(case['n_x'], case['n_p'], case['amp'], 1.5 + u[3], 0.5 * u[2], dev).to(torch.complex128)
    return coef, W0


def _wigner_instance(case, coef):
    import pywignercuda_b200 as P
    c = case
    pot, dpot = (POT_T, DPOT_T) if c['timedep'] else (POT, DPOT)
    base = {'gp': P.GPU_Wigner2D_GPitaevskii, 'kvn': P.GPU_FokkerPlank2D_FFT}.get(c['form'], P.GPU_Wigner2D_FFT)

    class Instance(base):
        def __init__(self):
            self.coefficients = coef
            self.dampingFunction, self.grossPitaevskiiCoefficient = c['damping'], 0.
            self.GPitaevskiiCoeff = 0.5
            self.fp_Damping_String = 'fabs(p)' if c['damping'] != 'ODM' else 'p*p/sqrt(p*p + 0.5)'
            self.epsilon, self.L_material = 0.5, 3.
            self.SetTimeTrack(c['dt'], c['steps'], c.get('skip', 10 ** 9), fileName='')
            args = (c['n_x'], c['n_p'], c['amp'], c['amp'], c['hbar'], c['mass'], c['gamma'], c['d_lambda'],
                    c['gamma'], pot, dpot)
            base.__init__(self, *(args if c['form'] == 'kvn' else args + ('0.5*p*p',)))
    return Instance()


def _batch_sizes(case):
    """The grids and damping rates of the batch (`pick` 0: the benchmark's 64 instances)."""
    rng = np.random.default_rng(case['pick'])
    sizes = [n for n in (64, 128, 256, 512, 1024) if case['low'] <= n <= case['high']]
    n_x = rng.choice(sizes, size=case['count'])
    n_p = n_x if case['pick'] == 0 else rng.choice(sizes, size=case['count'])
    gamma = rng.uniform(0., 0.2, case['count'])
    if case['pick']:
        gamma[rng.uniform(size=case['count']) < 0.2] = 0.
    return n_x, n_p, gamma


def _batch_inputs(case, seed, dev):
    n_x, n_p, gamma = _batch_sizes(case)
    rng = np.random.default_rng([seed, 78])
    out = []
    for nx, npp, g in zip(n_x, n_p, gamma):
        v4, v2, x0, p0 = rng.uniform(0.01, 0.1), rng.uniform(-1., 0.5), rng.uniform(-2., 2.), rng.uniform(-1., 1.)
        x = (20. / nx * _index(int(nx), dev))[None, :]
        p = (20. / npp * _index(int(npp), dev))[:, None]
        W = torch.exp(-((x - x0) ** 2 + (p - p0) ** 2))
        W = (W / (W.sum() * (400. / (nx * npp)))).float()
        out.append((dict(n_x=int(nx), n_p=int(npp), x_amplitude=10., dt=0.005, gamma=float(g), d_theta=float(g),
                         v4=float(v4), v2=float(v2)), W))
    return out


def _spinor(case, seed, dev):
    u = _draws(seed, 6)
    grid = [case[k] for k in ('n_z', 'n_y', 'n_x') if k in case]
    axes = [(24. / n * _index(n, dev)).reshape([-1 if i == j else 1 for j in range(len(grid))])
            for i, n in enumerate(grid)][::-1]                      # x, y(, z)
    mom = [4. + 2. * u[0], 2. * u[1] - 1., 2. * u[2] - 1.][:len(axes)]
    env = sum((q - (u[3 + i] - 0.5)) ** 2 for i, q in enumerate(axes))
    phase = sum(k * q for k, q in zip(mom, axes))
    rho = torch.exp(-0.5 * env) * torch.exp(1j * phase)
    p0 = math.sqrt(sum(k * k for k in mom) + C_LIGHT ** 2)
    pz = mom[2] if len(mom) > 2 else 0.
    return torch.stack([rho * (p0 + C_LIGHT), rho * 0., rho * pz, rho * complex(mom[0], mom[1])]).contiguous()


def _dirac_instance(case):
    import pywignercuda_b200 as P
    three = case['kind'] == 'dirac3'
    base, fields = (P.GPU_Dirac3D, FIELDS3) if three else (P.GPU_Dirac2D, FIELDS2)
    shape = tuple(case[k] for k in ('n_x', 'n_y', 'n_z') if k in case)

    class Instance(base):
        def __init__(self):
            self.mass, self.c, self.hBar, self.fileName = 1., C_LIGHT, 1., ''
            (self.Potential_0_String, self.Potential_1_String, self.Potential_2_String,
             self.Potential_3_String) = fields
            base.__init__(self, shape, (12.,) * len(shape), case['dt'], case['steps'], 10 ** 9)
    return Instance()


def _control_inputs(case, seed, dev):
    u = _draws(seed, 6)

    def packet(x0, p0):
        x = (20. / case['n_x'] * _index(case['n_x'], dev))[None, :]
        p = (20. / case['n_p'] * _index(case['n_p'], dev))[:, None]
        W = torch.exp(-((x - x0) ** 2 + (p - p0) ** 2))
        return W / (W.sum() * (400. / (case['n_x'] * case['n_p'])))
    eps = torch.from_numpy(np.random.default_rng([seed, 79]).normal(0., 0.1, case['steps'])).to(dev)
    coef = torch.tensor([0.05 + 0.01 * u[0], -1. + 0.1 * u[1]], dtype=torch.float64, device=dev)
    return packet(-2. + u[2], 0.5 * u[3]), packet(2. * u[4] - 1., 0.5 * u[5]), eps, coef


def prepare(case, seed):
    kind = case['kind']
    if kind == 'wigner':
        coef, W0 = _wigner_inputs(case, seed, DEV)
        inst = _wigner_instance(case, coef)
        if case['form'] == 'run':
            inst.W_init = W0.cpu().numpy()
        return dict(case=case, inst=inst, W0=W0)
    if kind == 'batch':
        from pywignercuda_b200.batch import WignerBatch, instance
        items = _batch_inputs(case, seed, DEV)
        # the 4-warp tile: what autotuning picks on the benchmark's batch, here without its three compilations
        batch = WignerBatch([instance(**d) for d, _ in items], warps=4, precision=case['precision'])
        W0 = torch.cat([W.reshape(-1) for _, W in items])
        return dict(case=case, inst=batch, W0=W0, W=torch.empty_like(W0))
    if kind in ('dirac2', 'dirac3'):
        return dict(case=case, inst=_dirac_instance(case), W0=_spinor(case, seed, DEV))
    from pywignercuda_b200.adjoint import WignerControl
    W0, target, eps, coef = _control_inputs(case, seed, DEV)
    inst = WignerControl(case['n_x'], case['n_p'], x_amplitude=10., dt=0.005, gamma=case['gamma'],
                         d_theta=case['gamma'], precision=case['precision'])
    return dict(case=case, inst=inst, W0=W0.to(inst.dtype), target=target, eps=eps, coef=coef)


def run(state):
    case, inst = state['case'], state['inst']
    if case['kind'] == 'wigner' and case['form'] == 'run':
        inst.Run()
        return [inst.W_end_complex, _run_observables(inst)]
    if case['kind'] == 'batch':
        state['W'].copy_(state['W0'])
        obs = inst.run(state['W'], case['steps'])
        return [state['W'], obs]
    if case['kind'] != 'control':
        W = state['W0'].clone()
        obs = inst.propagate(W, case['steps'])
        if case['kind'] == 'wigner' and case['form'] == 'gp':
            return [W, obs, inst.probability_square(case['steps'])]
        return [W, obs]
    W0 = state['W0'].clone().requires_grad_(True)
    eps = state['eps'].clone().requires_grad_(True)
    coef = state['coef'].clone().requires_grad_(True)
    WT = inst.propagate(W0, eps, coef, checkpoint=case['checkpoint'])
    loss = (WT.real.double() * state['target']).sum()
    loss.backward()
    return [WT.detach(), W0.grad, eps.grad, coef.grad]


def _run_observables(inst):
    return np.stack([inst.Norm_average, inst.X_average, inst.X2_average, inst.P_average, inst.P2_average,
                     inst.XP_average, inst.dPotentialdX_average, inst.PdPotentialdX_average,
                     inst.XdPotentialdX_average, inst.Hamiltonian_average, inst.negativeArea], 1)


# ---------------------------------------------------------------- what a pass cannot do without
def _fft_flops(points, n):
    return 5. * points * math.log2(n)


def work(case):
    """The state read and written once (and the outputs that a pass returns); the transforms of every step."""
    kind, steps = case['kind'], case['steps']
    if kind == 'batch':
        n_x, n_p, gamma = _batch_sizes(case)
        flops = sum(_fft_flops(float(a) * b, a) + _fft_flops(float(a) * b, b) * (4. if g else 1.)
                    for a, b, g in zip(n_x, n_p, gamma))            # two real sequences a transform
        return dict(bytes=8. * float(sum(int(a) * int(b) for a, b in zip(n_x, n_p))), flops=float(steps * flops))
    if kind in ('dirac2', 'dirac3'):
        grid = [case[k] for k in ('n_x', 'n_y', 'n_z') if k in case]
        pts = float(np.prod(grid))
        return dict(bytes=128. * pts, flops=steps * sum(8. * _fft_flops(pts, n) for n in grid))
    pts = float(case['n_x'] * case['n_p'])
    x, p = _fft_flops(pts, case['n_x']), _fft_flops(pts, case['n_p'])
    if kind == 'control':
        size = 16. if case['precision'] == 'c128' else 8.
        fwd = 2. * x + (8. if case['gamma'] else 2.) * p
        adj = 2. * x + (9. if case['gamma'] else 3.) * p
        return dict(bytes=3. * size * pts, flops=steps * (2. * fwd + adj))
    damped = case['gamma'] != 0.
    if damped and case['damping'] == 'ODM':
        step = 2. * x + 2. * p + 6. * x + 6. * p
    else:
        step = 2. * x + (8. if damped else 2.) * p
    if case['form'] == 'gp':
        step += 2. * p + 2. * x
    n = steps + (1 if case['form'] == 'run' else 0)
    return dict(bytes=32. * pts, flops=n * step)


# ---------------------------------------------------------------- the same in plain torch, 64 bits
def _f6(v):
    """A constant as the kernels of the complex128 classes see it: '%f' text."""
    return float('%f' % v)


def _lin(amp, n, dev):
    d = 2. * amp / n
    return torch.from_numpy(np.fft.fftshift(np.linspace(-amp, amp - d, n))).to(dev)


class _Wigner:
    """The Lie (or Strang / Gross-Pitaevskii) step of one complex128 Wigner instance."""

    def __init__(self, c, coef, dev):
        self.c, self.coef = c, coef
        nx, npp, amp = c['n_x'], c['n_p'], c['amp']
        self.dX, self.dP = 2. * amp / nx, 2. * amp / npp
        dth = 2. * np.pi / (2. * amp)
        dt, dx, dp, dk = _f6(c['dt']), _f6(self.dX), _f6(self.dP), _f6(dth)
        self.dt, self.hb, mass = dt, _f6(c['hbar']), _f6(c['mass'])
        self.X, self.P = _lin(amp, nx, dev)[None, :], _lin(amp, npp, dev)[:, None]
        self.Th, self.La = _lin(dth * npp / 2., npp, dev)[:, None], _lin(dth * nx / 2., nx, dev)[None, :]
        jx, jp = _index(nx, dev)[None, :], _index(npp, dev)[:, None]
        lam, p, self.x, self.th = dk * jx, dp * jp, dx * jx, dk * jp
        if c['form'] == 'gp':
            phase = dt * (0.5 * (p + self.hb * lam / 2.) ** 2 - 0.5 * (p - self.hb * lam / 2.) ** 2) / self.hb
        else:
            phase = dt * lam * p / mass
        self.K = torch.exp(-_f6(c['d_lambda']) * lam * lam) * torch.exp(-1j * phase)
        half = 0.5 if c['form'] == 'gp' else 1.
        xm, w2 = dx * (nx - 1.) / 2., (10. * dx) ** 2
        self.R = (torch.exp(-half * _f6(c['gamma']) * self.th ** 2 * dt) * (1. - torch.exp(-(self.x - xm) ** 2 / w2)) *
                  (1. - torch.exp(-(self.x + xm) ** 2 / w2)))
        self.half = half
        f = torch.abs(p) if c['damping'] != 'ODM' else p * p / torch.sqrt(p * p + 0.5)
        self.sfp = torch.where(p >= 0., f, -f)
        V0, dV = self.V(0., self.X), self.dV(0., self.X)
        one = torch.ones_like(self.X * self.P)
        self.tabs = [self.X * one, self.X ** 2 * one, self.P * one, self.P ** 2 * one, self.X * self.P, dV * one,
                     self.P * dV, self.X * dV * one, self.P ** 2 / (2. * c['mass']) + V0]

    def V(self, t, x):
        a, b, d = self.coef
        return a * x ** 4 + b * x ** 2 + d * x + (0.2 * x * math.sin(3. * t) if self.c['timedep'] else 0.)

    def dV(self, t, x):
        a, b, d = self.coef
        return 4. * a * x ** 3 + 2. * b * x + d + (0.2 * math.sin(3. * t) if self.c['timedep'] else 0.)

    def potential(self, W, t, gp=None):
        if self.c['form'] == 'kvn':
            phase = self.dt * (-self.dV(t, self.x) * self.th)
        else:
            u = self.hb * self.th / 2.
            phase = self.half * self.dt * (self.V(t, self.x - u) - self.V(t, self.x + u)) / self.hb
        f = self.R * torch.exp(-1j * phase)
        return torch.fft.ifft(torch.fft.fft(W, dim=0) * (f if gp is None else f * gp), dim=0)

    def kinetic(self, W):
        return torch.fft.ifft(torch.fft.fft(W, dim=1) * self.K, dim=1)

    def mean_field(self, W):
        px = W.sum(dim=0).real * self.dP
        shift = 0.5 * self.La * self.Th
        d = torch.fft.ifft(torch.fft.fft(px.to(W.dtype))[None, :] * (-2j * torch.sin(shift)), dim=1).real
        return torch.exp(-0.5j * self.dt * 0.5 * d / self.hb), float((px ** 2).sum() * self.dX)

    def damp(self, W):
        c = self.c
        if c['gamma'] == 0.:
            return W
        if c['damping'] == 'ODM':
            W = W + self.odm(W)
        else:
            g = c['dt'] * c['gamma']

            def D(B):
                return torch.fft.ifft(self.Th * torch.fft.fft(self.sfp * B, dim=0), dim=0)
            L = W + 2. / 3. * 1j * g * D(W)
            L = L + 1j * g * D(L)
            W = W + 2j * g * D(L)
        return W * (1. / (W.sum() * (self.dX * self.dP)))

    def odm(self, W):
        c, L, hb = self.c, 3., self.c['hbar']
        F = torch.fft.fft(W, dim=1)

        def g(q):
            q = torch.abs(q) + hb / (2. * L)
            return torch.sqrt(L * (q * q / torch.sqrt(q * q + 0.5)))
        pp, pm = self.P + 0.5 * hb * self.La, self.P - 0.5 * hb * self.La
        gp, gm = g(pp), g(pm)
        sp, sm = torch.sign(pp), torch.sign(pm)
        xp, xm = self.X + 0.5 * hb * self.Th, self.X - 0.5 * hb * self.Th

        def leg(t):
            return torch.fft.fft(torch.fft.ifft(F * t, dim=1), dim=0)
        S = leg(gp * gm) * (torch.cos(xp) * torch.cos(xm))
        S = S + leg(gp * gm * sm) * (1j * torch.cos(xm) * torch.sin(xp))
        S = S + leg(gp * sp * gm) * (-1j * torch.sin(xm) * torch.cos(xp))
        S = S + leg(gp * sp * gm * sm) * (torch.sin(xp) * torch.sin(xm)) + leg(-0.5 * (gp * gp + gm * gm))
        return torch.fft.ifft(S, dim=0) * (c['dt'] * 2. * c['gamma'])

    def sample(self, W):
        d = self.dX * self.dP
        out = [W.real.sum() * d] + [(W.real * t).sum() * d for t in self.tabs]
        return torch.stack(out + [torch.clamp(W.real, max=0.).sum() * d])

    def run(self, W):
        c = self.c
        W = W * (1. / (W.sum() * self.dX * self.dP))
        rows, psq = [self.sample(W)], []
        for n in range(c['steps'] + (1 if c['form'] == 'run' else 0)):
            t = n * c['dt']
            if c['form'] == 'gp':
                W = self.kinetic(self.potential(W, t, self.mean_field(W)[0]))
                gp, s = self.mean_field(W)
                psq.append(s)
                W = self.damp(self.potential(W, t, gp))
            else:
                W = self.damp(self.potential(self.kinetic(W), t))
            rows.append(self.sample(W))
        obs = torch.stack(rows).cpu().numpy()
        if c['form'] == 'run':
            return [W.cpu().numpy(), obs[:-1]]
        return [W, obs] + ([np.array(psq)] if c['form'] == 'gp' else [])


class _Control:
    """The polynomial-potential Lie step with exact constants (the batched and the adjoint form)."""

    def __init__(self, n_x, n_p, gamma, dt, dev):
        dx, dp, dk = 20. / n_x, 20. / n_p, 2. * math.pi / 20.
        jx, jp = _index(n_x, dev)[None, :], _index(n_p, dev)[:, None]
        self.x, self.p, lam, th = dx * jx, dp * jp, dk * jx, dk * jp
        self.K = torch.exp(-1j * dt * lam * self.p)
        xm, w2 = dx * (n_x - 1.) / 2., (10. * dx) ** 2
        self.R = (torch.exp(-gamma * th * th * dt) * (1. - torch.exp(-(self.x - xm) ** 2 / w2)) *
                  (1. - torch.exp(-(self.x + xm) ** 2 / w2)))
        self.u, self.th, self.dt, self.gamma, self.dxdp = th / 2., th, dt, gamma, dx * dp
        self.sfp = torch.where(self.p >= 0., torch.abs(self.p), -torch.abs(self.p))

    def D(self, W):
        return torch.fft.ifft(self.th * torch.fft.fft(self.sfp * W, dim=0), dim=0)

    def step(self, W, v4, v2, eps):
        x, u, g = self.x, self.u, self.dt * self.gamma
        dV = v4 * (-8. * x * u * (x * x + u * u)) + v2 * (-4. * x * u) + eps * (-2. * u)
        W = torch.fft.ifft(torch.fft.fft(W, dim=1) * self.K, dim=1)
        W = torch.fft.ifft(torch.fft.fft(W, dim=0) * (self.R * torch.exp(-1j * self.dt * dV)), dim=0)
        if self.gamma == 0.:
            return W
        L = W + 2. / 3. * 1j * g * self.D(W)
        L = L + 1j * g * self.D(L)
        W = W + 2j * g * self.D(L)
        return W / (W.sum() * self.dxdp)


def _exact_batch(case, seed, dev):
    states, rows = [], []
    for d, W in _batch_inputs(case, seed, dev):
        S = _Control(d['n_x'], d['n_p'], d['gamma'], d['dt'], dev)
        W = W.to(torch.complex128)
        W = W / (W.sum() * S.dxdp)
        v4, v2, x, p = d['v4'], d['v2'], S.x, S.p
        dV, V = (4. * v4 * x * x + 2. * v2) * x, (v4 * x * x + v2) * x * x
        one = torch.ones_like(x * p)
        tabs = [one, x * one, x * x * one, p * one, p * p * one, x * p, dV * one, p * dV, x * dV * one, 0.5 * p * p + V]
        obs = []
        for n in range(case['steps'] + 1):
            w = W.real
            obs.append(torch.stack([(w * t).sum() for t in tabs] + [torch.clamp(w, max=0.).sum()]) * S.dxdp)
            if n < case['steps']:
                W = S.step(W, v4, v2, 0.).real.to(torch.complex128)
        states.append(W.real.reshape(-1))
        rows.append(torch.stack(obs))
    return [torch.cat(states), torch.stack(rows).cpu().numpy()]


def _exact_control(case, seed, dev):
    W0, target, eps, coef = _control_inputs(case, seed, dev)
    S = _Control(case['n_x'], case['n_p'], case['gamma'], 0.005, dev)
    if case['precision'] == 'c64':
        W0 = W0.float()
    W0 = W0.to(torch.complex128).requires_grad_(True)
    eps, coef = eps.requires_grad_(True), coef.requires_grad_(True)
    W = W0
    for n in range(case['steps']):
        W = S.step(W, coef[0], coef[1], eps[n])
    (W.real * target).sum().backward()
    return [W.detach(), W0.grad, eps.grad, coef.grad]


def _exact_dirac(case, seed, dev):
    three = case['kind'] == 'dirac3'
    grid = [case[k] for k in ('n_z', 'n_y', 'n_x') if k in case]
    dims = tuple(range(1, len(grid) + 1))

    def axes(step):
        return [(step(n) * _index(n, dev)).reshape([-1 if i == j else 1 for j in range(len(grid))])
                for i, n in enumerate(grid)][::-1]
    dq = [24. / n for n in grid]
    x, p = axes(lambda n: _f6(24. / n)), axes(lambda n: _f6(2. * math.pi / 24.))
    m, c, dt = 1., C_LIGHT, _f6(case['dt'])
    mc2 = (0.5 if three else 1.) * m * c * c
    r2 = sum(q * q for q in x)
    A0, A1, A2 = -1. / torch.sqrt(r2 + 0.5), -0.5 * x[1] + 0. * r2, 0.5 * x[0] + 0. * r2
    F = torch.sqrt(mc2 ** 2 + (1. if three else c) * (A1 * A1 + A2 * A2))
    sF, cF, e = torch.sin(dt * F) / F, torch.cos(dt * F), torch.exp(-1j * dt * A0)
    px, py = p[0] + 0. * r2, p[1] + 0. * r2
    pz = p[2] + 0. * r2 if three else 0. * r2
    if three:
        E = c * torch.sqrt(px * px + py * py + pz * pz + (0.5 * m * c) ** 2)
        sK, cK, mk = c * torch.sin(E * dt) / E, torch.cos(E * dt), 0.5 * m * c
    else:
        pp = torch.sqrt(px * px + py * py + 1e-12)
        sK, cK, mk = torch.sin(c * dt * pp) / pp, torch.cos(c * dt * pp), 0.

    def mix_A(P):
        U11, U33, U31, U32 = cF - 1j * mc2 * sF, cF + 1j * mc2 * sF, 0., (A2 + 1j * A1) * sF
        U41 = (-A2 + 1j * A1) * sF
        return torch.stack([e * (U11 * P[0] + U32 * P[3]), e * (U11 * P[1] + U41 * P[2]),
                            e * (U32 * P[1] + U33 * P[2]), e * (U41 * P[0] + U33 * P[3])])

    def mix_K(Q):
        up, um = (py + 1j * px) * sK, (py - 1j * px) * sK
        z, d1, d3 = 1j * pz * sK, cK - 1j * mk * sK, cK + 1j * mk * sK
        return torch.stack([d1 * Q[0] - z * Q[2] - up * Q[3], d1 * Q[1] + um * Q[2] + z * Q[3],
                            -z * Q[0] - up * Q[1] + d3 * Q[2], um * Q[0] + z * Q[1] + d3 * Q[3]])
    B = None
    if not three:
        j = [_index(n, dev) + n // 2 for n in grid]
        b = [(1. - torch.exp(-k * k / (3. * n / 100.) ** 2)) * (1. - torch.exp(-(k - n + 1.) ** 2 / (3. * n / 100.) ** 2))
             for k, n in zip(j, grid)]
        B = b[0][:, None] * b[1][None, :]
    xe = [_lin(12., n, dev).reshape([-1 if i == j else 1 for j in range(len(grid))]) for i, n in enumerate(grid)][::-1]
    pe = [_lin(math.pi / d, n, dev).reshape([-1 if i == j else 1 for j in range(len(grid))])
          for i, (n, d) in enumerate(zip(grid, dq))][::-1]
    dV, dP = float(np.prod(dq)), float(np.prod([2. * math.pi / 24.] * len(grid)))

    def dens(P):
        return (P.real ** 2 + P.imag ** 2).sum(dim=0)
    P = _spinor(case, seed, dev)
    P = P / torch.sqrt(dens(P).sum() * dV)
    rows, kept, s1 = [], 1., None
    for n in range(case['steps']):
        rho = dens(P)
        a = [P[k] for k in range(4)]

        def re(u, v):
            return (u * v.conj()).real.sum()

        def im(u, v):
            return (u * v.conj()).imag.sum()
        pos = [(rho * q).sum() * dV for q in (x if three else xe)]
        al1 = 2. * (re(a[3], a[0]) + re(a[2], a[1])) * dV
        al2 = -2. * (im(a[0], a[3]) + im(a[2], a[1])) * dV
        a0 = (A0 * rho).sum() * dV
        Q = torch.fft.fftn(P, dim=dims)
        s = dens(Q).sum()
        if s1 is None or not three:
            s1 = s
        if not three:
            Q = Q / torch.sqrt(s * dP)
        sc = 1. / s1 if three else dP
        rq, q, kx = dens(Q), [Q[k] for k in range(4)], (p if three else pe)
        w = m * c * c * (rq - 2. * (Q[2:].real ** 2 + Q[2:].imag ** 2).sum(dim=0))
        w = w + 2. * c * kx[0] * ((q[3] * q[0].conj()).real + (q[2] * q[1].conj()).real)
        w = w + 2. * c * kx[1] * ((q[3] * q[0].conj()).imag + (q[1] * q[2].conj()).imag)
        if three:
            w = w + 2. * c * kx[2] * ((q[2] * q[0].conj()).real - (q[3] * q[1].conj()).real)
            al3 = 2. * (re(a[2], a[0]) - re(a[3], a[1])) * dV
        mom, en = [(rq * k).sum() * sc for k in kx], w.sum() * sc
        if three:
            rows.append(torch.stack(pos + [al1, al2, al3, a0] + mom + [en, rho.sum() * dV]))
        else:
            beta = (rho - 2. * (P[2:].real ** 2 + P[2:].imag ** 2).sum(dim=0)).sum() * dV
            rows.append(torch.stack(pos + [al1, al2, beta, en, a0] + mom + [torch.as_tensor(kept, device=dev).double()]))
        P = mix_A(torch.fft.ifftn(mix_K(Q), dim=dims))
        if not three:
            before = dens(P).sum()
            P = P * B
            after = dens(P).sum()
            kept = after / before
            P = P / torch.sqrt(after * dV)
    return [P, torch.stack(rows).cpu().numpy()]


def exact(case, seed):
    dev = DEV if torch.cuda.is_available() else 'cpu'
    if case['kind'] == 'wigner':
        coef, W0 = _wigner_inputs(case, seed, dev)
        return _Wigner(case, coef, dev).run(W0)
    if case['kind'] == 'batch':
        return _exact_batch(case, seed, dev)
    if case['kind'] == 'control':
        return _exact_control(case, seed, dev)
    return _exact_dirac(case, seed, dev)
