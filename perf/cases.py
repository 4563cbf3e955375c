"""Performance cases of the framework: what its users have it do.

Seven kinds of work, each through a public entry point of the package:

  vhs   batched single-species collision operator Q(f,f) (VHSOperator.eval),
        FP32 mode (Maxwellian split) and FP64 mode
  vss   mixture collision operator, every pair of every species
        (VSSOperator.eval_species), FP32 and FP64 mode
  dg    one explicit advection stage (DGOperator.advect, axnpby)
  imex  one penalised IMEX step of a Couette flow (DGFSABstd1D)
  fno_eval, fno_train   the learned surrogate of Q(f,f)

`listed` names fixed sizes; `draw` gives more cases of the same ranges.
"""
import math

import numpy as np
import torch

from dgfs1d_gpu_b200 import configs
from dgfs1d_gpu_b200.astd.solver import DGFSABstd1D
from dgfs1d_gpu_b200.basis import get_basis
from dgfs1d_gpu_b200.collision import VHSOperator, VSSOperator
from dgfs1d_gpu_b200.config import Config
from dgfs1d_gpu_b200.dg import DGOperator, axnpby
from dgfs1d_gpu_b200.sphericaldesign import get_sphquadrule
from dgfs1d_gpu_b200.surrogate import FNOSurrogate

DEV = 'cuda'
F64, F32, C128 = torch.float64, torch.float32, torch.complex128


def listed():
    return [
        # one point of a small grid, single-precision arrays: the reference's
        # per-point call (launches and latency count)
        dict(name='vhs32_n16_1pt', kind='vhs', precision='fp32', N=16, M=6,
             half=True, Nrho=8, points=1, L=5.0, omega=0.81, project=False,
             dtype='f32'),
        # a problem of the uneven multi-problem batch, with projection
        dict(name='vhs32_n24_24pt', kind='vhs', precision='fp32', N=24, M=12,
             half=False, Nrho=12, points=24, L=5.0, omega=0.81, project=True,
             dtype='f64'),
        # the Couette batch of bench.py (one stage: Ne=8, K=3)
        dict(name='vhs32_n32_24pt', kind='vhs', precision='fp32', N=32, M=12,
             half=False, Nrho=16, points=24, L=6.0, omega=0.81, project=False,
             dtype='f64'),
        # one stage of the Mach-1.5 normal shock (Ne=32, K=3, hard spheres)
        dict(name='vhs32_n48_96pt', kind='vhs', precision='fp32', N=48, M=32,
             half=False, Nrho=24, points=96, L=8.0, omega=0.5, project=True,
             dtype='f64'),
        # the Couette batch in the reference's precision
        dict(name='vhs64_n32_24pt', kind='vhs', precision='fp64', N=32, M=12,
             half=False, Nrho=16, points=24, L=6.0, omega=0.81, project=False,
             dtype='f64'),
        # the rule of the reference's Lax examples (N=48, half sphere)
        dict(name='vhs64_n48_24pt', kind='vhs', precision='fp64', N=48, M=6,
             half=True, Nrho=6, points=24, L=7.0, omega=0.77, project=False,
             dtype='f64'),
        # a mixture stage of the uneven batch (Ne=6, K=3, masses 1:2)
        dict(name='vss32_n24_18pt', kind='vss', precision='fp32', N=24, M=12,
             Mpre=192, Nrho=12, points=18, L=5.0, mass=2.0),
        # a mixture stage in the reference's precision (Ne=3, K=3)
        dict(name='vss64_n24_9pt', kind='vss', precision='fp64', N=24, M=6,
             Mpre=192, Nrho=12, points=9, L=5.0, mass=2.0),
        # advection stage of the normal-shock size, inlets at both ends
        dict(name='dg_n48_ne32', kind='dg', N=48, Ne=32, K=3, L=8.0,
             bc='inlet', dtype='f64'),
        # IMEX Couette step with the FP64 operator, diffuse walls
        dict(name='imex_n24_ne8', kind='imex', N=24, Ne=8, K=3, M=6, Nrho=6,
             L=6.0),
        # surrogate: one stage of the Couette batch
        dict(name='fno_eval_n32_24pt', kind='fno_eval', N=32, points=24,
             L=6.0),
        # surrogate: a segment of training steps, then the weights
        dict(name='fno_train_n32_b24', kind='fno_train', N=32, batch=24,
             steps=16, L=6.0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['vhs', 'vhs', 'vhs', 'vhs', 'vss', 'dg', 'imex',
                       'fno_eval', 'fno_train'])
    if kind == 'vhs':
        precision = rng.choice(['fp32', 'fp64'])
        N = rng.choice([8, 16, 24, 32, 48])
        half = rng.random() < 0.4
        M = 6 if half else rng.choice([6, 12, 32])
        Nrho = rng.randint(4, max(6, N // 2))
        points = _logint(rng, 1, 96)
        # no more than the largest listed case: 96 points, 24 x 16 terms, N=48
        # (FP64 takes at most three times as long as FP32)
        full = 96 * 24 * 16 * 48 ** 3
        Mu = M if half else M // 2
        while points > 1 and points * Nrho * Mu * N ** 3 * (
                1 if precision == 'fp32' else 4) > full:
            points //= 2
        return dict(kind=kind, precision=precision, N=N, M=M, half=half,
                    Nrho=Nrho, points=points, L=round(rng.uniform(5, 8), 2),
                    omega=rng.choice([0.5, 0.74, 0.81, 1.0]),
                    project=rng.random() < 0.5,
                    dtype=rng.choice(['f64', 'f64', 'f32']))
    if kind == 'vss':
        precision = rng.choice(['fp32', 'fp64'])
        N = rng.choice([8, 16, 24, 32])
        M = rng.choice([6, 12])
        Nrho = rng.randint(4, N // 2)
        points = _logint(rng, 1, 24)
        while points > 1 and points * Nrho * M * N ** 3 * (
                1 if precision == 'fp32' else 4) > 18 * 12 * 12 * 24 ** 3 * 4:
            points //= 2
        return dict(kind=kind, precision=precision, N=N, M=M,
                    Mpre=rng.choice([48, 192]), Nrho=Nrho, points=points,
                    L=round(rng.uniform(5, 7), 2),
                    mass=round(rng.uniform(1, 3), 2))
    if kind == 'dg':
        N = rng.choice([16, 24, 32, 48])
        return dict(kind=kind, N=N, Ne=_logint(rng, 2, 48),
                    K=rng.choice([2, 3, 5]), L=round(rng.uniform(5, 8), 2),
                    bc=rng.choice(['inlet', 'wall']),
                    dtype=rng.choice(['f64', 'f64', 'f32']))
    if kind == 'imex':
        return dict(kind=kind, N=rng.choice([16, 24, 32]),
                    Ne=rng.randint(2, 12), K=3, M=6,
                    Nrho=rng.randint(4, 8), L=round(rng.uniform(5, 7), 2))
    N = rng.choice([16, 32])
    if kind == 'fno_eval':
        return dict(kind=kind, N=N, points=_logint(rng, 1, 64),
                    L=round(rng.uniform(5, 7), 2))
    return dict(kind=kind, N=N, batch=rng.randint(2, 32),
                steps=rng.randint(4, 16), L=round(rng.uniform(5, 7), 2))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _grid(N, L):
    return np.linspace(-L + L / N, L - L / N, N)


def _vhs_params(c):
    N, M, L, omega = c['N'], c['M'], c['L'], c['omega']
    R = 2 * (L * 2.0 / (3.0 + math.sqrt(2.0)))
    z, w = np.polynomial.legendre.leggauss(c['Nrho'])
    if c['half']:
        sz = get_sphquadrule('symmetric', 'womersley', npts=2 * M).pts[:M]
        sw, sf = 2 * math.pi / M, 2.0
    else:
        sz = get_sphquadrule('symmetric', 'womersley', npts=M).pts
        sw, sf = 4 * math.pi / M, 1.0
    prefac = 10.0 / (2.0 ** (3 - omega) * math.gamma(2.5 - omega) * math.pi)
    return dict(N=N, L=L, qz=(R / 2) * (1 + z), qw=(R / 2) * w, sz=sz, sw=sw,
                sphere_factor=sf, gamma=2.0 * (1 - omega), prefac=prefac,
                cw=(2.0 * L / N) ** 3, c0=_grid(N, L))


def _maxwellians(c0, slots, seed, noise=0.01, mass=1.0, T0=1.0, dens=1.0):
    """Perturbed Maxwellians with a bulk velocity and temperature of their
    own, as the states of a slab between walls or across a shock are."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + 17)
    n = len(c0) ** 3
    c = torch.tensor(c0, device=DEV, dtype=F64)
    r = torch.rand((3, slots, 1, 1, 1), generator=g, device=DEV, dtype=F64)
    uy = 0.2 * r[0] - 0.1
    T = T0 * (0.95 + 0.1 * r[1])
    rho = dens * (0.9 + 0.2 * r[2])
    d2 = (c.view(1, -1, 1, 1) ** 2 + (c.view(1, 1, -1, 1) - uy) ** 2
          + c.view(1, 1, 1, -1) ** 2)
    f = rho * (mass / (math.pi * T)) ** 1.5 * torch.exp(-mass * d2 / T)
    f = f.reshape(slots, n)
    w = torch.rand((slots, n), generator=g, device=DEV, dtype=F64)
    return f * (1 + noise * (2 * w - 1))


def _dtype(c):
    return F32 if c.get('dtype') == 'f32' else F64


def _vss_params(c):
    N, M, L = c['N'], c['M'], c['L']
    m = [1.0, c['mass']]
    mr = max(m)
    S = min(L * 2. / (max(4. * mr / (1. + mr), 2.) + math.sqrt(1. + mr) + 1.),
            L * 2. / (max(4. / (1. + mr), 2.) + math.sqrt(1. + 1. / mr) + 1.))
    z, w = np.polynomial.legendre.leggauss(c['Nrho'])
    sz = get_sphquadrule('symmetric', 'womersley', npts=M).pts
    szpre = get_sphquadrule('symmetric', 'womersley', npts=c['Mpre']).pts
    one = np.ones((2, 2))
    return dict(N=N, L=L, qz=S * (1 + z), qw=S * w, sz=sz, sw=4 * np.pi / M,
                szpre=szpre, masses=m, gamma=0.38 * one, eta=0.4 * one,
                prefac=0.1 * one)


def _vss_inputs(c, seed):
    c0 = _grid(c['N'], c['L'])
    return [_maxwellians(c0, c['points'], 2 * seed + s, noise=0.02,
                         mass=m, T0=T, dens=0.5)
            for s, (m, T) in enumerate(((1.0, 1.0), (c['mass'], 1.2)))]


def _dg_inputs(c, seed):
    c0 = _grid(c['N'], c['L'])
    u = _maxwellians(c0, c['K'] * c['Ne'], seed)
    u = u.reshape(c['K'], c['Ne'], -1).to(_dtype(c)).contiguous()
    x = np.linspace(-0.5, 0.5, c['Ne'] + 1)
    f0 = []
    for uy, T in ((-0.1, 1.0), (0.1, 1.05)):
        e = [np.exp(-(c0 - s) ** 2 / T) for s in (0.0, uy, 0.0)]
        m = (e[0][:, None, None] * e[1][None, :, None] * e[2][None, None, :])
        f0.append((m / (math.pi * T) ** 1.5).ravel())
    return c0, u, 2.0 / np.diff(x), f0


def _imex_cfg(c):
    return Config(configs.couette_astd_ini(
        scheme='boltz-ars-111', penalty='boltz-bgk-direct-gll', dt=1e-3,
        nsteps=1, Ne=c['Ne'], K=c['K'], Nv=c['N'], Nrho=c['Nrho'], M=c['M'],
        dev=c['L'], sphere='half', precision_mode='fp64', ic='maxwellian'))


def _fno_weights(N, seed):
    """Weights with the spreads a trained network has, from the seed."""
    from dgfs1d_gpu_b200.surrogate import MODES, init_params
    return init_params(MODES[N], seed=seed % 1000)


def prepare(case, seed):
    c = case
    kind = c['kind']
    if kind == 'vhs':
        op = VHSOperator(**_vhs_params(c), precision=c['precision'],
                         max_evals=c['points'])
        if c['project']:
            op.set_projection(True)
        f = _maxwellians(_grid(c['N'], c['L']), c['points'], seed)
        f = f.to(_dtype(c)).contiguous()
        return dict(kind=kind, op=op, f=f, Q=torch.zeros_like(f))
    if kind == 'vss':
        op = VSSOperator(**_vss_params(c), max_evals=c['points'],
                         precision=c['precision'])
        fs = _vss_inputs(c, seed)
        return dict(kind=kind, op=op, fs=fs, Q=[torch.zeros_like(x) for x in fs])
    if kind == 'dg':
        c0, u, invjac, f0 = _dg_inputs(c, seed)
        basis = get_basis(Config(
            f"[basis]\nkind = nodal-sem-gll\nK = {c['K']}\nNqr = {c['K']}\n"))
        bc = 'dgfs-inlet' if c['bc'] == 'inlet' else 'dgfs-wall-diffuse'
        dg = DGOperator(basis, invjac, c0, (2 * c['L'] / c['N']) ** 3,
                        [(bc, f0[0], 0.0), (bc, f0[1], 0.0)])
        return dict(kind=kind, dg=dg, u=u, ux=torch.empty_like(u),
                    r=torch.empty_like(u), dt=1e-4)
    if kind == 'imex':
        s = DGFSABstd1D(_imex_cfg(c))
        u = _maxwellians(s.vm.c0(), c['K'] * c['Ne'], seed)
        return dict(kind=kind, solver=s, u=u.reshape(s.u.shape).contiguous())
    if kind == 'fno_eval':
        net = FNOSurrogate(c['N'], c['L'], q_scale=1.0,
                           max_batch=min(32, c['points']),
                           params=_fno_weights(c['N'], seed))
        f = _maxwellians(_grid(c['N'], c['L']), c['points'], seed)
        return dict(kind=kind, net=net, f=f, Q=torch.zeros_like(f))
    if kind == 'fno_train':
        N, B = c['N'], c['batch']
        f = _maxwellians(_grid(N, c['L']), B * c['steps'], seed)
        op = VHSOperator(**_vhs_params(dict(
            N=N, M=6, half=True, Nrho=N // 4, L=c['L'], omega=0.81)),
            precision='fp32', max_evals=B)
        Q = torch.zeros_like(f)
        op.eval(f, Q)
        # the output scale that makes the network's target O(1): Q is about
        # linear in f - M, and f - M is 1% uniform noise times f
        scale = float(Q.square().mean().sqrt() / f.square().mean().sqrt())
        net = FNOSurrogate(N, c['L'], q_scale=scale * math.sqrt(3.0) / 0.01,
                           max_batch=B, params=_fno_weights(N, seed))
        return dict(kind=kind, net=net, B=B, lr=1e-4,
                    batches=[(f[i:i + B], Q[i:i + B])
                             for i in range(0, B * c['steps'], B)])
    raise ValueError(kind)


def run(state):
    s = state
    kind = s['kind']
    if kind == 'vhs':
        s['Q'].zero_()
        s['op'].eval(s['f'], s['Q'])
        return s['Q']
    if kind == 'vss':
        for p in range(2):
            s['Q'][p].zero_()
            s['op'].eval_species(p, s['fs'], s['Q'][p])
        return s['Q']
    if kind == 'dg':
        s['dg'].advect(s['u'], s['ux'])
        axnpby(s['r'], 0.0, 1.0, s['u'], s['dt'], s['ux'])
        return s['ux'], s['r']
    if kind == 'imex':
        sol = s['solver']
        u = s['u'].clone()
        sol.odes.integrate(0.0, sol.dt, 0, u)
        return u
    if kind == 'fno_eval':
        s['Q'].zero_()
        s['net'].eval(s['f'], s['Q'])
        return s['Q']
    for f, Q in s['batches']:
        s['net'].train_step(f, Q, lr=s['lr'])
    return s['net'].params(), s['net'].last_loss(s['B'])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _fft(n):
    return 5.0 * n * math.log2(n)


def work(case):
    c = case
    kind = c['kind']
    n = c['N'] ** 3
    if kind in ('vhs', 'imex'):
        pts = c['points'] if kind == 'vhs' else c['K'] * c['Ne']
        half = c.get('half', True)
        Mu = c['M'] if half else c['M'] // 2   # antipodal pairs count once
        T = c['Nrho'] * Mu
        # a complex inverse transform per term (real and imaginary part both
        # used), a forward and a spectral product per radial point (two real
        # fields per transform), two more for f and the output
        flops = pts * ((T + c['Nrho'] / 2 + 2) * _fft(n) + T * 10 * n)
        it = 4 if c.get('dtype') == 'f32' else 8
        return dict(bytes=3.0 * pts * n * it, flops=flops)
    if kind == 'vss':
        T = c['Nrho'] * c['M']
        # per pair and term: two real fields by one complex inverse transform,
        # one real forward transform (two per complex one)
        flops = c['points'] * 4 * (T * (1.5 * _fft(n) + 14 * n) + 2 * _fft(n))
        return dict(bytes=c['points'] * n * 8 * 2 * 3.0
                    + 4.0 * T * n * (8 if c['precision'] == 'fp32' else 16),
                    flops=flops)
    if kind == 'dg':
        it = 4 if c.get('dtype') == 'f32' else 8
        m = c['K'] * c['Ne'] * n
        return dict(bytes=3.0 * m * it, flops=m * (2.0 * c['K'] + 12))
    K = {16: 8, 32: 12}[c['N']]
    B = c['points'] if kind == 'fno_eval' else c['batch']
    R, nm = B * n, K ** 3
    spec = 32 * B * (n * 2.5 * math.log2(c['N']) * (1 + K / c['N']
                                                     + (K / c['N']) ** 2))
    fwd = 4 * (2 * spec + 8.0 * B * nm * 1024 + 2.0 * R * 1024) \
        + 2.0 * R * 32 * 128
    w = 2.0 * nm * 1024
    if kind == 'fno_eval':
        return dict(bytes=R * 8 * 3.0 + 4 * w * 2, flops=fwd)
    # the batches, and the weights and both Adam moments in and out once
    return dict(bytes=c['steps'] * R * 8 * 2.0 + 4 * w * 4 * 6,
                flops=c['steps'] * 3 * fwd)


def tolerance(case):
    """About four times the error against `exact` that the ranges show."""
    kind = case['kind']
    if kind in ('vhs', 'vss') and case['precision'] == 'fp64':
        if case.get('dtype') == 'f32':          # results rounded to 32 bits
            return {'rel': 2e-7, 'max': 2e-6}
        return {'rel': 1e-12, 'max': 2e-11} if kind == 'vhs' \
            else {'rel': 1e-13, 'max': 2e-12}
    if kind == 'vhs':
        return {'rel': 2e-6, 'max': 3e-5}
    if kind == 'vss':
        return {'rel': 1e-7, 'max': 2e-6}
    if kind == 'dg':
        return {'rel': 2e-14, 'max': 2e-12} if case['dtype'] == 'f64' \
            else {'rel': 3e-7, 'max': 3e-6}
    if kind == 'imex':
        return {'rel': 2e-15, 'max': 2e-14}
    if kind == 'fno_train':      # FP32 weights after a few small steps
        return {'rel': 1e-3, 'max': 0.2}
    # BF16 activations and weights
    return {'rel': 2e-2, 'max': 0.4}


# ---------------------------------------------------------------------------
# the same values in plain 64-bit torch
# ---------------------------------------------------------------------------
def _lvec(N):
    return torch.fft.fftfreq(N, 1.0 / N, device=DEV, dtype=F64)


def _phases(l, k):
    """exp(i k.l) on the N^3 spectral grid for each row of k."""
    e = [torch.exp(1j * k[:, a:a + 1] * l) for a in range(3)]
    return e[0][:, :, None, None] * e[1][:, None, :, None] * e[2][:, None, None, :]


def _exact_vhs(p, f, project=False):
    N, L = p['N'], p['L']
    l = _lvec(N)
    d = math.pi / L
    cs = torch.sqrt(l.view(-1, 1, 1) ** 2 + l.view(1, -1, 1) ** 2
                    + l.view(1, 1, -1) ** 2)

    def sinc(s):
        return torch.sin(s + 1e-15) / (s + 1e-15)
    sz = torch.tensor(np.array(p['sz']), device=DEV, dtype=F64)
    out = torch.empty_like(f)
    step = max(1, (1 << 27) // (N ** 3 * 16 * 4 * len(sz)))
    b1s, b2 = [], 0
    for qz, qw in zip(p['qz'], p['qw']):
        b1s.append(p['sphere_factor'] * qw * p['sw'] / N ** 3
                   * qz ** (p['gamma'] + 2) * 4 * math.pi * sinc(d * qz / 2 * cs))
        b2 = b2 + qw * qz ** (p['gamma'] + 2) * 16 * math.pi ** 2 \
            * sinc(d * qz * cs)
    for i in range(0, len(f), step):
        fb = f[i:i + step].reshape(-1, N, N, N)
        F = torch.fft.fftn(fb.to(C128), dim=(1, 2, 3)) / N ** 3
        G = torch.zeros_like(F)
        for b1, qz in zip(b1s, p['qz']):
            E = _phases(l, d * qz / 2 * sz)
            S = 0
            for e in E:
                t3 = torch.fft.ifftn(e.real * F, dim=(1, 2, 3), norm='forward')
                t4 = torch.fft.ifftn(e.imag * F, dim=(1, 2, 3), norm='forward')
                S = S + t3 * t3 + t4 * t4
            G += b1 * torch.fft.fftn(S, dim=(1, 2, 3))
        g = torch.fft.ifftn(G, dim=(1, 2, 3), norm='forward').real
        lo = torch.fft.ifftn(b2 * F, dim=(1, 2, 3), norm='forward').real
        out[i:i + step] = (p['prefac'] * (g - fb * lo)).reshape(len(fb), -1)
    if project:
        c = torch.tensor(p['c0'], device=DEV, dtype=F64)
        x, y, z = torch.meshgrid(c, c, c, indexing='ij')
        phi = torch.stack([torch.ones_like(x), x, y, z, x * x + y * y + z * z])
        phi = phi.reshape(5, -1)
        lam = torch.linalg.solve(phi @ phi.T, phi @ out.T)
        out = out - lam.T @ phi
    return out


def _exact_vss(c, p, fs):
    N, n = c['N'], c['N'] ** 3
    l, d = _lvec(N), math.pi / c['L']
    sz = torch.tensor(np.array(p['sz']), device=DEV, dtype=F64)
    spre = torch.tensor(np.array(p['szpre']), device=DEV, dtype=F64)
    F = [torch.fft.fftn(f.reshape(-1, N, N, N).to(C128), dim=(1, 2, 3)) / n
         for f in fs]
    m = p['masses']
    out = []
    B = (1 + sz @ spre.T) ** p['eta'][0, 0]
    for a in range(2):
        Q = 0
        for b in range(2):
            r = m[b] / (m[a] + m[b])
            G = torch.zeros_like(F[a])
            cl = 0
            for qz, qw in zip(p['qz'], p['qw']):
                fb = 4 * math.pi / c['Mpre'] * qz ** (p['gamma'][0, 0] + 2)
                eb = _phases(l, -r * d * qz * spre).reshape(c['Mpre'], n)
                bt = (fb * (B.to(C128) @ eb)).reshape(-1, N, N, N)
                eb = _phases(l, -d * qz * spre).reshape(c['Mpre'], n)
                cl = cl + qw * p['sw'] * fb * (B.sum(0).to(C128) @ eb)
                Eu = _phases(l, r * d * qz * sz)
                Ev = _phases(l, -(1 - r) * d * qz * sz)
                for q in range(len(sz)):
                    u = torch.fft.ifftn(Eu[q] * F[a], dim=(1, 2, 3), norm='forward')
                    v = torch.fft.ifftn(Ev[q] * F[b], dim=(1, 2, 3), norm='forward')
                    G += (qw * p['sw'] / n) * bt[q] * torch.fft.fftn(
                        u * v, dim=(1, 2, 3))
            g = torch.fft.ifftn(G, dim=(1, 2, 3), norm='forward').real
            lo = torch.fft.ifftn(cl.reshape(N, N, N) * F[b], dim=(1, 2, 3),
                                 norm='forward').real
            Q = Q + p['prefac'][a, b] * (g.reshape(len(g), -1)
                                         - fs[a] * lo.reshape(len(g), -1))
        out.append(Q)
    return out


def _gll(K):
    P = np.polynomial.legendre.Legendre.basis(K - 1)
    z = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]])
    w = 2.0 / (K * (K - 1) * P(z) ** 2)
    D = np.zeros((K, K))
    for i in range(K):
        for j in range(K):
            if i != j:
                D[i, j] = P(z[i]) / P(z[j]) / (z[i] - z[j])
        D[i, i] = -D[i].sum()
    return z, w, D


def _exact_advect(u, c0, cw, invjac, f0, walls):
    """-c_x du/dx with upwind faces on (K, Ne, Nv); f0: wall or inlet
    Maxwellians entering at the two ends."""
    K, Ne, Nv = u.shape
    N = len(c0)
    _, w, D = _gll(K)
    D = torch.tensor(D, device=DEV, dtype=F64)
    cx = torch.tensor(c0, device=DEV, dtype=F64).repeat_interleave(N * N)
    uL = torch.empty((Ne + 1, Nv), device=DEV, dtype=F64)
    uR = torch.empty_like(uL)
    uL[1:], uR[:-1] = u[-1], u[0]
    for side, nrm, tr in ((0, -1.0, u[0, 0]), (1, 1.0, u[-1, -1])):
        fac = cx * nrm
        g = torch.tensor(f0[side], device=DEV, dtype=F64)
        if walls:
            g = g * -((fac * tr)[fac >= 0].sum() / (fac * g)[fac < 0].sum())
        g = torch.where(fac < 0, g, tr)
        if side == 0:
            uL[0] = g
        else:
            uR[-1] = g
    ac, hc = 0.5 * cx.abs(), 0.5 * cx
    jL = ac * (uL - uR) + hc * (uR - uL)
    jR = ac * (uL - uR) + hc * (uL - uR)
    ux = torch.einsum('km,mev->kev', D, u) * -cx
    ux[-1] -= jL[1:] / w[-1]
    ux[0] += jR[:-1] / w[0]
    return ux * torch.tensor(np.ravel(invjac), device=DEV, dtype=F64).view(1, -1, 1)


def _exact_imex(c, seed):
    cfg = _imex_cfg(c)
    K, Ne, N = c['K'], c['Ne'], c['N']
    R0 = 8.3144598
    T0, rho0, m0, H0 = (cfg.lookupfloat('non-dim', 'T0'),
                        cfg.lookupfloat('non-dim', 'rho0'),
                        cfg.lookupfloat('non-dim', 'molarMass0'),
                        cfg.lookupfloat('mesh', 'H0'))
    L, omega = float(c['L']), 0.81
    c0 = _grid(N, L)
    cw = (2 * L / N) ** 3
    u0 = math.sqrt(2 * R0 / m0 * T0)
    n0 = rho0 / m0 * 6.0221409e+23
    dRef = cfg.lookupfloat('scattering-model', 'dRef')
    invKn = H0 * math.sqrt(2.0) * math.pi * n0 * dRef * dRef
    den = 2.0 ** (3 - omega) * math.gamma(2.5 - omega) * math.pi
    p = _vhs_params(dict(N=N, M=c['M'], half=True, Nrho=c['Nrho'], L=L,
                         omega=omega))
    p['prefac'] = invKn / den
    nup, dt = 100 * invKn / den, 1e-3
    f = _maxwellians(c0, K * Ne, seed)
    cc = torch.tensor(c0, device=DEV, dtype=F64)
    x, y, z = (a.reshape(-1) for a in torch.meshgrid(cc, cc, cc, indexing='ij'))
    phi = torch.stack([torch.ones_like(x), x, y, z, x * x + y * y + z * z]) * cw

    def gauss(U):
        u = U[:, 1:4] / U[:, 0:1]
        T = (U[:, 4:5] / U[:, 0:1] - (u * u).sum(1, keepdim=True)) / 1.5
        d2 = (x - u[:, 0:1]) ** 2 + (y - u[:, 1:2]) ** 2 + (z - u[:, 2:3]) ** 2
        return (U[:, 0:1] / (math.pi * T) ** 1.5 * torch.exp(-d2 / T),
                nup * U[:, 0:1] * T ** (1 - omega))
    U0 = f @ phi.T
    M0, nu0 = gauss(U0)
    xm = np.linspace(0.0, 1.0, Ne + 1)
    f0 = []
    for s in ('soln-bcs-xlo', 'soln-bcs-xhi'):
        uy, T = cfg.lookupfloat(s, 'uy') / u0, cfg.lookupfloat(s, 'T') / T0
        f0.append((torch.exp(-(x ** 2 + (y - uy) ** 2 + z ** 2) / T)
                   / (math.pi * T) ** 1.5).cpu().numpy())
    ad = _exact_advect(f.reshape(K, Ne, -1), c0, cw, 2.0 / np.diff(xm), f0,
                       True).reshape(f.shape)
    U1 = U0 + dt * (ad @ phi.T)
    rhs = f + dt * (ad + _exact_vhs(p, f) - nu0 * (M0 - f))
    M1, nu1 = gauss(U1)
    return ((rhs + dt * nu1 * M1) / (1 + dt * nu1)).reshape(K, Ne, -1)


def _exact_fno(c, f, w):
    """The network in 64 bits (the framework rounds activations to BF16)."""
    N, L, n = c['N'], c['L'], c['N'] ** 3
    K = {16: 8, 32: 12}[N]
    nm = K ** 3
    w = torch.tensor(w, device=DEV).to(torch.bfloat16).to(F64)
    o = 0

    def take(*shape):
        nonlocal o
        k = int(np.prod(shape))
        o += k
        return w[o - k:o].reshape(shape)
    P, pb = take(4, 32), take(32)
    layers = [(take(nm, 32, 32, 2), take(32, 32), take(32)) for _ in range(4)]
    Q1, q1, q2, q2b = take(32, 128), take(128), take(128), take(1)
    cc = torch.tensor(_grid(N, L), device=DEV, dtype=F64)
    cw = (2.0 * L / N) ** 3
    x, y, z = (a.reshape(-1) for a in torch.meshgrid(cc, cc, cc, indexing='ij'))
    cv = torch.stack([x, y, z])
    c2 = (cv ** 2).sum(0)
    ks = torch.tensor([k if k < K // 2 else k - K for k in range(K)],
                      device=DEV, dtype=F64)
    Ft = torch.exp(-2j * math.pi / N * ks[:, None]
                   * torch.arange(N, device=DEV, dtype=F64)[None])
    Gt = Ft.conj().T.contiguous() / N

    def gelu(v):
        return torch.nn.functional.gelu(v, approximate='tanh')

    phi = torch.cat([torch.ones_like(x)[None], cv, c2[None]])
    Gram = phi @ phi.T
    out = torch.empty_like(f)
    for i in range(len(f)):
        fi = f[i]
        rho = fi.sum() * cw
        u = (cv @ fi) * cw / rho
        T = (2.0 / 3.0) * ((fi @ c2) * cw / rho - (u * u).sum())
        r2 = ((cv - u[:, None]) ** 2).sum(0) / T
        g = (fi - rho / (math.pi * T) ** 1.5 * torch.exp(-r2)) / rho
        sig = g.square().mean().sqrt()
        g = g / sig
        v = torch.stack([fi / rho, g, g * r2.sqrt(), g * r2], -1) @ P + pb
        for k, (W, D, d) in enumerate(layers):
            t = v.reshape(N, N, N, 32).to(C128)
            t = torch.einsum('kx,xyzc->kyzc', Ft, t)
            t = torch.einsum('ky,xyzc->xkzc', Ft, t)
            t = torch.einsum('kz,xyzc->xykc', Ft, t)
            t = torch.einsum('mi,mio->mo', t.reshape(nm, 32),
                             torch.complex(W[..., 0], W[..., 1]))
            t = t.reshape(K, K, K, 32)
            t = torch.einsum('xk,kyzc->xyzc', Gt, t)
            t = torch.einsum('yk,xkzc->xyzc', Gt, t)
            t = torch.einsum('zk,xykc->xyzc', Gt, t)
            v2 = v @ D + d + t.reshape(n, 32).real
            v = gelu(v2) if k < 3 else v2
        q = rho * rho * sig * (gelu(v @ Q1 + q1) @ q2 + q2b)
        out[i] = q - torch.linalg.solve(Gram, phi @ q) @ phi
    return out


def exact(case, seed):
    c = case
    kind = c['kind']
    if kind == 'vhs':
        f = _maxwellians(_grid(c['N'], c['L']), c['points'], seed)
        return _exact_vhs(_vhs_params(c), f.to(_dtype(c)).to(F64), c['project'])
    if kind == 'vss':
        return _exact_vss(c, _vss_params(c), _vss_inputs(c, seed))
    if kind == 'dg':
        c0, u, invjac, f0 = _dg_inputs(c, seed)
        u = u.to(F64)
        ux = _exact_advect(u, c0, (2 * c['L'] / c['N']) ** 3, invjac, f0,
                           c['bc'] == 'wall')
        return ux, u + 1e-4 * ux
    if kind == 'imex':
        return _exact_imex(c, seed)
    if kind == 'fno_eval':
        f = _maxwellians(_grid(c['N'], c['L']), c['points'], seed)
        return _exact_fno(c, f, _fno_weights(c['N'], seed))
    return None     # a training segment in 64 bits takes over 20 seconds
