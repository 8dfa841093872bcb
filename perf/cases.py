"""The work a user of this framework has it do, as timed cases.

Every case goes through the public entry points (scattering models, systems,
steppers, the hybrid collider).  ``listed`` gives fixed sizes, ``draw`` more
of the same ranges; ``prepare`` builds what a program holds before the call,
``run`` is one pass, ``work`` the bytes and operations of a pass, and
``exact`` the same outputs in 64-bit torch, written independently of the
package.

Kinds
  collide   Q of one gas on one velocity grid (``sm.collide``; ``point``: the
            per-point call ``sm.fs``)
  pair      two species grids (24^3 and 32^3) in one launch (``VHSCollider``)
  mixture   Q_p of a gas mixture (``vss-gll``)
  advect    one FR stage of the second RK stage (``advect_combine``)
  relax     one step of the relaxation system ('adgfs')
  moments   macroscopic fields of a state bank (the moment writer's call)
  hybrid    the surrogate / spectral collision call
  step      one SSP-RK2 step of the 'dgfs' system
"""
import math
from fractions import Fraction

import numpy as np
import torch

T0, H0, RHO0, MOLAR0 = 273.0, 1e-3, 0.00011140244750324529, 39.96e-3
R0, NA = 8.3144598, 6.0221409e+23
N0 = RHO0 / MOLAR0 * NA
U0 = math.sqrt(2 * R0 / MOLAR0 * T0)
DREF, OMEGA, MUREF = 4.17e-10, 0.81, 2.117e-5
SCHEMES = ('adgfs-ars-111', 'adgfs-ars-222', 'adgfs-ars-443', 'adgfs-bdf-2')
MODELS = ('bgk-direct-gll', 'esbgk-direct-gll', 'shakov-direct-gll')


def listed():
    return [
        # the reference's per-point call: one distribution, latency bound
        dict(name='q_point', kind='collide', Nv=24, Nrho=12, M=12, dev=6, ndof=1, fp64=False,
             family='grad', point=True),
        # a short, ragged list of cells (what a hybrid solve sends to the spectral operator)
        dict(name='q_cells', kind='collide', Nv=24, Nrho=12, M=12, dev=6, ndof=97, fp64=False,
             family='mixed', point=False),
        # every DOF of the 16x8 P3 Couette channel
        dict(name='q_couette', kind='collide', Nv=24, Nrho=12, M=12, dev=6, ndof=2048, fp64=False,
             family='grad', point=False),
        # two species on grids of their own, batched in one launch
        dict(name='q_two_grids', kind='pair', Nrho=16, M=12, dev=6, n24=1500, n32=501),
        # the small double-precision configuration: 4x4 P2 elements, hard spheres
        dict(name='q_fp64', kind='collide', Nv=16, Nrho=8, M=6, dev=5, ndof=144, fp64=True,
             family='mixed', point=False),
        # binary argon-krypton mixture
        dict(name='mixture', kind='mixture', Nv=24, Nrho=12, M=12, Mpre=12, dev=6, ndof=370,
             fp64=False, heavy=83.798e-3),
        # FR advection of a 3-D lid-driven cavity, P2 hexes, diffuse walls
        dict(name='fr_cavity', kind='advect', ndims=3, nx=6, ny=5, nz=7, order=2, Nv=24, dev=6,
             fp64=False),
        # BGK channel: ARS-222 step at the Couette size
        dict(name='relax_ars', kind='relax', nx=16, ny=8, order=3, Nv=24, dev=6, fp64=False,
             scheme='adgfs-ars-222', model='bgk-direct-gll'),
        # Shakov channel with backward differences on an odd mesh
        dict(name='relax_bdf', kind='relax', nx=7, ny=5, order=2, Nv=24, dev=6, fp64=False,
             scheme='adgfs-bdf-2', model='shakov-direct-gll'),
        # the moment writer on a cavity-sized state
        dict(name='moments', kind='moments', Nv=24, dev=6, ndof=5670, fp64=False),
        # learned surrogate on near-equilibrium cells, spectral operator on the rest
        dict(name='hybrid', kind='hybrid', Nv=24, Nrho=12, M=12, dev=6, ndof=3001, far=0.02,
             modes=512, width=1024, center=False),
        # one whole SSP-RK2 step of the Couette channel
        dict(name='step_couette', kind='step', nx=16, ny=8, order=3, Nv=24, Nrho=12, M=12, dev=6,
             fp64=False),
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(['collide', 'collide', 'collide', 'pair', 'mixture', 'advect', 'relax',
                       'relax', 'moments', 'hybrid', 'step'])
    if kind == 'collide':
        Nv = rng.choice([16, 24, 24, 24, 32])
        fp64 = Nv == 16 and rng.random() < 0.6
        top = {16: 2048, 24: 2048, 32: 600}[Nv] if not fp64 else 400
        return dict(kind=kind, Nv=Nv, Nrho=rng.choice([Nv // 2 - 3, Nv // 2]) if Nv < 32 else 16,
                    M=6 if Nv == 16 else rng.choice([6, 12, 12, 12]), dev=5 if Nv == 16 else 6,
                    ndof=_logint(rng, 1, top), fp64=fp64,
                    family=rng.choice(['grad', 'mixed']), point=False)
    if kind == 'pair':
        return dict(kind=kind, Nrho=rng.choice([12, 16]), M=12, dev=6, n24=_logint(rng, 8, 1500),
                    n32=_logint(rng, 8, 500))
    if kind == 'mixture':
        Nv = rng.choice([16, 24, 24])
        fp64 = Nv == 16 and rng.random() < 0.4
        return dict(kind=kind, Nv=Nv, Nrho=Nv // 2 - rng.choice([0, 1, 4]), M=rng.choice([6, 12]),
                    Mpre=12, dev=5 if Nv == 16 else 6, ndof=_logint(rng, 1, 100 if fp64 else 370),
                    fp64=fp64, heavy=rng.choice([83.798e-3, 20.18e-3]))
    if kind == 'advect':
        nd = rng.choice([2, 3])
        fp64 = rng.random() < 0.25
        Nv = 16 if fp64 else rng.choice([16, 24])
        order = rng.choice([1, 2, 3]) if nd == 2 else rng.choice([1, 2])
        nx, ny, nz = rng.randint(2, 6 if nd == 3 else 16), rng.randint(2, 5 if nd == 3 else 8), \
            rng.randint(2, 7) if nd == 3 else 1
        return dict(kind=kind, ndims=nd, nx=nx, ny=ny, nz=nz, order=order, Nv=Nv,
                    dev=5 if Nv == 16 else 6, fp64=fp64)
    if kind == 'relax':
        Nv = rng.choice([16, 24])
        return dict(kind=kind, nx=rng.randint(2, 14), ny=rng.randint(2, 8), order=rng.choice([2, 3]),
                    Nv=Nv, dev=5 if Nv == 16 else 6, fp64=Nv == 16 and rng.random() < 0.4,
                    scheme=rng.choice(SCHEMES), model=rng.choice(MODELS))
    if kind == 'moments':
        Nv = rng.choice([12, 16, 24, 32])
        return dict(kind=kind, Nv=Nv, dev=4 if Nv == 12 else 5 if Nv == 16 else 6,
                    ndof=_logint(rng, 16, 2300 if Nv == 32 else 5670), fp64=rng.random() < 0.2)
    if kind == 'hybrid':
        return dict(kind=kind, Nv=24, Nrho=12, M=12, dev=6, ndof=_logint(rng, 50, 3001),
                    far=rng.choice([0.0, 0.02, 0.05]), modes=rng.choice([256, 512]),
                    width=1024, center=rng.random() < 0.35)
    return dict(kind='step', nx=rng.randint(2, 14), ny=rng.randint(2, 8), order=rng.choice([2, 3]),
                Nv=24, Nrho=12, M=12, dev=6, fp64=False)


# ------------------------------------------------------------------ configs
def _ini(c, scat, extra='', velocity=''):
    return f"""
[backend]
precision = {'double' if c.get('fp64') else 'single'}
[constants]
Nv = {c['Nv']}
Nrho = {c.get('Nrho', 4)}
[non-dim]
T0 = {T0}
H0 = {H0}
rho0 = {RHO0}
molarMass0 = {MOLAR0}
[velocity-mesh]
dev = {c['dev']}
cmax = 0
Tmax = {T0}
{velocity}
[spherical-design-rule]
ssrule = womersley
M = {c.get('M', 6)}
[scattering-model]
{scat}
{extra}
"""


def _omega(c):
    return 0.5 if c.get('fp64') else OMEGA


def _vhs(c):
    return f"type = vhs-gll\nomega = {_omega(c)}\ndRef = {DREF}\nTref = {T0}"


def _bcs(sects):
    return '\n'.join(f"[soln-bcs-{name}]\ntype = dgfs-wall-diffuse\nrho = {RHO0}\nT = {T0 * T}\n"
                     f"ux = {ux * U0}\nuy = 0\nuz = 0\n" for name, T, ux in sects)


def _solver(system, order, scheme, dt):
    return f"""
[solver]
system = {system}
order = {order}
[solver-time-integrator]
scheme = {scheme}
controller = none
tstart = 0.0
tend = 1.0
dt = {dt}
[soln-ics]
type = maxwellian
rho = {RHO0}
T = {T0}
ux = 0
uy = 0
uz = 0
"""


CHANNEL = (('y-', 1.0, -0.3), ('y+', 1.1, 0.3))
CAVITY = (('lid', 1.0, 0.5), ('walls', 1.0, 0.0))
CAVITY_SIDES = {'x-': 'walls', 'x+': 'walls', 'y-': 'walls', 'y+': 'lid', 'z-': 'walls', 'z+': 'walls'}
DT = 5e-4


# ------------------------------------------------------------------ distributions
def _grid(Nv, L):
    return np.linspace(-L + L / Nv, L - L / Nv, Nv)


def _rand(seed, *shape):
    g = torch.Generator(device='cuda').manual_seed(1000003 * int(seed) + 17)
    return torch.rand(*shape, generator=g, device='cuda', dtype=torch.float64)


def _maxwellians(c0, rho, u, T, m=1.0):
    """Rows rho (m/(pi T))^1.5 exp(-m |c - u|^2 / T); rho, T [n], u [n, 3]."""
    x = torch.as_tensor(c0, device='cuda')[None, None, :] - u[:, :, None]
    e = torch.exp(-m * x * x / T[:, None, None])
    a = rho * (m / (math.pi * T))**1.5
    f = (a[:, None] * e[:, 0])[:, :, None, None] * e[:, 1][:, None, :, None] * e[:, 2][:, None, None, :]
    return f, x / T.sqrt()[:, None, None]


def _grad_rows(c0, seed, n, amp, dtype, chunk=512):
    """Maxwellians with Grad-type shear-stress and heat-flux parts, the shape
    of a rarefied flow's distributions; amp: [n] sizes of the parts."""
    r = _rand(seed, n, 9)
    out = torch.empty(n, len(c0)**3, dtype=dtype, device='cuda')
    for i in range(0, n, chunk):
        q = r[i:i + chunk]
        rho, T = 0.8 + 0.4 * q[:, 0], 0.85 + 0.35 * q[:, 1]
        u = torch.stack([0.7 * (q[:, 2] - 0.5), 0.2 * (q[:, 3] - 0.5), 0.2 * (q[:, 4] - 0.5)], 1)
        f, x = _maxwellians(c0, rho, u, T)
        X, Y, Z = x[:, 0][:, :, None, None], x[:, 1][:, None, :, None], x[:, 2][:, None, None, :]
        w = (2 * q[:, 5:9] - 1) * amp[i:i + chunk, None]
        v = lambda k: w[:, k][:, None, None, None]
        P = v(0) * X * Y + v(1) * Y * Z + v(2) * (X * X - Y * Y) / math.sqrt(2) \
            + v(3) * Y * (X * X + Y * Y + Z * Z - 2.5) / math.sqrt(2.5)
        out[i:i + chunk] = (f * torch.clamp(1 + P, min=0.0)).reshape(len(q), -1).to(dtype)
    return out


def _mixed_rows(c0, seed, n, dtype, noise=0.01, chunk=512):
    """Sums of two Maxwellians with 1 % relative noise."""
    r = _rand(seed, n, 10)
    out = torch.empty(n, len(c0)**3, dtype=dtype, device='cuda')
    g = torch.Generator(device='cuda').manual_seed(int(seed) + 5)
    for i in range(0, n, chunk):
        q = r[i:i + chunk]
        f = 0.0
        for k in (0, 5):
            f = f + _maxwellians(c0, 0.2 + 1.3 * q[:, k], 1.1 * (q[:, k + 1:k + 4] - 0.5),
                                 0.6 + 1.2 * q[:, k + 4])[0]
        f = f.reshape(len(q), -1)
        f = f * (1 + noise * (2 * torch.rand(f.shape, generator=g, device='cuda',
                                             dtype=torch.float64) - 1))
        out[i:i + chunk] = f.to(dtype)
    return out


def _dtype(c):
    return torch.float64 if c.get('fp64') else torch.float32


def _gas_rows(c, seed, n):
    c0 = _grid(c['Nv'], float(c['dev']))
    if c.get('family') == 'mixed':
        return _mixed_rows(c0, seed, n, _dtype(c))
    return _grad_rows(c0, seed, n, 0.3 * _rand(seed + 1, n), _dtype(c))


def _mixture_masses(c):
    return [1.0, c['heavy'] / MOLAR0]


def _mixture_rows(c, seed):
    c0 = _grid(c['Nv'], float(c['dev']))
    out = []
    for p, m in enumerate(_mixture_masses(c)):
        r = _rand(seed + 31 * p, c['ndof'], 10)
        f = 0.0
        for k in (0, 5):
            f = f + _maxwellians(c0, 0.3 + 0.9 * r[:, k], 0.6 * (r[:, k + 1:k + 4] - 0.5),
                                 0.7 + 0.6 * r[:, k + 4], m)[0]
        out.append(f.reshape(c['ndof'], -1).to(_dtype(c)))
    return out


def _hybrid_rows(c, seed):
    """Mostly near-equilibrium rows; a fraction ``far`` well past the threshold."""
    n = c['ndof']
    far = _rand(seed + 2, n) < c['far']
    amp = torch.where(far, torch.full_like(far, 0.6, dtype=torch.float64), 0.02 * _rand(seed + 1, n))
    r = _grad_rows(_grid(c['Nv'], float(c['dev'])), seed, n, amp, torch.float32)
    if bool(far.any()):                    # a second beam keeps them away from equilibrium
        k = int(far.sum())
        one = torch.ones(k, device='cuda', dtype=torch.float64)
        u = torch.tensor([[1.2, 0.4, 0.0]], device='cuda', dtype=torch.float64).expand(k, 3)
        beam = _maxwellians(_grid(c['Nv'], float(c['dev'])), 0.6 * one, u, 0.7 * one)[0]
        r[far] += beam.reshape(k, -1).float()
    return r


def _surrogate_state(c, seed):
    """Seeded weights in the layout of a saved surrogate."""
    n, k, w = c['Nv']**3, c['modes'], c['width']
    g = torch.Generator(device='cuda').manual_seed(int(seed) + 77)
    rn = lambda *s: torch.randn(*s, generator=g, device='cuda')
    nq = 24 if c['center'] else 0
    kin = (k + 4 + 15) // 16 * 16
    if c['center']:
        kin += 2 * k + (nq * (nq + 1) // 2 + 15) // 16 * 16
    W = [rn(o, i) * math.sqrt(s / i) for o, i, s in ((w, kin, 2), (w, w, 2), (w, w, 2), (3 * k, w + kin, 1))]
    return dict(Bd=rn(k, n) / math.sqrt(n), Bq=rn(3 * k, n) / math.sqrt(n), mu=0.01 * rn(k),
                sigma=torch.full((k,), 0.05, device='cuda'), hscale=torch.tensor([0.01, 0.3, 0.1], device='cuda'),
                W=W, b=[0.02 * rn(x.shape[0]) for x in W], k=k, w=w, Nv=c['Nv'], center=c['center'],
                split_out=False, nquad=nq)


# ------------------------------------------------------------------ prepare
def _gas_model(c):
    from frfs_b200.backend import CUDABackend
    from frfs_b200.inifile import Inifile
    from frfs_b200.scattering import DGFSVHSGLLScatteringModel
    from frfs_b200.velocitymesh import DGFSVelocityMesh
    cfg = Inifile(_ini(c, _vhs(c)))
    be = CUDABackend(cfg)
    return DGFSVHSGLLScatteringModel(be, cfg, DGFSVelocityMesh(be, cfg))


def _mesh(c):
    from frfs_b200.mesh import StructuredMesh
    if c.get('ndims', 2) == 3:
        return StructuredMesh((c['nx'], c['ny'], c['nz']), (0, 0, 0), (1.0, 0.8, 1.1), periodic='',
                              bcnames=CAVITY_SIDES)
    return StructuredMesh((c['nx'], c['ny']), (0.0, -0.5), (2.0, 0.5), periodic='x')


def _ndof(c):
    nd = c.get('ndims', 2)
    return c['nx'] * c['ny'] * (c['nz'] if nd == 3 else 1) * (c['order'] + 1)**nd


def _flow_rows(c, seed):
    n = _ndof(c)
    return _grad_rows(_grid(c['Nv'], float(c['dev'])), seed, n, 0.3 * _rand(seed + 1, n), _dtype(c))


def prepare(case, seed):
    c, kind = case, case['kind']
    from frfs_b200.backend import CUDABackend
    from frfs_b200.inifile import Inifile
    if kind == 'collide':
        f = _gas_rows(c, seed, c['ndof'])
        return dict(c=c, sm=_gas_model(c), f=f.view(c['ndof'], 1, -1), q=torch.empty_like(f).view(c['ndof'], 1, -1))
    if kind == 'pair':
        from frfs_b200.autotune import tune_vhs
        from frfs_b200.scattering import VHSCollider, VHSGrid, vhs_prefactor
        from frfs_b200.velocitymesh import DGFSVelocityMesh
        grids, batches = [], []
        for i, (Nv, n, mass) in enumerate(((24, c['n24'], 1.0), (32, c['n32'], 2.0))):
            d = dict(c, Nv=Nv, family='mixed')
            cfg = Inifile(_ini(d, _vhs(d)))
            be = CUDABackend(cfg)
            vm = DGFSVelocityMesh(be, cfg)
            gam, pref, _ = vhs_prefactor(vm, OMEGA, DREF, T0, mass=mass)
            grids.append(VHSGrid(Nv, vm.L(), vm.qz(), vm.qw(), vm.sz(), vm.sw(), gam, pref, vm.cw(),
                                 vm.c0(), be.fpdtype, be.device))
            f = _gas_rows(d, seed + i, n)
            batches.append((i, f, torch.empty_like(f), None))
        tune_vhs(grids, be.device)
        return dict(c=c, col=VHSCollider(grids, be.device), batches=batches)
    if kind == 'mixture':
        from frfs_b200.dgfsbi import DGFSBiVelocityMesh, DGFSBiVSSGLLScatteringModel
        pairs = '\n'.join(f'alpha{p}{q} = 1.3\nomega{p}{q} = {OMEGA}\ndRef{p}{q} = {DREF}\nTref{p}{q} = {T0}'
                          for p in range(2) for q in range(2))
        cfg = Inifile(_ini(c, f"type = vss-gll\nMpre = {c['Mpre']}\nssrulepre = womersley\n{pairs}",
                           velocity=f"molarMass1 = {MOLAR0}\nmolarMass2 = {c['heavy']}"))
        be = CUDABackend(cfg)
        fs = _mixture_rows(c, seed)
        return dict(c=c, sm=DGFSBiVSSGLLScatteringModel(be, cfg, DGFSBiVelocityMesh(be, cfg, 2)), fs=fs,
                    qs=[torch.empty_like(f) for f in fs])
    if kind == 'moments':
        from frfs_b200.velocitymesh import DGFSVelocityMesh
        cfg = Inifile(_ini(c, _vhs(c)))
        be = CUDABackend(cfg)
        return dict(c=c, vm=DGFSVelocityMesh(be, cfg), f=_gas_rows(c, seed, c['ndof']))
    if kind == 'hybrid':
        from frfs_b200.surrogate import HybridCollider, QSurrogate
        sm = _gas_model(c)
        q = QSurrogate(sm.grid, nmodes=c['modes'], width=c['width'], center=c['center'])
        q.load_state_dict(_surrogate_state(c, seed))
        f = _hybrid_rows(c, seed)
        return dict(c=c, hc=HybridCollider(q, threshold=0.05, recheck=0.02), f=f, q=torch.empty_like(f))
    if kind == 'relax':
        from frfs_b200.adgfs import ADGFSSystem
        from frfs_b200.integrators import STEPPERS, get_integrator
        cfg = Inifile(_ini(c, f"type = {c['model']}\nomega = {OMEGA}\nmuRef = {MUREF}\nTref = {T0}",
                           _solver('adgfs', c['order'], c['scheme'], DT) + _bcs(CHANNEL)))
        be = CUDABackend(cfg)
        s = ADGFSSystem(be, _mesh(c), cfg, nreg=STEPPERS[c['scheme']].nregs)
        s.eles_scal_upts_inb_full[0].view(-1).copy_(_flow_rows(c, seed).view(-1))
        integ = get_integrator(be, s, cfg)
        if 'bdf' in c['scheme']:           # the start-up calls belong to the program's past
            integ.step(0.0, DT)
        return dict(c=c, integ=integ)
    from frfs_b200.system import DGFSSystem
    bcs = CAVITY if c.get('ndims', 2) == 3 else CHANNEL
    cfg = Inifile(_ini(c, _vhs(c) + ('\ntile = 0' if kind == 'advect' else ''),
                       _solver('dgfs', c['order'], 'dgfs-tvd-rk2', DT) + _bcs(bcs)))
    be = CUDABackend(cfg)
    s = DGFSSystem(be, _mesh(c), cfg, nreg=4 if kind == 'advect' else 3)
    banks = s.eles_scal_upts_inb_full
    if kind == 'advect':
        # stage input, Q-like increment, step start; the result has a bank of its own
        for i in (1, 2, 0):
            banks[i].view(-1).copy_(_flow_rows(c, seed + 10 * i).view(-1))
        return dict(c=c, s=s)
    from frfs_b200.integrators import get_integrator
    banks[0].view(-1).copy_(_flow_rows(c, seed).view(-1))
    return dict(c=c, integ=get_integrator(be, s, cfg))


# ------------------------------------------------------------------ run
def run(state):
    c = state['c']
    kind = c['kind']
    if kind == 'collide':
        if c['point']:
            state['sm'].fs(state['f'], state['q'], 0, 0)
        else:
            state['sm'].collide(state['f'], state['q'])
        return {'Q': state['q']}
    if kind == 'pair':
        state['col'](state['batches'])
        return {'Q24': state['batches'][0][2], 'Q32': state['batches'][1][2]}
    if kind == 'mixture':
        state['sm'].collide(state['fs'], state['qs'])
        return {'Q0': state['qs'][0], 'Q1': state['qs'][1]}
    if kind == 'moments':
        from frfs_b200.system import macroscopic
        rho, U, T, q, P = macroscopic(state['f'], state['vm'])
        return {'rho': rho, 'U': U, 'T': T, 'q': q, 'P': P}
    if kind == 'hybrid':
        state['hc'](state['f'], state['q'], seed=5)
        return {'Q': state['q']}
    if kind == 'advect':
        s = state['s']
        s.advect_combine(0.0, 1, 3, a=0.5, b=0.5 * DT, x1=2, c1=0.5 * DT, x2=0, c2=0.5)
        return {'u': s.eles_scal_upts_inb_full[3]}
    state['integ'].step(0.0, DT)
    return {'u': state['integ'].soln}


# ------------------------------------------------------------------ work
def _q_flops(Nv, Nrho, M):
    n = Nv**3
    return (M * Nrho + Nrho + 2) * 5.0 * n * math.log2(n) + 8.0 * M * Nrho * n


def work(case):
    c, kind = case, case['kind']
    es = 8 if c.get('fp64') else 4
    if kind == 'pair':
        return {'bytes': 8.0 * (c['n24'] * 24**3 + c['n32'] * 32**3),
                'flops': c['n24'] * _q_flops(24, c['Nrho'], c['M']) + c['n32'] * _q_flops(32, c['Nrho'], c['M'])}
    n = c['Nv']**3
    if kind == 'collide':
        return {'bytes': 2.0 * es * n * c['ndof'], 'flops': c['ndof'] * _q_flops(c['Nv'], c['Nrho'], c['M'])}
    if kind == 'mixture':
        P = c['Nrho'] * c['M']
        item = (2 * (3 * P + 1) + 2) * 5.0 * n * math.log2(n) + 38.0 * 2 * P * n
        return {'bytes': 4.0 * es * n * c['ndof'] + 4 * P * n * 2.0 * es, 'flops': 2.0 * c['ndof'] * item}
    if kind == 'moments':
        return {'bytes': (es * n + 112.0) * c['ndof'], 'flops': 31.0 * n * c['ndof']}
    if kind == 'hybrid':
        k, w = c['modes'], c['width']
        kin = (k + 4 + 15) // 16 * 16 + (2 * k + 304 if c['center'] else 0)
        near = c['ndof'] * (1 - c['far'])
        gemm = n * k + kin * w + 2 * w * w + (w + kin) * 3 * k + 3 * k * n
        return {'bytes': 8.0 * n * c['ndof'] + 2.0 * gemm,
                'flops': 2.0 * near * gemm + (c['far'] + 0.02) * c['ndof'] * _q_flops(24, c['Nrho'], c['M'])}
    nd, el = _ndof(c), n * _ndof(c)
    d, p = c.get('ndims', 2), c['order'] + 1
    fr = (2 * d * p + 6 * d * 2) * 1.0 * el                      # line derivatives and face terms
    if kind == 'advect':
        return {'bytes': 4.0 * es * el, 'flops': fr}
    if kind == 'relax':
        s = {'adgfs-ars-111': 1, 'adgfs-ars-222': 2, 'adgfs-ars-443': 4, 'adgfs-bdf-2': 1}[c['scheme']]
        # per stage: L(f) in and out, then the earlier fields in and the new one out
        rows = sum(2 + 2 * a + 2 for a in range(s)) if 'ars' in c['scheme'] else 2 + 4 + 1
        return {'bytes': 1.0 * es * el * rows, 'flops': s * (fr + 40.0 * el)}
    return {'bytes': 2.0 * es * el * 5, 'flops': 2.0 * (fr + nd * _q_flops(c['Nv'], c['Nrho'], c['M']))}


# ------------------------------------------------------------------ exact
def _half_design(M):
    if M == 3:
        return np.eye(3)[[2, 0, 1]]
    if M == 6:
        r, z = 2 / math.sqrt(5), 1 / math.sqrt(5)
        a = -2 * math.pi * np.arange(5) / 5
        return np.concatenate([[[0.0, 0.0, 1.0]], np.stack([r * np.cos(a), r * np.sin(a), np.full(5, z)], 1)])
    s = math.sqrt(3 + math.sqrt(10))
    pts = []
    for pos in range(3):
        o = [i for i in range(3) if i != pos]
        for a in (1.0, -1.0):
            for b in (1.0, -1.0):
                v = [0.0] * 3
                v[pos], v[o[0]], v[o[1]] = s, a, b
                pts.append(v)
    return np.array(pts) / math.sqrt(2 + s * s)


def _full_design(M):
    h = _half_design(M // 2)
    return np.concatenate([h, -h])


def _radial(Nrho, R):
    z, w = np.polynomial.legendre.leggauss(Nrho)
    return R / 2 * (1 + z), R / 2 * w


def _wave(N):
    k = torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64, device='cuda')
    return k[:, None, None], k[None, :, None], k[None, None, :]


def _sinc(x):
    return torch.sin(x + 1e-15) / (x + 1e-15)


def _phi(c0):
    c = torch.as_tensor(c0, device='cuda')
    x, y, z = torch.meshgrid(c, c, c, indexing='ij')
    return torch.stack([torch.ones_like(x), x, y, z, x * x + y * y + z * z]).reshape(5, -1)


def _exact_q(f, Nv, dev, Nrho, M, omega, mass=1.0):
    """Projected Q of the rows f (any float type) in 64 bits."""
    L = float(dev)
    qz, qw = _radial(Nrho, 2 * (L * 2.0 / (3.0 + math.sqrt(2.0))))
    sz = _half_design(M)
    sw, n = 2 * math.pi / M, Nv**3
    gam = 2 * (1 - omega)
    pref = H0 * math.sqrt(2) * math.pi * N0 * DREF**2 / (
        math.sqrt(2) * (mass / 2)**(omega - 0.5) * 4 * math.gamma(2.5 - omega) * math.pi)
    lx, ly, lz = _wave(Nv)
    lm = torch.sqrt(lx * lx + ly * ly + lz * lz)
    bb2 = sum(qw[p] * qz[p]**(gam + 2) * 16 * math.pi**2 * _sinc(math.pi / L * qz[p] * lm) for p in range(Nrho))
    phi = _phi(_grid(Nv, L))
    gram = torch.linalg.inv(phi @ phi.T)
    out = torch.empty(f.shape[0], n, dtype=torch.float64, device='cuda')
    step = max(1, (48 << 20) // n)
    ift = lambda a: torch.fft.ifftn(a, dim=(1, 2, 3), norm='forward')
    for i in range(0, f.shape[0], step):
        x = f[i:i + step].double().view(-1, Nv, Nv, Nv)
        F = torch.fft.fftn(x, dim=(1, 2, 3)) / n
        G = torch.zeros_like(F)
        for p in range(Nrho):
            S = 0.0
            for s in sz:
                a = math.pi / L * qz[p] / 2 * (s[0] * lx + s[1] * ly + s[2] * lz)
                S = S + ift(torch.cos(a) * F)**2 + ift(torch.sin(a) * F)**2
            bb1 = qz[p]**(gam + 2) * 4 * math.pi * _sinc(math.pi / L * qz[p] / 2 * lm)
            G += (2 * qw[p] * sw / n) * bb1 * torch.fft.fftn(S, dim=(1, 2, 3))
        q = (pref * (ift(G).real - x * ift(bb2 * F).real)).reshape(-1, n)
        out[i:i + step] = q - (q @ phi.T) @ gram @ phi
    return out


def _exact_mixture(c, seed):
    fs = [f.double() for f in _mixture_rows(c, seed)]
    Nv, L, Nrho, M, n = c['Nv'], float(c['dev']), c['Nrho'], c['M'], c['Nv']**3
    m = _mixture_masses(c)
    mr = max(m)
    S = min(L * 2 / (max(4 * mr / (1 + mr), 2) + math.sqrt(1 + mr) + 1),
            L * 2 / (max(4 / (1 + mr), 2) + math.sqrt(1 + 1 / mr) + 1))
    qz, qw = _radial(Nrho, 2 * S)
    sz, szp = _full_design(M), _full_design(c['Mpre'])
    sw, swp = 4 * math.pi / M, 4 * math.pi / c['Mpre']
    # 1 + s.t with one rounding per fused multiply-add: its value at t = -s matters
    fma = lambda a, b, d: float(Fraction(a) * Fraction(b) + Fraction(d))
    opc = np.array([[max(fma(s[2], t[2], fma(s[1], t[1], fma(s[0], t[0], 1.0))), 0.0) for t in szp.tolist()]
                    for s in sz.tolist()])
    alpha, gam = 1.3, 2 * (1 - OMEGA)
    B = torch.as_tensor(opc**(alpha - 1), device='cuda').to(torch.complex128)
    lx, ly, lz = _wave(Nv)
    dot = lambda s: s[0] * lx + s[1] * ly + s[2] * lz
    tl = torch.stack([dot(t) for t in szp])
    ift = lambda a: torch.fft.ifftn(a, dim=(1, 2, 3), norm='forward')
    F = [torch.fft.fftn(f.view(-1, Nv, Nv, Nv), dim=(1, 2, 3)) / n for f in fs]
    out = []
    for p in range(2):
        Q = 0.0
        for q in range(2):
            mu, fq = m[p] * m[q] / (m[p] + m[q]), m[q] / (m[p] + m[q])
            pref = math.pi * N0 * DREF**2 * H0 * alpha / (
                mu**(OMEGA - 0.5) * 2**(1 + alpha) * math.gamma(2.5 - OMEGA) * math.pi)
            G = torch.zeros_like(F[0])
            cc = 0.0
            for r in range(Nrho):
                fac = math.pi / L * qz[r]
                fb = swp * qz[r]**(gam + 2)
                eb = torch.exp(-1j * fq * fac * tl)
                ec = torch.exp(-1j * fac * tl)
                cc = cc + qw[r] * sw * fb * torch.tensordot(B.sum(0), ec, dims=([0], [0]))
                for k, s in enumerate(sz):
                    a = fac * dot(s)
                    t = ift(torch.exp(1j * fq * a) * F[p]) * ift(torch.exp(-1j * (1 - fq) * a) * F[q])
                    b = fb * torch.tensordot(B[k], eb, dims=([0], [0]))
                    G += (qw[r] * sw / n) * b * torch.fft.fftn(t, dim=(1, 2, 3))
            Q = Q + pref * (ift(G).real - fs[p].view(-1, Nv, Nv, Nv) * ift(cc * F[q]).real)
        out.append(Q.reshape(-1, n))
    phi = _phi(_grid(Nv, L))
    z = torch.zeros(n, dtype=torch.float64, device='cuda')
    A = torch.stack([torch.cat([phi[0], z]), torch.cat([z, phi[0]])]
                    + [torch.cat([m[0] * phi[k], m[1] * phi[k]]) for k in (1, 2, 3, 4)])
    q = torch.cat(out, dim=1)
    q = q - (q @ A.T) @ torch.linalg.inv(A @ A.T) @ A
    return {'Q0': q[:, :n].contiguous(), 'Q1': q[:, n:].contiguous()}


class _Advection:
    """L(u) = -div(c u) on a box of tensor elements: upwind DG with
    Gauss-Lobatto points, exact mass matrix, diffuse walls."""

    def __init__(self, c):
        self.c, self.nd = c, c.get('ndims', 2)
        n = self.n = c['order'] + 1
        P = np.polynomial.legendre
        top = [0.0] * (n - 1) + [1.0]
        x = np.concatenate([[-1.0], np.sort(P.legroots(P.legder(top))), [1.0]])
        w = 2.0 / (n * (n - 1) * P.legval(x, top)**2)
        V = P.legvander(x, n - 1)
        dV = np.stack([P.legval(x, P.legder([0.0] * k + [1.0])) if k else 0 * x for k in range(n)], 1)
        K = V @ np.diag(np.arange(n) + 0.5) @ V.T                    # sum (k + 1/2) P_k P_k
        dv = lambda a: torch.as_tensor(np.ascontiguousarray(a), device='cuda')
        self.D, self.KW, self.Km, self.Kp = dv(dV @ np.linalg.inv(V)), dv(K * w), dv(K[:, 0]), dv(K[:, -1])
        shape = (c['nx'], c['ny'], c['nz']) if self.nd == 3 else (c['nx'], c['ny'])
        size = (1.0, 0.8, 1.1) if self.nd == 3 else (2.0, 1.0)
        self.shape, self.h = shape, [s / k for s, k in zip(size, shape)]
        c0 = _grid(c['Nv'], float(c['dev']))
        self.cw = (2.0 * c['dev'] / c['Nv'])**3
        g = torch.as_tensor(c0, device='cuda')
        self.cv = torch.stack([a.reshape(-1) for a in torch.meshgrid(g, g, g, indexing='ij')])
        one = torch.ones(1, device='cuda', dtype=torch.float64)
        self.walls = {}
        for name, T, ux in (CAVITY if self.nd == 3 else CHANNEL):
            u = torch.tensor([[ux, 0.0, 0.0]], device='cuda', dtype=torch.float64)
            self.walls[name] = (u[0], _maxwellians(c0, one, u, T * one)[0].reshape(-1))

    def _wall(self, axis, side):
        if self.nd == 2:
            return None if axis == 0 else self.walls['y+' if side > 0 else 'y-']
        return self.walls[CAVITY_SIDES['xyz'[axis] + ('+' if side > 0 else '-')]]

    def __call__(self, u):
        nd, n = self.nd, self.n
        # [z, y, x elements][z, y, x points][v]: element axes first, slowest first
        U = u.reshape(tuple(self.shape[::-1]) + (n,) * nd + (-1,))
        out = torch.zeros_like(U)
        for d in range(nd):
            e, p = nd - 1 - d, 2 * nd - 1 - d                        # element and point axis
            cd, s = self.cv[d], 2.0 / self.h[d]
            term = torch.movedim(torch.tensordot(self.D, U, dims=([1], [p])), 0, p) * cd
            lo, hi = U.select(p, 0), U.select(p, n - 1)
            left, right = torch.roll(hi, 1, e), torch.roll(lo, -1, e)     # neighbours' face values
            for side, own, nb in ((-1, lo, left), (+1, hi, right)):
                w = self._wall(d, side)
                if w is not None:
                    at = 0 if side < 0 else self.shape[d] - 1
                    uo = own.select(e, at)
                    fac = side * (cd - w[0][d])
                    b0 = (torch.clamp(fac, min=0) * uo).sum(-1, keepdim=True) * self.cw
                    b1 = (torch.clamp(fac, max=0) * w[1]).sum() * self.cw
                    nb.select(e, at).copy_(torch.where(fac < 0, w[1] * (-b0 / b1), uo))
            jl = torch.clamp(cd, min=0) * (left - lo)                    # f* - f at the left face
            jr = torch.clamp(cd, max=0) * (right - hi)
            for j, k, sg in ((jl, self.Km, -1.0), (jr, self.Kp, 1.0)):
                for t in range(nd - 1):                                   # tangential quadrature
                    j = torch.movedim(torch.tensordot(self.KW, j, dims=([1], [nd + t])), 0, nd + t)
                shp = [1] * U.dim()
                shp[p] = n
                term = term + sg * k.view(shp) * j.unsqueeze(p)
            out -= s * term
        return out.reshape(u.shape)


class _Relaxation:
    """Moments, targets and the IMEX updates of the three relaxation models."""

    def __init__(self, c):
        self.model = c['model'].split('-')[0]
        g = torch.as_tensor(_grid(c['Nv'], float(c['dev'])), device='cuda')
        self.cv = torch.stack([a.reshape(-1) for a in torch.meshgrid(g, g, g, indexing='ij')])
        x, y, z = self.cv
        r2 = (self.cv**2).sum(0)
        rows = [torch.ones_like(x), x, y, z, r2, x * x, y * y, z * z, x * y, y * z, z * x, r2 * x, r2 * y, r2 * z]
        self.rows = torch.stack(rows[:{'bgk': 5, 'esbgk': 11, 'shakov': 14}[self.model]]) * (2.0 * c['dev'] / c['Nv'])**3
        self.Pr = 1.0 if self.model == 'bgk' else 2.0 / 3.0
        self.pref = (H0 / U0) * (N0 * R0 / NA * T0) / MUREF * (self.Pr if self.model == 'esbgk' else 1.0)

    def mom(self, f):
        return f @ self.rows.T

    def _st(self, U):
        rho, u = U[:, 0], U[:, 1:4] / U[:, :1]
        return rho, u, (U[:, 4] - (U[:, 1:4]**2).sum(1) / rho) / (1.5 * rho)

    def nu(self, U):
        rho, _, T = self._st(U)
        return (self.pref * rho * T**(1 - OMEGA))[:, None]

    def _stress(self, U):
        return torch.stack([U[:, [5, 8, 10]], U[:, [8, 6, 9]], U[:, [10, 9, 7]]], 1)

    def _heat(self, U):
        """2 P u - rho |u|^2 u + 1.5 rho T u (Q - q)."""
        rho, u, T = self._st(U)
        return 2 * (self._stress(U) @ u[:, :, None])[:, :, 0] + ((1.5 * rho * T - rho * (u * u).sum(1))[:, None]) * u

    def target(self, U):
        rho, u, T = self._st(U)
        d = self.cv[None] - u[:, :, None]
        if self.model == 'esbgk':
            k = 2 * (1 - 1 / self.Pr)
            A = k * (self._stress(U) / rho[:, None, None] - u[:, :, None] * u[:, None, :]) \
                + (T / self.Pr)[:, None, None] * torch.eye(3, device='cuda', dtype=torch.float64)
            q = (d * (torch.linalg.inv(A) @ d)).sum(1)
            return (rho / (math.pi**1.5 * torch.sqrt(torch.linalg.det(A))))[:, None] * torch.exp(-q)
        d2 = (d * d).sum(1)
        M = (rho / (math.pi * T)**1.5)[:, None] * torch.exp(-d2 / T[:, None])
        if self.model == 'shakov':
            q = U[:, 11:14] - self._heat(U)
            M = M * (1 + (2 * (1 - self.Pr) / (5 * rho * T * T))[:, None] * (q[:, :, None] * d).sum(1)
                     * (2 * d2 / T[:, None] - 5))
        return M

    def _second(self, U):
        rho, u, T = self._st(U)
        h = 0.5 * rho * T
        return torch.stack([h + rho * u[:, 0]**2, h + rho * u[:, 1]**2, h + rho * u[:, 2]**2, rho * u[:, 0] * u[:, 1],
                            rho * u[:, 1] * u[:, 2], rho * u[:, 2] * u[:, 0]], 1)

    def _hsrc(self, U):
        rho, u, T = self._st(U)
        return ((rho * (u * u).sum(1) + 2.5 * rho * T)[:, None]) * u - (1 - self.Pr) * self._heat(U)

    def solve(self, N, a, w, past=()):
        """Moments of the implicit stage: a U = N + w rate (target - U) for the
        higher rows; past: (weight, U) of earlier implicit parts."""
        U = N / a
        nu = self.nu(U)
        s2 = 1 / self.Pr if self.model == 'esbgk' else 1.0
        if self.model != 'bgk':
            num = N[:, 5:11] + sum(x * s2 * self.nu(V) * (self._second(V) - V[:, 5:11]) for x, V in past)
            U[:, 5:11] = (num + w * s2 * nu * self._second(U)) / (a + w * s2 * nu)
        if self.model == 'shakov':
            num = N[:, 11:14] + sum(x * self.nu(V) * (self._hsrc(V) - self.Pr * V[:, 11:14]) for x, V in past)
            U[:, 11:14] = (num + w * nu * self._hsrc(U)) / (a + w * self.Pr * nu)
        return U

    def ars(self, f0, dt, adv, E, I):
        s = len(E) - 1
        F, Ls, LU, U = [f0], [], [], [self.mom(f0)]
        for a in range(1, s + 1):
            Ls.append(adv(F[-1]))
            LU.append(self.mom(Ls[-1]))
            past = [(I[a][j] * dt, U[j]) for j in range(1, a)]
            w = I[a][a] * dt
            U.append(self.solve(U[0] + dt * sum(E[a][j] * LU[j] for j in range(a)), 1.0, w, past))
            num = F[0] + sum(E[a][j] * dt * Ls[j] for j in range(a))
            for j in range(1, a):
                num += I[a][j] * dt * self.nu(U[j]) * (self.target(U[j]) - F[j])
            nu = self.nu(U[a])
            F.append((num + w * nu * self.target(U[a])) / (1 + w * nu))
        return F[-1]


_G = 1 - math.sqrt(2) / 2
_DL = 1 - 1 / (2 * _G)
ARS = {
    'adgfs-ars-111': ([[0, 0], [1, 0]], [[0, 0], [0, 1]]),
    'adgfs-ars-222': ([[0, 0, 0], [_G, 0, 0], [_DL, 1 - _DL, 0]], [[0, 0, 0], [0, _G, 0], [0, 1 - _G, _G]]),
    'adgfs-ars-443': ([[0] * 5, [1 / 2, 0, 0, 0, 0], [11 / 18, 1 / 18, 0, 0, 0], [5 / 6, -5 / 6, 1 / 2, 0, 0],
                       [1 / 4, 7 / 4, 3 / 4, -7 / 4, 0]],
                      [[0] * 5, [0, 1 / 2, 0, 0, 0], [0, 1 / 6, 1 / 2, 0, 0], [0, -1 / 2, 1 / 2, 1 / 2, 0],
                       [0, 3 / 2, -3 / 2, 1 / 2, 1 / 2]]),
}


def _exact_relax(c, seed):
    f = _flow_rows(c, seed).double()
    R, A = _Relaxation(c), _Advection(c)
    adv = lambda x: A(x)
    if c['scheme'] in ARS:
        return R.ars(f, DT, adv, *ARS[c['scheme']])
    g = f
    for _ in range(10):                                        # BDF-2 start-up: ARS-222 sub-steps
        g = R.ars(g, DT / 10, adv, *ARS['adgfs-ars-222'])
    h = [f, g]
    L = [adv(x) for x in h]
    a, b, gx = (1 / 3, -4 / 3, 1.0), 2 / 3, (2 / 3, -4 / 3)
    N = -sum(a[i] * R.mom(h[i]) + gx[i] * DT * R.mom(L[i]) for i in range(2))
    U = R.solve(N, a[2], b * DT)
    Nf = -sum(a[i] * h[i] + gx[i] * DT * L[i] for i in range(2))
    w = b * DT * R.nu(U)
    return (Nf + w * R.target(U)) / (a[2] + w)


def _exact_moments(f, c):
    g = torch.as_tensor(_grid(c['Nv'], float(c['dev'])), device='cuda')
    cv = torch.stack([a.reshape(-1) for a in torch.meshgrid(g, g, g, indexing='ij')])
    cw = (2.0 * c['dev'] / c['Nv'])**3
    o = [[], [], [], [], []]
    for i in range(0, f.shape[0], 256):
        x = f[i:i + 256].double()
        rho = x.sum(1) * cw
        U = x @ cv.T * cw / rho[:, None]
        d = cv[None] - U[:, :, None]
        d2 = (d * d).sum(1)
        T = (x * d2).sum(1) * (2.0 / 3.0) * cw / rho
        q = (d * (x * d2)[:, None]).sum(2) * cw
        P = 2 * cw * torch.stack([(x * d[:, a] * d[:, b]).sum(1) for a, b in
                                  ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], 1)
        for k, v in enumerate((rho, U, T, q, P)):
            o[k].append(v)
    return dict(zip(('rho', 'U', 'T', 'q', 'P'), (torch.cat(v) for v in o)))


def _mix(x):
    """The re-check hash (splitmix64 finaliser, upper half)."""
    m = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & m
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & m
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & m
    return (x ^ (x >> 31)) >> 32


def _shift(x, a, N, sign):
    """Rows of x (cubes) moved by sign * a grid cells per axis (trigonometric)."""
    k = torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64, device='cuda')
    X = x.view(-1, N, N, N).to(torch.complex128)
    for d in range(3):
        ph = torch.exp(1j * 2 * math.pi * sign * a[:, d:d + 1] * k[None] / N)
        ph[:, N // 2] = ph[:, N // 2].real.to(torch.complex128)
        shp = [len(x), 1, 1, 1]
        shp[1 + d] = N
        X = torch.fft.ifft(torch.fft.fft(X, dim=1 + d) * ph.view(shp), dim=1 + d)
    return X.real.reshape(x.shape)


def _exact_hybrid(c, seed):
    f = _hybrid_rows(c, seed)
    s = {k: ([x.double() for x in v] if isinstance(v, list) else v.double() if torch.is_tensor(v) else v)
         for k, v in _surrogate_state(c, seed).items()}
    Nv, dev, n, k = c['Nv'], float(c['dev']), c['Nv']**3, c['modes']
    c0 = _grid(Nv, dev)
    cw = (2.0 * dev / Nv)**3
    phi = _phi(c0)
    gram = torch.linalg.inv(phi @ phi.T)
    out = torch.empty(f.shape, dtype=torch.float64, device='cuda')
    spectral = []
    sc = s['hscale'].repeat_interleave(k)
    for i in range(0, len(f), 256):
        x = f[i:i + 256].double()
        m = x @ phi.T
        rho, u = m[:, 0] * cw, m[:, 1:4] / m[:, :1]
        T = (m[:, 4] / m[:, 0] - (u * u).sum(1)) * (2.0 / 3.0)
        d = x - _maxwellians(c0, rho, u, T)[0].reshape(len(x), -1)
        size = d.norm(dim=1)
        near = (size / x.norm(dim=1) < 0.05).tolist()
        for j in range(len(x)):
            again = _mix((5 * 0x100000001B3 + i + j) & ((1 << 64) - 1)) < 0.02 * 4294967296.0
            if not near[j] or again:
                spectral.append(i + j)
        a = u / (c0[1] - c0[0])
        dh = d / size[:, None]
        if c['center']:
            dh = _shift(dh, a, Nv, 1.0)
        e = (dh @ s['Bd'].T - s['mu']) / s['sigma']
        t = (T - 1)[:, None]
        cols = [e, 0 * u if c['center'] else u, t, torch.zeros(len(x), (k + 4 + 15) // 16 * 16 - k - 4, device='cuda',
                                                            dtype=torch.float64)]
        if c['center']:
            nq = s['nquad']
            iu = torch.triu_indices(nq, nq, device='cuda')
            quad = e[:, iu[0]] * e[:, iu[1]]
            pad = (nq * (nq + 1) // 2 + 15) // 16 * 16 - nq * (nq + 1) // 2
            cols += [t * e, t * t * e, quad, torch.zeros(len(x), pad, device='cuda', dtype=torch.float64)]
        z = torch.cat(cols, 1)
        h = z
        for l in range(3):
            h = torch.nn.functional.gelu(h @ s['W'][l].T + s['b'][l], approximate='none')
        Y = (torch.cat([h, z], 1) @ s['W'][3].T + s['b'][3]) * sc
        sz = (size / rho)[:, None]
        Y = torch.cat([Y[:, :k], sz * Y[:, k:2 * k], sz * sz * Y[:, 2 * k:]], 1)
        q = (rho * rho)[:, None] * (Y @ s['Bq'])
        if c['center']:
            q = _shift(q, a, Nv, -1.0)
        out[i:i + 256] = q - (q @ phi.T) @ gram @ phi
    if spectral:
        idx = torch.tensor(spectral, device='cuda')
        out[idx] = _exact_q(f[idx], Nv, c['dev'], c['Nrho'], c['M'], OMEGA)
    return out


def exact(case, seed):
    c, kind = case, case['kind']
    if kind == 'collide':
        q = _exact_q(_gas_rows(c, seed, c['ndof']), c['Nv'], c['dev'], c['Nrho'], c['M'], _omega(c))
        return {'Q': q.view(c['ndof'], 1, -1)}
    if kind == 'pair':
        r = {}
        for i, (Nv, n, mass) in enumerate(((24, c['n24'], 1.0), (32, c['n32'], 2.0))):
            f = _gas_rows(dict(c, Nv=Nv, family='mixed'), seed + i, n)
            r[f'Q{Nv}'] = _exact_q(f, Nv, c['dev'], c['Nrho'], c['M'], OMEGA, mass)
        return r
    if kind == 'mixture':
        return _exact_mixture(c, seed)
    if kind == 'moments':
        return _exact_moments(_gas_rows(c, seed, c['ndof']), c)
    if kind == 'hybrid':
        return {'Q': _exact_hybrid(c, seed)}
    n = c['Nv']**3
    ne = _ndof(c) // (c['order'] + 1)**c.get('ndims', 2)
    shape = (ne, _ndof(c) // ne, n)
    if kind == 'relax':
        return {'u': _exact_relax(c, seed).view(shape)}
    A = _Advection(c)
    if kind == 'advect':
        u1 = _flow_rows(c, seed + 10).double()
        r = 0.5 * u1 + 0.5 * DT * A(u1)
        r += 0.5 * DT * _flow_rows(c, seed + 20)
        r += 0.5 * _flow_rows(c, seed)
        return {'u': r.view(shape)}
    Q = lambda x: _exact_q(x, c['Nv'], c['dev'], c['Nrho'], c['M'], OMEGA)
    u = _flow_rows(c, seed).double()
    u1 = u + DT * (A(u) + Q(u))
    return {'u': (0.5 * u + 0.5 * u1 + 0.5 * DT * (A(u1) + Q(u1))).view(shape)}
