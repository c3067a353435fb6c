"""The solver's work as its users have it done, as cases that can be timed.

A case is a dict of plain values.  ``kind`` says which public entry points a
pass goes through:

* ``steps``      ``psik = ...``, ``full_steps(n)``, read ``psik``;
* ``loop``       the same with one ``full_step()`` per step, as scripts that
                 look at the state between steps write it;
* ``pops``       ``full_steps(n, pops)``: populations after every step, the
                 way ``prop_loop`` advances the state;
* ``prop_loop``  the whole ``prop_loop`` call with its ``PropResult``;
* ``fft``        ``fft_2d`` and ``ifft_2d`` of a CUDA spinor;
* ``batch``      ``PropagatorBatch.full_steps`` of several uneven solves.

``problem`` names the physics (see ``PROBLEMS``), ``dtype`` the arithmetic:
``c64``, ``c128`` (the default of the original package) or ``df``
(double-float).  Inputs are made from the seed alone: a Thomas-Fermi state
with +/-0.01 rad phase noise, vortices where the problem has them.
"""
import math
import os
import sys
import tempfile
import types

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    'spinor-gpe_gb300')
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

# Physics of the measured problems (spacing dx, trap aspect lam, couplings g,
# Raman coupling omega with recoil kl, detuning delta, time and its step).
PROBLEMS = {
    # plain imaginary-time ground state, no coupling
    'ground': dict(dx=0.125, lam=1.0, g=(1000.0, 995.0, 990.0), omega=None,
                   kl=1.0, delta=0.0, time='imag', dt=0.02, vortices=0),
    # Raman-dressed gas after a detuning quench, real time
    'quench': dict(dx=0.0625, lam=1.0, g=(1000.0, 1000.0, 990.0), omega=1.0,
                   kl=3.0, delta=0.5, time='real', dt=1e-3, vortices=0),
    # anisotropic trap with vortices, imaginary time, Raman coupling
    'vortex': dict(dx=96.0 / 2048, lam=1.2, g=(2000.0, 1990.0, 1980.0),
                   omega=0.5, kl=2.0, delta=0.0, time='imag', dt=0.01,
                   vortices=8),
    # a lattice at an angle to the grid on top of the trap: the potential has
    # no separable form, so the operators are full fields
    'lattice': dict(dx=0.125, lam=1.0, g=(800.0, 796.0, 792.0), omega=0.8,
                    kl=3.0, delta=0.2, time='imag', dt=0.02, vortices=0),
}
SIDES = (32, 64, 128, 192, 256, 384, 512, 768, 1024, 2048, 4096)
BATCH_SIDES = (128, 192, 256, 384, 512, 768, 1024)
DTYPE = {'c64': 64, 'c128': 128, 'df': 'double-float'}


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest solves, stepped one call at a time: launch latency
        dict(name='loop_64_c64', kind='loop', problem='ground', dtype='c64',
             nx=64, ny=64, n=32),
        # the original package's default: 256 x 256 in complex128
        dict(name='ground_256_c128', kind='steps', problem='ground',
             dtype='c128', nx=256, ny=256, n=33),
        # a medium solve with its populations recorded every step
        dict(name='pops_512_c64', kind='pops', problem='quench', dtype='c64',
             nx=512, ny=512, n=40),
        # the headline problem in each precision
        dict(name='quench_1024_c64', kind='steps', problem='quench',
             dtype='c64', nx=1024, ny=1024, n=25),
        dict(name='quench_1024_df', kind='steps', problem='quench',
             dtype='df', nx=1024, ny=1024, n=17),
        dict(name='quench_1024_c128', kind='steps', problem='quench',
             dtype='c128', nx=1024, ny=1024, n=9),
        # a vortex lattice start: the state is as large as the L2
        dict(name='vortex_2048_c64', kind='steps', problem='vortex',
             dtype='c64', nx=2048, ny=2048, n=9),
        # ragged sides and operators that are full fields
        dict(name='lattice_768x384_c64', kind='steps', problem='lattice',
             dtype='c64', nx=768, ny=384, n=17),
        # both transform directions on their own, as set-up and analysis
        # scripts call them
        dict(name='fft_512x768_c128', kind='fft', problem='quench',
             dtype='c128', nx=512, ny=768, n=1),
        # the whole drop-in call: populations every step, energies, derived
        # fields and host copies of the result
        dict(name='prop_loop_256x128_c128', kind='prop_loop',
             problem='quench', dtype='c128', nx=256, ny=128, n=48),
        # a parameter scan: independent solves of uneven sizes together
        dict(name='batch_12_c64', kind='batch', problem='ground',
             dtype='c64', nx=0, ny=0, n=17, solves=12, mix=4),
        # the largest grid
        dict(name='vortex_4096_c64', kind='steps', problem='vortex',
             dtype='c64', nx=4096, ny=4096, n=3),
    ]


# rough cost of one point of one step by precision, complex64 = 1
_COST = {'c64': 1.0, 'df': 4.7, 'c128': 26.0}


def draw(rng):
    kind = rng.choice(('loop', 'steps', 'steps', 'pops', 'fft', 'prop_loop',
                       'batch'))
    dtype = rng.choice(('c64', 'c64', 'c128', 'df'))
    problem = rng.choice(tuple(PROBLEMS))
    if kind == 'batch':
        return dict(kind=kind, problem='ground', dtype='c64', nx=0, ny=0,
                    n=rng.randint(3, 17), solves=rng.randint(2, 12),
                    mix=rng.randint(0, 10**6))
    if kind == 'prop_loop' and dtype == 'c64':
        dtype = 'c128'   # populations and energies come in 64 bits
    if kind == 'fft':
        dtype = 'c128' if dtype == 'c128' else 'c64'
    while True:
        nx, ny = rng.choice(SIDES), rng.choice(SIDES)
        if max(nx, ny) > 8 * min(nx, ny):
            continue
        if kind == 'loop' and nx * ny > 512 * 512:
            continue
        if kind == 'prop_loop' and nx * ny > 1024 * 1024:
            continue
        if problem == 'lattice' and nx * ny > 1024 * 1024:
            continue
        n = 1 if kind == 'fft' else int(round(math.exp(
            rng.uniform(math.log(3), math.log(64)))))
        if nx * ny * n <= 3 * 4096**2 and nx * ny * n * _COST[dtype] <= 2.4e8:
            return dict(kind=kind, problem=problem, dtype=dtype, nx=nx,
                        ny=ny, n=n)


def _solves(case):
    """The solves of a case: one, or the batch's uneven set."""
    base = PROBLEMS[case['problem']]
    if case['kind'] != 'batch':
        return [dict(base, nx=case['nx'], ny=case['ny'],
                     lattice=case['problem'] == 'lattice')]
    r = np.random.RandomState(case['mix'])
    out = []
    for _ in range(case['solves']):
        side, guu = int(r.choice(BATCH_SIDES)), float(r.uniform(100, 2000))
        out.append(dict(base, nx=side, ny=side, lattice=False,
                        lam=float(r.uniform(0.5, 2.0)),
                        g=(guu, 0.995 * guu, 0.99 * guu),
                        omega=float(r.uniform(0, 2)), kl=3.0,
                        delta=float(r.uniform(-0.5, 0.5))))
    return out


def work(case):
    """One pass: the state read once and written once (a transform's input
    and its two results for ``fft``), and the flops of the transforms
    (5 N log2 N) and of the point-wise operators (about 60 per point and
    component with the interaction phase)."""
    elem = 8 if case['dtype'] == 'c64' else 16
    nbytes = flops = 0.0
    for s in _solves(case):
        pts = 2.0 * s['nx'] * s['ny']
        transform = 5.0 * pts * math.log2(s['nx'] * s['ny'])
        if case['kind'] == 'fft':
            nbytes += 3 * pts * elem
            flops += 2 * transform
        else:
            nbytes += 2 * pts * elem
            flops += case['n'] * 3 * (2 * transform + 60.0 * pts)
        if case['kind'] == 'prop_loop':   # psi, psik, densities, phases
            nbytes += pts * (elem + 3 * 8)
    return {'bytes': nbytes, 'flops': flops}


# ------------------------------------------------------------------ inputs
def _grid(s):
    """1-D grids and volume elements, as the spinor set-up defines them."""
    half = [s['nx'] * s['dx'] / 2, s['ny'] * s['dx'] / 2]
    num = (s['nx'], s['ny'])
    lin = [np.linspace(-h, h, num=n, endpoint=False) for h, n in zip(half, num)]
    dr = np.array([2 * h / n for h, n in zip(half, num)])
    dk = np.array([np.pi / h for h in half])
    klin = [np.linspace(-np.pi / d, np.pi / d, num=n, endpoint=False)
            for d, n in zip(dr, num)]
    return lin, klin, dr, dk


def _lattice(x, y):
    return 3.0 * np.sin(0.9 * x + 0.5 * y)**2


def _state(s, seed, ctype):
    """Real-space Thomas-Fermi spinor with seeded phase noise and vortices."""
    (x, y), _, _, _ = _grid(s)
    dev = 'cuda'
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    xt = torch.as_tensor(x, device=dev)[None, :]
    yt = torch.as_tensor(y, device=dev)[:, None]
    g_eff = 0.5 * (s['g'][0] + s['g'][2])
    mu = math.sqrt(g_eff * s['lam'] / math.pi)
    pot = 0.5 * (xt**2 + (s['lam'] * yt)**2)
    prof = torch.sqrt(torch.clamp(mu - pot, min=0.0) / g_eff * 0.5)
    psi = []
    for _ in range(2):
        ph = torch.rand(prof.shape, generator=gen, device=dev,
                        dtype=torch.float64) * 0.02 - 0.01
        psi.append(torch.polar(prof, ph))
    r = np.random.RandomState(seed % (1 << 31))
    for k in range(s['vortices']):
        a, b = r.uniform(-0.4, 0.4, 2) * math.sqrt(2 * mu)
        sgn = 1 if k % 2 == 0 else -1
        dx, dy = xt - a, yt - b
        d = torch.sqrt(dx**2 + dy**2) / 0.3
        f = torch.polar(d / torch.sqrt(d**2 + 1), sgn * torch.atan2(dy, dx))
        psi = [p * f for p in psi]
    return [p.to(ctype) for p in psi]


def _fft(psi, dr):
    c = float(np.prod(dr)) / (2 * math.pi)
    return [torch.fft.fftshift(torch.fft.fft2(p) * c) for p in psi]


def _inputs(case, s, seed):
    """(psi, psik) of one solve in the precision its user hands over."""
    ctype = torch.complex64 if case['dtype'] == 'c64' else torch.complex128
    _, _, dr, _ = _grid(s)
    psi = _state(s, seed, torch.complex128)
    return [p.to(ctype) for p in psi], [p.to(ctype) for p in _fft(psi, dr)]


def _propagator(case, s, psik):
    from spinor_gpe.pspinor.device_spinor import DeviceSpinor
    from spinor_gpe.pspinor.operators import SepField
    from spinor_gpe.pspinor.pspinor import PSpinor
    from spinor_gpe.pspinor.tensor_propagator import TensorPropagator
    path = os.path.join(tempfile.mkdtemp(prefix='sgpe_case_'), 'run')
    cls = PSpinor if s['lattice'] else DeviceSpinor
    ps = cls(path, overwrite=True, atom_num=1.0,
             mesh_points=(s['nx'], s['ny']),
             r_sizes=(s['nx'] * s['dx'] / 2, s['ny'] * s['dx'] / 2))
    ps.g_sc = dict(zip(('uu', 'dd', 'ud'), s['g']))
    if s['lattice']:
        xm, ym = ps.space['x_mesh'], ps.space['y_mesh']
        ps.pot_eng = 0.5 * (xm**2 + (s['lam'] * ym)**2) + _lattice(xm, ym)
    else:
        ps.pot_eng = SepField(ps.space['x']**2 / 2,
                              (s['lam'] * ps.space['y'])**2 / 2)
    if s['omega'] is not None:
        ps.coupling_setup(kin_shift=False)
        ps.kL_recoil = s['kl']
        ps.rot_coupling = False
        ps.coupling_uniform(s['omega'])
        ps.detuning_uniform(s['delta'])
    ps.psik = psik
    return TensorPropagator(ps, s['dt'], case['n'], 'cuda', time=s['time'],
                            dtype=DTYPE[case['dtype']])


def prepare(case, seed):
    st = types.SimpleNamespace(case=case)
    solves = _solves(case)
    data = [_inputs(case, s, seed + 1000 * i) for i, s in enumerate(solves)]
    if case['kind'] == 'fft':
        import spinor_gpe.pspinor.tensor_tools as ttools
        st.ttools, st.psi, st.dr = ttools, data[0][0], _grid(solves[0])[2]
        return st
    st.psik0 = [psik for _, psik in data]
    st.props = [_propagator(case, s, psik) for s, psik in zip(solves, st.psik0)]
    if case['kind'] == 'batch':
        from spinor_gpe.batch import PropagatorBatch
        st.batch = PropagatorBatch(st.props)
    return st


# -------------------------------------------------------------------- pass
def run(st):
    case = st.case
    kind, n = case['kind'], case['n']
    if kind == 'fft':
        psik = st.ttools.fft_2d(st.psi, st.dr)
        return {'psik': psik, 'psi': st.ttools.ifft_2d(psik, st.dr)}
    for prop, psik in zip(st.props, st.psik0):
        prop.psik = psik
    if kind == 'batch':
        st.batch.full_steps(n)
        return [prop.psik for prop in st.props]
    prop = st.props[0]
    if kind == 'steps':
        prop.full_steps(n)
        return {'psik': prop.psik}
    if kind == 'loop':
        for _ in range(n):
            prop.full_step()
        return {'psik': prop.psik}
    if kind == 'pops':
        pops = torch.empty((n, 2), dtype=torch.float64, device='cuda')
        prop.full_steps(n, pops)
        psik = prop.psik          # also fills the last row of pops
        # kept at the precision of the solve
        return {'psik': psik,
                'pops': pops.float() if case['dtype'] == 'c64' else pops}
    res = prop.prop_loop(n)
    return {'psi': res.psi, 'psik': res.psik, 'pops': res.pops['vals'],
            'energy': [float(e) for e in res.eng_final], 'dens': res.dens,
            'densk': res.densk, 'phase': res.phase,
            'separation': float(res.calc_separation())}


# ------------------------------------------------------------------- exact
def _exact_steps(s, psik, n, want_pops=False):
    """The split step in complex128 with plain torch operations: psik after
    n full steps in centred order, and the populations after each."""
    (x, y), (kx, ky), dr, dk = _grid(s)
    dev = 'cuda'
    nat = torch.fft.ifftshift

    def mesh(a, b):
        return (torch.as_tensor(a, device=dev)[None, :],
                torch.as_tensor(b, device=dev)[:, None])
    xm, ym = mesh(x, y)
    kxm, kym = mesh(np.fft.ifftshift(kx), np.fft.ifftshift(ky))
    kin = (kxm**2 + kym**2) / 2
    pot = 0.5 * (xm**2 + (s['lam'] * ym)**2)
    if s['lattice']:
        pot = pot + 3.0 * torch.sin(0.9 * xm + 0.5 * ym)**2
    coupled = s['omega'] is not None
    det = s['delta'] / 2 if coupled else 0.0
    pots = [pot + det, pot - det]
    dv_r, dv_k = float(np.prod(dr)), float(np.prod(dk))
    c = dv_r / (2 * math.pi)
    dt = -1j * s['dt'] if s['time'] == 'imag' else s['dt'] + 0j
    gam = 1 / (2 + 2**(1 / 3))
    subs = []
    theta = 2 * s['kl'] * xm
    for t in (dt * gam, dt * (1 - 2 * gam)):
        # each of the two coupling half steps rotates by omega t / 4
        arg = torch.tensor((s['omega'] or 0.0) * t / 4, dtype=torch.complex128)
        cc = complex(torch.cos(arg))
        sc = complex(-1j * torch.sin(arg))
        ph = torch.polar(torch.ones_like(theta), theta)
        subs.append((t, torch.exp(-1j * (t / 2) * kin),
                     [torch.exp(-1j * t * v) for v in pots],
                     cc, sc * ph.conj(), sc * ph))
    g = s['g']
    pk = [nat(p.to(torch.complex128)) for p in psik]

    def normed(z, dv):
        f = sum((p.real**2 + p.imag**2).sum() for p in z) * dv
        return [p / torch.sqrt(f) for p in z]
    pops = []
    for _ in range(n):
        for i in (0, 1, 0):
            t, k, v, cc, s01, s10 = subs[i]
            z = [torch.fft.ifft2(k * p) / c for p in pk]
            z = normed(z, dv_r)
            d = [p.real**2 + p.imag**2 for p in z]
            e = [g[0] * d[0] + g[2] * d[1], g[1] * d[1] + g[2] * d[0]]
            io = [torch.exp(-1j * (t / 2) * w) for w in e]
            z = [o * p for o, p in zip(io, z)]
            if coupled:
                z = [cc * z[0] + s01 * z[1], s10 * z[0] + cc * z[1]]
            z = [w * p for w, p in zip(v, z)]
            if coupled:
                z = [cc * z[0] + s01 * z[1], s10 * z[0] + cc * z[1]]
            z = [o * p for o, p in zip(io, z)]
            pk = normed([k * (torch.fft.fft2(p) * c) for p in z], dv_k)
        if want_pops:
            pops.append(torch.stack([(p.real**2 + p.imag**2).sum() * dv_k
                                     for p in pk]))
    return ([torch.fft.fftshift(p) for p in pk],
            torch.stack(pops) if want_pops else None)


def exact(case, seed):
    kind, n = case['kind'], case['n']
    solves = _solves(case)
    data = [_inputs(case, s, seed + 1000 * i) for i, s in enumerate(solves)]
    if kind == 'fft':
        dr = _grid(solves[0])[2]
        psi = [p.to(torch.complex128) for p in data[0][0]]
        return {'psik': _fft(psi, dr), 'psi': psi}
    if kind == 'batch':
        return [_exact_steps(s, d[1], n)[0] for s, d in zip(solves, data)]
    s = solves[0]
    pk, pops = _exact_steps(s, data[0][1], n, kind in ('pops', 'prop_loop'))
    if kind in ('steps', 'loop'):
        return {'psik': pk}
    if kind == 'pops':
        return {'psik': pk, 'pops': pops}
    (x, y), (kx, ky), dr, dk = _grid(s)
    dv_r, dv_k = float(np.prod(dr)), float(np.prod(dk))
    psi = [torch.fft.ifft2(torch.fft.ifftshift(p)) * (2 * math.pi / dv_r)
           for p in pk]
    dens = [p.real**2 + p.imag**2 for p in psi]
    densk = [p.real**2 + p.imag**2 for p in pk]
    phase = [torch.where(d < d.max() * 1e-6, torch.zeros_like(d),
                         torch.angle(p)) for p, d in zip(psi, dens)]
    xm = torch.as_tensor(x, device='cuda')[None, :]
    ym = torch.as_tensor(y, device='cuda')[:, None]
    kxm = torch.as_tensor(kx, device='cuda')[None, :]
    kym = torch.as_tensor(ky, device='cuda')[:, None]
    coupled = s['omega'] is not None
    w = (kxm**2 + kym**2) / 2 + (s['kl'] * kxm if coupled else 0.0)
    pot = 0.5 * (xm**2 + (s['lam'] * ym)**2)
    if s['lattice']:
        pot = pot + 3.0 * torch.sin(0.9 * xm + 0.5 * ym)**2
    det = s['delta'] / 2 if coupled else 0.0
    g = s['g']
    e_kin = float(sum((w * d).sum() for d in densk)) * dv_k / dv_r
    e_pot = float(((pot + det) * dens[0] + (pot - det) * dens[1]).sum())
    e_int = float((g[0] * dens[0]**2 + g[1] * dens[1]**2
                   + g[2] * dens[0] * dens[1]).sum())
    e_cpl = float((psi[0].conj() * psi[1]).real.sum()) * (s['omega'] or 0.0)
    sep = 1 - float((dens[0] * dens[1]).sum() / torch.sqrt(
        (dens[0]**2).sum() * (dens[1]**2).sum()))
    return {'psi': psi, 'psik': pk, 'pops': pops,
            'energy': [e_kin + e_pot + e_int + e_cpl, e_kin, e_pot, e_int],
            'dens': dens, 'densk': densk, 'phase': phase, 'separation': sep}
