"""The complex128 passes in 64-bit fixed point: the sizes, scales and values
where a line's exponent, headroom or series could go wrong, against NumPy
transforms and the complex128 oracle.

Bounds: a transform's error is at most crest * sqrt(N) * 2^-60 per axis
(crest: largest value over rms of a line), below 2e-15 for random lines of up
to 4096 points and 8e-15 for a single peak; steps keep the 1e-10 of the
complex128 parity tests, here tightened to 1e-12 over a few steps.
"""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import OracleInputs, OraclePropagator

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def tp():
    assert torch.cuda.is_available(), 'these tests need a CUDA device'
    from spinor_gpe.pspinor import tensor_propagator
    return tensor_propagator


@pytest.mark.parametrize('scale', [1.0, 1e-250, 1e250])
@pytest.mark.parametrize('shape', [(32, 32), (64, 4096), (4096, 64), (192, 768), (384, 512), (128, 2048)])
def test_transforms_at_any_scale(shape, scale):
    from spinor_gpe.pspinor import tensor_tools as ttools
    rng = np.random.default_rng(sum(shape))
    psi = [rng.standard_normal(shape) + 1j * rng.standard_normal(shape) for _ in range(2)]
    psi[1] *= 1e-12                     # each line has its own exponent
    dev = [torch.as_tensor(p * scale, device='cuda') for p in psi]
    got = ttools.fft_2d(dev, (1.0, 2 * np.pi))
    back = ttools.ifft_2d(got, (1.0, 2 * np.pi))
    for g, b, p in zip(got, back, psi):
        ref = np.fft.fftshift(np.fft.fftn(p))
        assert rel_l2(g.cpu().numpy() / scale, ref) <= 2e-15
        assert rel_l2(b.cpu().numpy() / scale, p) <= 2e-15


@pytest.mark.parametrize('shape', [(32, 64), (4096, 32), (768, 192)])
def test_transforms_of_peaks_zeros_and_nan(shape):
    from spinor_gpe.pspinor import tensor_tools as ttools
    peak = np.zeros(shape, dtype=complex)
    peak[shape[0] // 3, 5] = 1.0 - 2.0j
    zero = torch.zeros(shape, dtype=torch.complex128, device='cuda')
    got = ttools.fft_2d([torch.as_tensor(peak, device='cuda'), zero], (1.0, 2 * np.pi))
    ref = np.fft.fftshift(np.fft.fftn(peak))
    assert rel_l2(got[0].cpu().numpy(), ref) <= 8e-15
    assert not got[1].any()
    for bad in (np.nan, np.inf):
        peak[1, 1] = bad
        got = ttools.fft_2d([torch.as_tensor(peak, device='cuda'), zero], (1.0, 2 * np.pi))
        assert not torch.isfinite(torch.view_as_real(got[0])).any()
        assert not got[1].any()


# a line whose values all add up in one bin, with parts that fill their
# exponent (1.9 +- 1.9i in four domains of constant phase): the largest sums a
# transform can meet
@pytest.mark.parametrize('side', [32, 64, 128, 192, 256, 384, 512, 768, 1024, 2048, 4096])
def test_transforms_of_full_lines(side):
    from spinor_gpe.pspinor import tensor_tools as ttools
    line = (1.9 + 1.9j) * 1j**(np.arange(side) * 4 // side)
    for shape, field in (((32, side), np.ones((32, 1)) * line), ((side, 32), line[:, None] * np.ones(32))):
        psi = [field, np.roll(field, 3, (0, 1)).conj()]
        got = ttools.fft_2d([torch.as_tensor(p, device='cuda') for p in psi], (1.0, 2 * np.pi))
        back = ttools.ifft_2d([torch.as_tensor(np.fft.fftshift(p), device='cuda') for p in psi], (1.0, 2 * np.pi))
        for g, b, p in zip(got, back, psi):
            assert rel_l2(g.cpu().numpy(), np.fft.fftshift(np.fft.fftn(p))) <= 8e-15
            assert rel_l2(b.cpu().numpy(), np.fft.ifftn(p)) <= 8e-15


# steps of states that are such lines in k space (flat spectra, whose rows add
# up in one point): a point in real space, and the four domains along kx and ky
@pytest.mark.parametrize('state', ['point', 'domains'])
@pytest.mark.parametrize('nx,ny', [(64, 512), (512, 64), (32, 32), (1024, 128), (64, 1024)])
def test_steps_of_full_lines_match_oracle(tp, tmp_path, nx, ny, state):
    ps = _problem(tmp_path, nx, ny, (1000.0, 995.0, 990.0), 0.7)
    ps.g_sc = {'uu': 1e-3, 'dd': 1e-3, 'ud': 1e-3}
    if state == 'point':
        psi = np.zeros((ny, nx), dtype=complex)
        psi[ny // 2, nx // 2] = 1.0
        psi = np.fft.fftshift(np.fft.fft2(psi))
    else:
        psi = (1.9 + 1.9j) * 1j**(np.arange(nx) * 4 // nx) * 1j**(np.arange(ny) * 4 // ny)[:, None]
    ps.psik = [psi, 0.9 * psi.conj()]
    ref, _ = _oracle(ps, 1e-3, 'real', 2)
    prop = tp.TensorPropagator(ps, 1e-3, 2, 'cuda', time='real', dtype=128)
    prop.full_steps(2)
    got = np.array([t.cpu().numpy() for t in prop.psik])
    assert rel_l2(got, ref) <= 1e-12


def _problem(tmp_path, nx, ny, g, omega, dtype=np.complex128, **kw):
    from spinor_gpe import workloads
    from spinor_gpe.pspinor import pspinor as spin
    from spinor_gpe.pspinor import tensor_tools as ttools
    return workloads.build(spin.PSpinor, ttools.fft_2d, str(tmp_path / 'p') + '/',
                           nx=nx, ny=ny, half_x=nx * 0.125 / 2, half_y=ny * 0.125 / 2,
                           g=g, omega=omega, k_l=2.0, seed=11, **kw)


def _oracle(ps, dt, time, n):
    inp = OracleInputs(
        psik=[np.asarray(p) for p in ps.psik],
        kin_eng_spin=[np.asarray(k) for k in ps.kin_eng_spin],
        pot_eng_spin=[np.asarray(v) for v in ps.pot_eng_spin],
        coupling=np.asarray(ps.coupling, dtype=np.float64),
        x_mesh=ps.space['x_mesh'], dr=ps.space['dr'],
        dv_r=float(ps.space['dv_r']), dv_k=float(ps.space['dv_k']),
        g_sc=dict(ps.g_sc), atom_num=float(ps.atom_num),
        kL_recoil=float(ps.kL_recoil), rot_coupling=bool(ps.rot_coupling),
        is_coupling=bool(ps.is_coupling))
    orc = OraclePropagator(inp, dt, time, 128)
    pops = orc.run(n)
    return orc.psik_numpy(), pops


# small steps (series), steps whose phases leave the series (dt = 0.2: phases
# of several radians at the centre, small ones at the rim), both time
# directions, with and without coupling, an attractive gas (growing factors)
@pytest.mark.parametrize('time,dt,g,omega', [
    ('real', 1e-3, (1000.0, 995.0, 990.0), 1.0),
    ('real', 0.2, (1000.0, 995.0, 990.0), 1.0),
    ('real', 0.2, (1000.0, 995.0, 990.0), None),
    ('imag', 0.02, (1000.0, 995.0, 990.0), 1.0),
    ('imag', 0.3, (1000.0, 995.0, 990.0), None),
    ('imag', 0.05, (-60.0, 995.0, 300.0), 0.7),
    ('real', 0.05, (0.0, 0.0, 0.0), 0.7),
])
@pytest.mark.parametrize('nx,ny', [(64, 32), (192, 128), (512, 256)])
def test_steps_match_oracle(tp, tmp_path, nx, ny, time, dt, g, omega):
    if (nx, ny, dt) == (64, 32, 0.2):
        # the gas overfills this box: a 1e-15 change of the initial state
        # moves the oracle's own result by 3e-11 over these three steps, so
        # it says nothing about the kernels
        pytest.skip('ill-conditioned')
    ps = _problem(tmp_path, nx, ny, (1000.0, 995.0, 990.0), omega, delta=0.3 if omega else 0.0)
    ps.g_sc = dict(zip(('uu', 'dd', 'ud'), g))
    ref, ref_pops = _oracle(ps, dt, time, 3)
    prop = tp.TensorPropagator(ps, dt, 3, 'cuda', time=time, dtype=128)
    pops = torch.empty((3, 2), dtype=torch.float64, device='cuda')
    prop.full_steps(3, pops)
    got = np.array([t.cpu().numpy() for t in prop.psik])
    assert rel_l2(got, ref) <= 1e-12
    np.testing.assert_allclose(pops.cpu().numpy(), ref_pops, rtol=1e-12, atol=1e-13)


# one step on either side of the longest that runs in fixed point: 1/4 rad (or
# e-folding) per interaction factor at the mean density, here 3.016 dt
@pytest.mark.parametrize('time', ['real', 'imag'])
@pytest.mark.parametrize('dt', [0.01, 0.04, 0.0796, 0.0862, 0.3])
def test_longest_steps_match_oracle(tp, tmp_path, time, dt):
    ps = _problem(tmp_path, 64, 64, (1000.0, 995.0, 990.0), 0.7, delta=0.3)
    ref, _ = _oracle(ps, dt, time, 1)
    prop = tp.TensorPropagator(ps, dt, 1, 'cuda', time=time, dtype=128)
    prop.full_steps(1)
    got = np.array([t.cpu().numpy() for t in prop.psik])
    assert rel_l2(got, ref) <= 1e-12


@pytest.mark.parametrize('amp', [1e-9, 0.0])
def test_minority_component_keeps_its_precision(tp, tmp_path, amp):
    ps = _problem(tmp_path, 128, 64, (1000.0, 995.0, 990.0), None)
    ps.psik = [ps.psik[0], ps.psik[1] * amp]
    ref, _ = _oracle(ps, 1e-2, 'real', 3)
    prop = tp.TensorPropagator(ps, 1e-2, 3, 'cuda', time='real', dtype=128)
    prop.full_steps(3)
    got = np.array([t.cpu().numpy() for t in prop.psik])
    assert rel_l2(got[0], ref[0]) <= 1e-12
    if amp:
        assert rel_l2(got[1], ref[1]) <= 1e-12
    else:
        assert not got[1].any()


# A component of 10^-k of the other's amplitude under a coupling, down to one
# that the coupling alone fills, and a matrix whose rows differ (a detuning of
# 500 damps one component by e^-10 in an imaginary step).  Each component's own
# error: the FP64 oracle's is 1e-15 to 2e-15 of a component over three steps,
# the bound five times that.
@pytest.mark.parametrize('time,omega,delta', [
    ('real', 1.0, 0.3), ('real', 1e-3, 0.3), ('real', 1e-6, 0.0), ('imag', 1e-3, 0.3), ('imag', 0.5, 500.0)])
@pytest.mark.parametrize('amp', [(1.0, 1e-3), (1.0, 1e-6), (1e-6, 1.0), (1.0, 1e-9), (1.0, 0.0)])
@pytest.mark.parametrize('nx,ny,n', [(64, 64, 1), (128, 64, 3), (512, 32, 3), (192, 384, 3), (2048, 32, 2)])
def test_coupled_minority_component_keeps_its_precision(tp, tmp_path, nx, ny, n, amp, time, omega, delta):
    ps = _problem(tmp_path, nx, ny, (1000.0, 995.0, 990.0), omega, delta=delta)
    ps.psik = [p * a for p, a in zip(ps.psik, amp)]
    dt = 1e-3 if time == 'real' else 0.02
    ref, _ = _oracle(ps, dt, time, n)
    prop = tp.TensorPropagator(ps, dt, n, 'cuda', time=time, dtype=128)
    prop.full_steps(n)
    for got, want in zip(prop.psik, ref):
        assert rel_l2(got.cpu().numpy(), want) <= 1e-14


# populations of a minority: each to its own 1e-13 (they are sums of squares
# that the oracle has to 1e-15)
@pytest.mark.parametrize('amp', [1e-3, 1e-6, 1e-9])
@pytest.mark.parametrize('omega', [None, 1e-4])
@pytest.mark.parametrize('nx,ny', [(64, 64), (512, 128), (2048, 32)])
def test_population_of_a_minority(tp, tmp_path, nx, ny, omega, amp):
    ps = _problem(tmp_path, nx, ny, (1000.0, 995.0, 990.0), omega)
    ps.psik = [ps.psik[0] * amp, ps.psik[1]]
    _, ref = _oracle(ps, 1e-3, 'real', 4)
    prop = tp.TensorPropagator(ps, 1e-3, 4, 'cuda', time='real', dtype=128)
    pops = torch.empty((4, 2), dtype=torch.float64, device='cuda')
    prop.full_steps(4, pops)
    prop.psik
    np.testing.assert_allclose(pops.cpu().numpy(), ref, rtol=1e-13)


# states without a norm: empty, or so small that every |psi|^2 underflows; and
# one whose norm is subnormal, which still propagates like its multiple (the
# subnormal sums carry 40 bits and more)
@pytest.mark.parametrize('nx', [64, 512, 2048])
@pytest.mark.parametrize('omega', [None, 1.0])
def test_state_without_a_norm_stays_visible(tp, tmp_path, nx, omega):
    ps = _problem(tmp_path, nx, 64, (1000.0, 995.0, 990.0), omega)
    prop = tp.TensorPropagator(ps, 1e-3, 3, 'cuda', time='real', dtype=128)
    psik = [p.clone() for p in prop.psik]
    for scale in (0.0, 1e-200):
        prop.psik = [p * scale for p in psik]
        pops = torch.zeros((3, 2), dtype=torch.float64, device='cuda')
        prop.full_steps(3, pops)
        for p in prop.psik:
            assert not torch.isfinite(torch.view_as_real(p)).any()
        assert not torch.isfinite(pops).any()
    got = []
    for scale in (1.0, 1e-155):
        prop.psik = [p * scale for p in psik]
        prop.full_steps(3)
        got.append(np.array([t.cpu().numpy() for t in prop.psik]))
    assert rel_l2(got[1], got[0]) <= 1e-10


def test_bad_state_stays_visible(tp, tmp_path):
    ps = _problem(tmp_path, 64, 64, (1000.0, 995.0, 990.0), 1.0)
    prop = tp.TensorPropagator(ps, 1e-3, 3, 'cuda', time='real', dtype=128)
    psik = [p.clone() for p in prop.psik]
    psik[0][3, 7] = float('nan')
    prop.psik = psik
    prop.full_steps(3)
    for p in prop.psik:
        assert not torch.isfinite(torch.view_as_real(p)).any()


# steps with populations: eager ones, the graphs of long steps (made within the
# first call) and those made after 128 steps all give the same bits
@pytest.mark.parametrize('dtype', [64, 128, 'double-float'])
@pytest.mark.parametrize('nx,ny', [(64, 64), (512, 256)])
def test_population_graphs_match_eager_steps(tp, tmp_path, monkeypatch, dtype, nx, ny):
    ps = _problem(tmp_path, nx, ny, (1000.0, 995.0, 990.0), 1.0)
    props = [tp.TensorPropagator(ps, 1e-3, 20, 'cuda', time='real', dtype=dtype)]
    monkeypatch.setenv('SGPE_DISABLE_GRAPHS', '1')
    props.append(tp.TensorPropagator(ps, 1e-3, 20, 'cuda', time='real', dtype=dtype))
    for n in (20, 2, 110, 9, 21):
        out = []
        for p in props:
            pops = torch.full((n, 2), -1.0, dtype=torch.float64, device='cuda')
            p.full_steps(n, pops)
            out.append([t.cpu().numpy() for t in p.psik] + [pops.cpu().numpy()])
        for a, b in zip(*out):
            np.testing.assert_array_equal(a, b)


# a stream that the caller captures gets the launches of the steps
@pytest.mark.parametrize('nx,ny', [(64, 64), (512, 256)])
def test_populations_on_a_captured_stream(tp, tmp_path, nx, ny):
    ps = _problem(tmp_path, nx, ny, (1000.0, 995.0, 990.0), 1.0)
    a, b = (tp.TensorPropagator(ps, 1e-3, 20, 'cuda', time='real', dtype=128) for _ in range(2))
    out = []
    for p in (a, b):
        pops = torch.zeros((12, 2), dtype=torch.float64, device='cuda')
        p.full_steps(12, pops)     # makes the merged tables
        p.full_steps(1)
        pops.zero_()
        if p is a:
            p.full_steps(12, pops)
        else:
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                p.full_steps(12, pops)
            graph.replay()
        out.append([t.cpu().numpy() for t in p.psik] + [pops.cpu().numpy()])
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)


# solves of one size stepped by the grouped fixed-point kernels, next to ones
# that keep FP64 passes (long steps; an attractive gas, whose rows alone do) and
# one that new physics moves across that line between two calls
@pytest.mark.parametrize('time', ['real', 'imag'])
@pytest.mark.parametrize('side,shape', [(32, 0), (64, 0), (64, 1), (128, 2), (192, 0), (256, 2)])
def test_grouped_batch_matches_solves_alone(tp, tmp_path, side, shape, time):
    from spinor_gpe.batch import PropagatorBatch
    g = (1000.0, 995.0, 990.0)
    dt = 1e-3 if time == 'real' else 0.02
    spins = [_problem(tmp_path / str(i), side, side, g, w) for i, w in enumerate((1.0, 0.5, None, 1.0, 0.7, 0.3))]
    spins[4].g_sc = dict(uu=-60.0, dd=995.0, ud=300.0)
    factor = [1.0, 1.1, 0.9, 1e4, 1.0, 1.0]    # member 3: long steps

    def scaled(p, f):
        p._plan.set_physics(*(f * p.g_sc[k] for k in ('uu', 'dd', 'ud')), float(p.atom_num),
                            float(p._space_np['dv_r']), float(p._space_np['dv_k']), p.is_coupling)

    def make():
        out = []
        for s, f in zip(spins, factor):
            p = tp.TensorPropagator(s, dt, 20, 'cuda', time=time, dtype=128)
            if shape:
                p.kernel_shapes = (shape, shape)
            scaled(p, f)
            out.append(p)
        return out
    alone, together = make(), make()
    batch = PropagatorBatch(together)
    for move in (None, (5, 1e4), (3, 1.0)):
        if move is not None:
            for props in (alone, together):
                scaled(props[move[0]], move[1])
        for p in alone:
            p.full_steps(11)
        batch.full_steps(11)
        for a, b in zip(alone, together):
            np.testing.assert_array_equal([t.cpu().numpy() for t in a.psik], [t.cpu().numpy() for t in b.psik])
    batch.close()
