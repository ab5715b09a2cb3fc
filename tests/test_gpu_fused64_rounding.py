"""fused_fp64 divides: by a uniform damping factor, by the thickness (wind
stress, potential vorticity).  Each quotient is compared at points where
everything else in it is exact, or where the rest is far smaller."""
import numpy as np
import pytest

from harness import rel_l2, run_case
from swm_gb300.host import synthetic
from swm_gb300.model import GpuModel

pytestmark = pytest.mark.gpu


def one_step(case, path='fused_fp64'):
    g = GpuModel(path)
    run_case(case, g, nsteps=1, with_diag=False)
    return g


def uniform_damping(gamma):
    return [dict(term=t, type=0, value=gamma, sl_length=1.0, sl_cutoff=15.0, loc=0, file_data=None) for t in (0, 1)]


@pytest.mark.parametrize('strength', [1e-3, 1.0, 1e6, 1e12])
def test_uniform_damping_keeps_its_digits(strength):
    """u / (1 + dt gamma), dt gamma = strength, against plain_fp64.  A step of
    1e-3 s changes u (0.5 to 1.5 m/s) by less than 1e-6, so that the tendency's
    roundings are below 1e-6 x 64 x 2^-53 of it: the two sums are at most one
    ulp apart and each quotient half an ulp off, 2 ulps or 4 x 2^-53 together."""
    dt = 1e-3
    case = synthetic.double_gyre((45, 37), biharmonic=False, dt=dt, nsteps=1)
    case['damping'] = uniform_damping(strength / dt)
    rng = np.random.default_rng(4)
    H = case['H']
    case['ic'] = {f: rng.choice([-1.0, 1.0], H.shape) * (0.5 + rng.random(H.shape)) for f in ('u', 'v')}
    a, b = one_step(case), one_step(case, 'plain_fp64')
    for f in ('u', 'v'):
        x, y, m = a.field(f), b.field(f), a.ocean(f).astype(bool)
        assert (y[m] != 0).all()
        assert (np.abs(x - y)[m] <= 4 * 2.0 ** -53 * np.abs(y)[m]).all()
    a.close()
    b.close()


def test_infinite_velocity_under_uniform_damping():
    """An infinite velocity stays infinite under a finite damping factor: u holds
    its infinity where plain_fp64's does, and no NaN."""
    case = synthetic.linear_rg(40, 24, nsteps=1)
    case['config'].update(lateral_mixing=0)
    case['ic'] = {f: np.zeros_like(case['H']) for f in ('u', 'v', 'eta')}
    case['ic']['u'][6, 20] = np.inf
    a, b = one_step(case), one_step(case, 'plain_fp64')
    x, y = a.field('u'), b.field('u')
    assert np.isinf(y[6, 20]) and not np.isnan(y).any()
    assert np.array_equal(np.isinf(x), np.isinf(y)) and not np.isnan(x).any()
    a.close()
    b.close()


def wet_surroundings(H, r=3):
    """Points whose neighbours up to r cells away are all ocean."""
    m = H > 0
    for axis in (0, 1):
        m = np.logical_and.reduce([np.roll(m, s, axis) for s in range(-r, r + 1)])
    return m


def integer_depths(shape):
    """A box of depths H that are whole multiples of 32 m: their means at the
    eta points (D) and the means of two and of four of those are exact."""
    H = 32.0 * np.random.default_rng(6).integers(5, 50, shape)
    H[:, 0] = H[:, -1] = H[0] = H[-1] = 0.0
    return H


def west(a):
    return np.roll(a, 1, 1)


def south(a):
    return np.roll(a, 1, 0)


def north(a):
    return np.roll(a, -1, 0)


def test_wind_over_thickness_is_the_quotient():
    """From rest, the tendency of u is tau / rho0 over the thickness: the
    quotient of the two, correctly rounded (rho0 is a power of two)."""
    case = synthetic.double_gyre((65, 49), biharmonic=False, nsteps=1)
    case['config'].update(lateral_mixing=0)
    case['H'] = integer_depths(case['H'].shape)
    case['damping'] = []
    g = one_step(case)
    m = wet_surroundings(case['H'])
    D = g.field('D')
    want = case['streams'][0]['rec1'][0] / case['config']['RHO0'] / np.where(m, 0.5 * (D + west(D)), 1.0)
    assert m.sum() > 1000 and np.array_equal(g.field('G_u')[m], want[m])
    g.close()


def test_potential_vorticity_is_the_quotient():
    """Linear, u = eta = 0, v a whole number: the tendency of u is
    (f/D + f/D) / 2 times the mean mass flux.  With f over 8 the quotients are
    one rounding each, their sum one and its product with the (whole) sum of
    four mass fluxes one."""
    case = synthetic.linear_rg(64, 48, nsteps=1)
    H = case['H'] = integer_depths(case['H'].shape)
    case['config'].update(lateral_mixing=0, H_overwrite=0.0)
    case['damping'] = []
    case['ic'] = {'v': np.random.default_rng(7).integers(-3, 4, H.shape).astype(float)}
    g = one_step(case)
    D, v = g.field('D'), case['ic']['v'] * g.ocean('v')
    Dh = 0.25 * ((D + west(D)) + (south(D) + south(west(D))))
    pot = (g.lat('f_H') / 8)[:, None] / np.where(Dh > 0, Dh, 1.0)
    mv = 0.5 * (D + south(D)) * v
    want = (north(pot) + pot) * ((north(mv) + west(mv)) + (north(west(mv)) + mv))
    m = wet_surroundings(H)
    assert m.sum() > 1000 and np.array_equal(g.field('G_u')[m], want[m])
    g.close()


@pytest.mark.parametrize('flow,tendency', [('u', 'G_v'), ('v', 'G_eta')])
def test_uniform_flow_differences_cancel(flow, tendency):
    """A uniform flow of 1 m/s over 512 m without rotation: what is left of
    divergence and vorticity is the change of cos(lat) from row to row, whose
    products and differences are exact.  At most four roundings follow on
    fused_fp64 and three on plain_fp64 (powers of two aside), each 2^-53."""
    case = synthetic.double_gyre((45, 37), biharmonic=False, nsteps=1)
    case['config'].update(lateral_mixing=0, OMEGA=0.0)
    case['H'] = np.where(np.pad(np.ones((36, 44)), 1) > 0, 512.0, 0.0)
    case['damping'], case['streams'] = [], []
    case['ic'] = {flow: np.ones_like(case['H'])}
    a, b = one_step(case), one_step(case, 'plain_fp64')
    m = wet_surroundings(case['H'])
    x, y = a.field(tendency)[m], b.field(tendency)[m]
    assert m.sum() > 500 and (y != 0).mean() > 0.9   # (0 where two rows are as far from the equator)
    assert (np.abs(x - y) <= 8 * 2.0 ** -53 * np.abs(y)).all()
    a.close()
    b.close()


@pytest.mark.parametrize('physics', ['laplacian', 'biharmonic'])
@pytest.mark.parametrize('shape', [(31, 7), (32, 8), (97, 23)])
def test_forty_steps(shape, physics):
    """Relative L2 difference from plain_fp64 after 40 steps from a random
    state: below 40 steps x 100 roundings x 2^-53 = 4.4e-13."""
    case = synthetic.double_gyre(shape, biharmonic=physics == 'biharmonic', nsteps=40)
    rng = np.random.default_rng(shape[0])
    case['ic'] = {f: 0.1 * rng.standard_normal(case['H'].shape) for f in ('u', 'v', 'eta')}
    a, b = GpuModel('fused_fp64'), GpuModel('plain_fp64')
    for g in (a, b):
        run_case(case, g, nsteps=40, with_diag=False)
    for f in ('u', 'v', 'eta'):
        assert rel_l2(a.field(f), b.field(f), a.ocean(f).astype(bool)) <= 4.4e-13, f
    a.close()
    b.close()
