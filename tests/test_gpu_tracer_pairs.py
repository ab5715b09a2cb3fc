"""FP32 tracers: two share a launch in packed instructions, and windows that
are all ocean run a body without mask tests.  Neither changes a tracer's bits:
each tracer equals itself alone, in any company and order, at widths around
the 28-column strips and 32-lane warps, next to coasts and away from them.
"""
import numpy as np
import pytest

from harness import rel_l2, run_case
from oracle import OracleBackend
from swm_gb300.host import synthetic
from swm_gb300.model import GpuModel

pytestmark = pytest.mark.gpu

STEPS = 30


def model(case, picks):
    c = dict(case, tracers=[case['tracers'][t] for t in picks])
    g = GpuModel('fused_fp32c', tracer_nan_guard=True)
    run_case(c, g, nsteps=0, with_diag=False)
    g.run(0, STEPS)
    out = [g.tracer_field(q, 'CH') for q in range(len(picks))]
    g.close()
    return out


@pytest.mark.parametrize('flux', [0, 1])
@pytest.mark.parametrize('cells', [(27, 9), (28, 40), (55, 33), (57, 64), (84, 31), (120, 17)])
def test_company_does_not_matter(cells, flux):
    case = synthetic.double_gyre(cells, biharmonic=False, nsteps=STEPS)
    case['config'].update(tracer=1, tracer_flux=flux, tracer_nan_guard=1)
    rng = np.random.default_rng(cells[0])
    shape = case['H'].shape
    if cells[0] == 120:   # an island
        case['H'][7:10, 60:64] = 0.0
    case['ic'] = {f: 0.2 * rng.standard_normal(shape) for f in ('u', 'v')}
    case['tracers'] = [dict(varid='C%d' % t, kappa_h=(50.0, 5e3, 200.0)[t], cons=(0.0, 1e-6, 0.0)[t],
                            gamma_c=(0.0, 1e-7, 4e-7)[t], field_C=rng.random(shape), field_C0=rng.random(shape),
                            field_gamma_C=None, field_cons=None) for t in range(3)]
    alone = [model(case, [t])[0] for t in range(3)]
    for picks in ([0, 1], [1, 0], [0, 1, 2], [2, 2, 1, 0]):
        for t, got in zip(picks, model(case, picks)):
            assert np.array_equal(got, alone[t]), (picks, t)
    o = OracleBackend(tracer_nan_guard=True)
    run_case(case, o, nsteps=STEPS, with_diag=False)
    m = o.ocean('eta').astype(bool)
    for t in range(3):
        assert rel_l2(alone[t], o.tracer_field(t, 'CH0'), m) <= 1e-5


def test_rows_beyond_a_pole():
    """Rows whose cosine is negative (a grid that reaches beyond the poles):
    the upwind side is the velocity's, not the transport's.  One step against
    the oracle: binary32 rounding of values of order one and of an increment
    of order 1e-2, below 1e-6."""
    case = synthetic.double_gyre((40, 60), biharmonic=False, nsteps=1)
    # 3.4 degrees of a sphere of 85 km: 5 km cells, the smallest cosine above 1e-3
    case['config'].update(tracer=1, tracer_flux=1, tracer_nan_guard=1, A=85e3, lon_s=-67.0, lon_e=67.0,
                          lat_s=-101.0, lat_e=101.0)
    rng = np.random.default_rng(5)
    shape = case['H'].shape
    case['ic'] = {f: 0.2 * rng.standard_normal(shape) for f in ('u', 'v')}
    case['tracers'] = [dict(varid='C0', kappa_h=0.0, cons=0.0, gamma_c=0.0, field_C=rng.random(shape),
                            field_C0=rng.random(shape), field_gamma_C=None, field_cons=None)]
    out = []
    for b in (GpuModel('fused_fp32c', tracer_nan_guard=True), OracleBackend(tracer_nan_guard=True)):
        run_case(case, b, nsteps=1, with_diag=False)
        out.append(b)
    m = out[1].ocean('eta').astype(bool)
    want = out[1].tracer_field(0, 'CH0')
    assert rel_l2(out[0].tracer_field(0, 'CH'), want, m) <= 1e-6
    out[0].close()
