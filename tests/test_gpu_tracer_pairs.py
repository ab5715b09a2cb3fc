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
