"""A field set on plain_fp64 that nothing kept depends on costs no more than
its copy: the steps that follow launch what they launched before, and replay
the captured steps."""
import numpy as np
import pytest

from harness import run_case
from swm_gb300.host import synthetic
from swm_gb300.model import GpuModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('field', ['F_x', 'F_eta', 'D', 'mu', 'zeta', 'G_u', 'gamma_lin_u', 'u', 'eta'])
def test_nothing_is_formed_again(field):
    case = synthetic.linear_rg(40, 24, nsteps=100)
    case['config'].update(lateral_mixing=0)   # (the stress of a state that was set is formed again)
    g = GpuModel('plain_fp64')
    run_case(case, g, nsteps=0, with_diag=False)
    g.run(0, 20)
    g.synchronize()

    def launches(call):
        n = g.launch_count()
        call()
        return g.launch_count() - n

    def single(itt):
        g.step(itt)
        g.advance(itt)

    before = launches(lambda: single(21))
    g.set_field(field, g.field(field))
    assert launches(lambda: single(22)) == before
    # replayed: as many launches as steps, no kernel beside them
    g.run(22, 14)   # (up to the phase that the captured steps start from)
    before = launches(lambda: g.run(36, 24))
    g.set_field(field, g.field(field))
    assert launches(lambda: g.run(60, 24)) == before
    g.close()
