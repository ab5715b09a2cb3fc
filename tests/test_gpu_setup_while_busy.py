"""A model set up while another one's steps fill the GPU is the model that is
set up on an idle one: its fields' zeroing and uploads are ordered on its own
stream, with the kernels that read them."""
import threading

import numpy as np
import pytest

from harness import run_case
from swm_gb300.host import synthetic
from swm_gb300.model import GpuModel

pytestmark = pytest.mark.gpu

FIELDS = ('u', 'v', 'eta')


def busy(steps=1500):
    """A model with a few tenths of a second of queued steps."""
    g = GpuModel('fused_fp64')
    run_case(synthetic.double_gyre(1024), g, nsteps=0, with_diag=False)
    g.run(0, steps)
    return g


def case(shape=(300, 200)):
    c = synthetic.double_gyre(shape, biharmonic=False, nsteps=20)
    rng = np.random.default_rng(1)
    c['ic'] = {f: 0.1 * rng.standard_normal(c['H'].shape) for f in FIELDS}
    c['config'].update(tracer=1, tracer_nan_guard=1)
    c['tracers'] = [dict(varid='C', kappa_h=50.0, cons=0.0, gamma_c=1e-7, field_C=rng.random(c['H'].shape),
                         field_C0=rng.random(c['H'].shape), field_gamma_C=None, field_cons=None)]
    return c


def result(path, c):
    g = GpuModel(path, tracer_nan_guard=True)
    run_case(c, g, nsteps=0, with_diag=False)
    g.run(0, 20)
    out = [g.field(f) for f in FIELDS] + [g.tracer_field(0, 'CH'), g.integrals()]
    g.close()
    return out


@pytest.mark.parametrize('path', ['plain_fp64', 'fused_fp64', 'fused_fp32c'])
def test_setup_beside_running_steps(path):
    c = case()
    want = result(path, c)
    for _ in range(3):
        other = busy()
        got = result(path, c)
        other.close()
        for a, b in zip(got, want):
            assert np.isfinite(b).all() and np.array_equal(a, b)


def test_setup_from_several_threads():
    """Contexts created at once zero their fields on their own streams."""
    c = case((90, 70))
    want = result('plain_fp64', c)
    got = [None] * 6

    def work(k):
        got[k] = result('plain_fp64', c)

    for _ in range(3):
        threads = [threading.Thread(target=work, args=(k,)) for k in range(len(got))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for out in got:
            for a, b in zip(out, want):
                assert np.array_equal(a, b)
