"""Increments set between steps (swm_gpu_set_field of G_u, G_v, G_eta) are
those the next steps weight, on every path."""
import numpy as np
import pytest

from harness import run_case, rel_l2
from swm_gb300.host import synthetic
from swm_gb300.model import GpuModel

pytestmark = pytest.mark.gpu

PAIRS = [('u', 'G_u'), ('v', 'G_v'), ('eta', 'G_eta')]


def model(path):
    case = synthetic.double_gyre((45, 37), biharmonic=False, nsteps=20)
    rng = np.random.default_rng(8)
    case['ic'] = {f: 0.1 * rng.standard_normal(case['H'].shape) for f in ('u', 'v', 'eta')}
    g = GpuModel(path)
    run_case(case, g, nsteps=20, with_diag=False)
    return case, g


@pytest.mark.parametrize('path', ['plain_fp64', 'fused_fp64', 'fused_fp32c'])
def test_increment_is_kept_and_used(path):
    """Read back, the increment is what was set (binary32 on the pair path);
    the next step differs from an untouched model's by dt ab1 (set - before)
    over the damping factor, ab1 = -16/12, to the paths' 1e-5."""
    case, g = model(path)
    _, h = model(path)
    want = {}
    for k, (f, G) in enumerate(PAIRS):
        before = g.field(G)
        new = (before + np.abs(before).max() * np.random.default_rng(k).standard_normal(before.shape)) * g.ocean(f)
        if path == 'fused_fp32c':
            new = new.astype(np.float32).astype(np.float64)
        g.set_field(G, new)
        assert np.array_equal(g.field(G), new), G
        want[f] = case['config']['dt'] * (-16.0 / 12.0) * (new - before) / g.field('impl_' + f)
    for m in (g, h):
        m.step(21)
        m.advance(21)
    for f, _ in PAIRS:
        got = g.field(f) - h.field(f)
        assert np.abs(want[f]).max() > 0 and rel_l2(got, want[f], g.ocean(f).astype(bool)) <= 1e-5, f
    g.close()
    h.close()


@pytest.mark.parametrize('field', ['G_u', 'G_eta'])
def test_setting_one_increment_keeps_the_rest(field):
    """On the pair path, an increment set to the value it has changes nothing:
    the steps that follow are an untouched model's, bit for bit."""
    _, g = model('fused_fp32c')
    _, h = model('fused_fp32c')
    g.set_field(field, g.field(field))
    for m in (g, h):
        m.run(20, 12)
    for f, _ in PAIRS:
        assert np.array_equal(g.field(f), h.field(f)), f
    g.close()
    h.close()
