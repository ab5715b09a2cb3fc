"""The FP64 step kernels against the FP64 oracle at the edges of their blocks
(32 x 8 points), with every term that has its own branch: mixing, drag,
damping factors that are one, uniform or vary, wind on either component, land.
plain_fp64 bit for bit, fused_fp64 to 1e-11 relative L2 after 40 steps (its
stated tolerance), and a state set between two steps taken up by the next.
"""
import numpy as np
import pytest

from harness import run_case, rel_l2
from oracle import OracleBackend
from swm_gb300.host import synthetic
from swm_gb300.model import GpuModel

pytestmark = pytest.mark.gpu

STEPS = 40
SIZES = [(30, 6), (31, 7), (32, 8), (63, 15), (64, 17), (97, 23)]   # cells: one point more each way


def damping(term, value, varying):
    return dict(term=term, type=1 if varying else 0, value=value, sl_length=0.02, sl_cutoff=15.0, loc=15,
                file_data=None)


def make(shape, physics):
    if physics == 'linear':
        return synthetic.linear_rg(*shape, nsteps=STEPS)
    case = synthetic.double_gyre(shape, biharmonic=physics == 'biharmonic', nsteps=STEPS)
    rng = np.random.default_rng(shape[0])
    H = case['H']
    case['ic'] = {f: 0.1 * rng.standard_normal(H.shape) for f in ('u', 'v', 'eta')}
    if physics == 'drag':
        case['config'].update(quadratic_friction=1)
        case['damping'] = [damping(0, 1e-5, True), damping(1, 1e-6, False), damping(3, 2e-6, False),
                           damping(4, 2e-6, False)]
    if physics == 'winds':   # a second, meridional stress, scaled
        case['config'].update(lateral_mixing=0, tau_scale=0.7)
        case['streams'].append(dict(case['streams'][0], comp=1))
        case['damping'] = [damping(2, 1e-6, True)]
    return case


@pytest.mark.parametrize('path', ['plain_fp64', 'fused_fp64'])
@pytest.mark.parametrize('physics', ['linear', 'laplacian', 'biharmonic', 'drag', 'winds'])
def test_block_edges(path, physics):
    for shape in SIZES:
        case = make(shape, physics)
        o, g = OracleBackend(), GpuModel(path)
        run_case(case, o, nsteps=STEPS, with_diag=False)
        run_case(case, g, nsteps=STEPS, with_diag=False)
        for f in ('u', 'v', 'eta'):
            a, b = g.field(f), o.field(f)
            if path == 'plain_fp64':
                assert np.array_equal(a, b), (shape, f)
            else:
                err = rel_l2(a, b, o.ocean(f).astype(bool))
                assert err <= 1e-11, (shape, f, err)
        g.close()


@pytest.mark.parametrize('physics', ['laplacian', 'biharmonic'])
def test_state_set_between_steps(physics):
    """plain_fp64 keeps the stress of the advanced state for the next step:
    u and v set in between are what that step mixes, in single steps and in
    replayed ones."""
    case = make((45, 37), physics)
    rng = np.random.default_rng(5)
    new = {f: 0.1 * rng.standard_normal(case['H'].shape) for f in ('u', 'v')}
    runs = []
    for replay in (True, False):
        g = GpuModel('plain_fp64')
        run_case(case, g, nsteps=8, with_diag=False)
        if replay:
            g.run(8, 24)
        else:
            for itt in range(9, 33):
                g.step(itt)
                g.advance(itt)
        for f, x in new.items():
            g.set_field(f, x * g.ocean(f))
        if replay:
            g.run(32, 24)
        else:
            for itt in range(33, 57):
                g.step(itt)
                if itt == 33:
                    mixed = g.field('latmix_u')
                g.advance(itt)
        runs.append([g.field(f) for f in ('u', 'v', 'eta')])
        g.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
    # the mixing of step 33 is that of the new state, not of the advanced one
    h = GpuModel('plain_fp64')
    run_case(dict(case, ic={**new, 'eta': case['ic']['eta']}), h, nsteps=1, with_diag=False)
    scale = np.abs(h.field('latmix_u')).max()
    assert np.abs(mixed - h.field('latmix_u')).max() < 0.2 * scale
    h.close()


def test_state_set_on_the_pair_path():
    """A field set on fused_fp32c between two steps changes that field alone:
    the run that follows is fused_fp64's with the same field set, to the path's
    stated 1e-5 (fields not read back before are not lost).  Both form every
    diagnostic from the state they step; plain_fp64 keeps those of its last
    advance, as the reference's arrays do."""
    case = make((45, 37), 'biharmonic')
    new = 0.1 * np.random.default_rng(5).standard_normal(case['H'].shape)
    out = []
    for path in ('fused_fp64', 'fused_fp32c'):
        g = GpuModel(path)
        run_case(case, g, nsteps=20, with_diag=False)
        g.set_field('u', new * g.ocean('u'))
        assert np.allclose(g.field('u'), new * g.ocean('u'), rtol=1e-12, atol=0)
        g.run(20, 20)
        out.append({f: g.field(f) for f in ('u', 'v', 'eta')} | {'m': {f: g.ocean(f) for f in ('u', 'v', 'eta')}})
        g.close()
    for f in ('u', 'v', 'eta'):
        err = rel_l2(out[1][f], out[0][f], out[0]['m'][f].astype(bool))
        assert err <= 1e-5, (f, err)


@pytest.mark.parametrize('flux', [0, 1])
@pytest.mark.parametrize('shape', [(31, 7), (40, 24), (65, 33)])
def test_tracer_steps_replayed(shape, flux):
    """Three FP64 tracers in an evolving flow: replayed steps equal single
    steps bit for bit, also after a tracer is added to a model whose steps
    were captured without it, and both equal the oracle."""
    case = make(shape, 'laplacian')
    case['config'].update(tracer=1, tracer_flux=flux, tracer_nan_guard=1)
    rng = np.random.default_rng(shape[1])
    case['tracers'] = [dict(varid='C%d' % t, kappa_h=50.0, cons=[0.0, 1e-6, 0.0][t], gamma_c=1e-7 * t,
                            field_C=rng.random(case['H'].shape), field_C0=rng.random(case['H'].shape),
                            field_gamma_C=None, field_cons=None) for t in range(3)]
    o = OracleBackend(tracer_nan_guard=True)
    run_case(case, o, nsteps=STEPS, with_diag=False)
    single = GpuModel('plain_fp64', tracer_nan_guard=True)
    run_case(case, single, nsteps=STEPS, with_diag=False)
    replayed = GpuModel('plain_fp64', tracer_nan_guard=True)
    run_case(case, replayed, nsteps=0, with_diag=False)
    replayed.run(0, STEPS)
    for t in range(3):
        for f in ('CH', 'C', 'uhc', 'vhc', 'diff'):
            assert np.array_equal(replayed.tracer_field(t, f), single.tracer_field(t, f)), (t, f)
        assert np.array_equal(single.tracer_field(t, 'CH'), o.tracer_field(t, 'CH0')), t
    late = []
    for replay in (True, False):
        g = GpuModel('plain_fp64', tracer_nan_guard=True)
        run_case(dict(case, tracers=[]), g, nsteps=0, with_diag=False)
        g.run(0, 20)
        g.add_tracer(case['tracers'][1])
        g.tracer_init()
        if replay:
            g.run(20, 20)
        else:
            for itt in range(21, 41):
                g.step(itt)
                g.advance(itt)
        late.append(g.tracer_field(0, 'CH'))
    assert np.array_equal(*late)


@pytest.mark.parametrize('shape', [(77, 41), (511, 255), (512, 256)])   # either side of a megabyte
def test_async_fields_pinned_and_pageable(shape):
    """A field of the pair state read into a pinned array (a small one is
    written there by the joining kernel), a pageable one (copied) and by the
    blocking call is the same, of the state when it was asked for."""
    import torch
    case = make(shape, 'laplacian')
    g = GpuModel('fused_fp32c')
    run_case(case, g, nsteps=10, with_diag=False)
    now = {f: g.field(f) for f in ('u', 'v', 'eta', 'G_u', 'D')}
    shape = now['u'].shape
    got = {}
    for f in now:
        pinned, plain = torch.empty(shape, dtype=torch.float64).pin_memory().numpy(), np.empty(shape)
        got[f] = (pinned, plain, g.field_async(f, pinned), g.field_async(f, plain))
    g.run(10, 12)
    for f, (pinned, plain, t, s) in got.items():
        g.wait(t)
        g.wait(s)
        assert np.array_equal(pinned, now[f]) and np.array_equal(plain, now[f]), f
    g.close()


@pytest.mark.parametrize('field', ['H_u', 'H_v', 'H', 'pot', 'impl_u'])
@pytest.mark.parametrize('depths', ['flat', 'varied'])
def test_linear_mode_grid_fields_set_between_steps(field, depths):
    """The linear modes divide by thicknesses that do not change and keep their
    potential vorticity: a grid field set between steps reaches the steps that
    follow, replayed or single, as it does in a model that has always formed
    everything again (set anew before every step)."""
    case = synthetic.linear_rg(40, 24, nsteps=STEPS)
    if depths == 'varied':
        case['config']['H_overwrite'] = 0.0
        case['H'] = np.where(case['H'] > 0, 150.0 + 100.0 * np.random.default_rng(2).random(case['H'].shape), 0.0)
    runs = []
    for mode in ('replayed', 'single', 'anew'):
        g = GpuModel('plain_fp64')
        run_case(case, g, nsteps=0, with_diag=False)
        g.run(0, 20)
        new = g.field(field)
        new[5:12, 6:30] *= 1.25
        g.set_field(field, new)
        if mode == 'replayed':
            g.run(20, 20)
        else:
            for itt in range(21, 41):
                if mode == 'anew' and itt > 21:   # the same values: only what is kept is dropped
                    g.set_field('gamma_lin_u', g.field('gamma_lin_u'))
                g.step(itt)
                g.advance(itt)
        runs.append([g.field(f) for f in ('u', 'v', 'eta', 'pot')])
        g.close()
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            assert np.array_equal(a, b)
