"""The reference SOR with its cells on few blocks and its iterations in short
launches: several cells and several trips per thread, remainders of both, many
launches of odd length, and a launch that the GPU refuses because its blocks
do not fit at once.  Iterates equal the oracle's bit for bit."""
import numpy as np
import pytest

from harness import run_case
from oracle import OracleBackend
from swm_gb300.host import synthetic
from swm_gb300.model import GpuModel

pytestmark = pytest.mark.gpu


def problem(shape):
    case = synthetic.double_gyre(shape, biharmonic=False, nsteps=1)
    o = OracleBackend()
    run_case(case, o, nsteps=1, with_diag=False)
    o.sor_init()
    rng = np.random.default_rng(3)
    u, v = (rng.standard_normal(case['H'].shape) for _ in range(2))
    return case, o, o.divergence(u * o.ocean('u'), v * o.ocean('v'))


def gpu(case, monkeypatch, blocks, batch):
    for name, value in (('BLOCKS', blocks), ('BATCH', batch)):
        monkeypatch.setenv('SWM_GB300_SOR_' + name, str(value))
    g = GpuModel('plain_fp64')
    run_case(case, g, nsteps=0, with_diag=False)
    g.sor_init()
    return g


@pytest.mark.parametrize('shape', [(127, 64), (128, 65), (200, 100)])   # cells: 128, 129 and 201 points a row
def test_capped_solve(shape, monkeypatch):
    """A call that may not converge runs max_count iterations: the same
    iterate from every split."""
    case, o, B = problem(shape)
    chi0 = np.random.default_rng(1).standard_normal(B.shape) * o.ocean('eta')
    want, its, _ = o.sor_solve(B, chi0, 1e-40, False)
    assert its < 0
    for blocks, batch in ((1, 5000), (2, 7), (3, 64), (5, 1), (40, 333), (0, 17)):
        g = gpu(case, monkeypatch, blocks, batch)
        got, n, _ = g.sor_solve(B, chi0, 1e-40, False)
        assert n == its and np.array_equal(got, want), (blocks, batch)
        g.close()


@pytest.mark.parametrize('blocks,batch', [(1, 5), (3, 4), (0, 3)])
def test_converged_solve(blocks, batch, monkeypatch):
    """The stop test in any of the launches: the oracle's iteration (or the one
    next to it, where the order of the norm's sum decides) and its iterate."""
    case, o, B = problem((96, 41))
    want, its, norm = o.sor_solve(B, np.zeros_like(B), 1e-4, True)
    assert its > 2 * batch
    g = gpu(case, monkeypatch, blocks, batch)
    got, n, _ = g.sor_solve(B, np.zeros_like(B), 1e-4, True)
    assert abs(n - its) <= 1
    if n == its:
        assert np.array_equal(got, want)
    g.close()


def test_more_blocks_than_fit(monkeypatch):
    """Thousands of blocks cannot be on the GPU at once: the refused launch is
    made again with fewer, and the solve is that of one block per SM."""
    case, _, B = problem((700, 500))
    out = []
    for blocks in (0, 100000):
        g = gpu(case, monkeypatch, blocks, 0)
        out.append(g.sor_solve(B, np.zeros_like(B), 1e-40, False))
        out.append(g.sor_solve(B, np.zeros_like(B), 1e-40, False))   # and the next one
        g.close()
    for x, n, _ in out[1:]:
        assert n == out[0][1] and np.array_equal(x, out[0][0])


@pytest.mark.parametrize('shape,blocks', [((64, 48), 0), ((200, 100), 3)])   # every block a neighbour, or two of them
def test_a_wait_that_runs_out(shape, blocks, monkeypatch):
    """Blocks that wait for one that never comes give up and say so; the
    context solves as before afterwards."""
    case, o, B = problem(shape)
    want, its, _ = o.sor_solve(B, np.zeros_like(B), 1e-40, False)
    g = gpu(case, monkeypatch, blocks, 0)
    assert g.L.swm_gpu_check_sor_wait(g.ctx, 20) == 5
    assert b'waited too long' in g.L.swm_gpu_last_error()
    for limit in (0, -1, 1001):
        assert g.L.swm_gpu_check_sor_wait(g.ctx, limit) == 1
    got, n, _ = g.sor_solve(B, np.zeros_like(B), 1e-40, False)
    assert n == its and np.array_equal(got, want)
    g.close()
