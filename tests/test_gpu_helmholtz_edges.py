"""The FP64 Helmholtz kernels at the edges of their blocks, against the oracle:
sweeps (256 cells of a colour per block, rows of even and odd length) and A psi
bit for bit; the residual (128 columns by 32 rows per block) by its norm.  The
norm is a sum of n squares in another order, of differences whose terms are
rounded otherwise: relative error below 1e-12 where nothing cancels (one sweep
from zero leaves a residual of the size of the right-hand side).
"""
import numpy as np
import pytest

from oracle import helmholtz_apply, helmholtz_coeffs, helmholtz_sor
from swm_gb300.model import GpuHelmholtz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nx,ny', [(3, 3), (4, 31), (127, 33), (128, 32), (129, 31), (130, 65), (257, 64), (512, 5)])
def test_edges(nx, ny):
    rng = np.random.default_rng(nx * 1000 + ny)
    H = rng.uniform(50.0, 5000.0, (ny, nx))
    ocean = (rng.random((ny, nx)) < 0.9).astype(np.int8)
    ocean[1, 1] = 1
    rhs = 1e-10 * rng.standard_normal((ny, nx)) * ocean
    dx, lam = 5e3, 1.6e-12
    cx, cy, cc = helmholtz_coeffs(1.0 / H, lam, dx, dx)
    h = GpuHelmholtz(H, ocean, dx, dx, lam)
    psi = rng.standard_normal((ny, nx))
    assert np.array_equal(h.apply(psi), helmholtz_apply(cx, cy, cc, ocean, psi))
    m = ocean == 1
    for sweeps in (1, 7):
        want, _, _ = helmholtz_sor(cx, cy, cc, ocean, rhs, np.zeros_like(H), 1.9, 1e-30, sweeps)
        got, n, _, rel, _ = h.solve(rhs, omega=1.9, rtol=1e-30, max_sweeps=sweeps, raise_on_fail=False)
        assert n == sweeps and np.array_equal(got, want)
        if sweeps == 1:
            r = rhs - helmholtz_apply(cx, cy, cc, ocean, want)
            norm = np.linalg.norm(r[m]) / np.linalg.norm(rhs[m])
            assert abs(rel - norm) <= 1e-12 * norm
    mixed, _, _, rel, rc = h.solve(rhs, omega=1.5, rtol=1e-10, mixed=True)
    r = rhs - helmholtz_apply(cx, cy, cc, ocean, mixed)
    assert rc == 0 and np.linalg.norm(r[m]) < 1e-10 * np.linalg.norm(rhs[m])
    h.close()
