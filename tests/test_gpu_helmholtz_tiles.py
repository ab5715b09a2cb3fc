"""The tiled FP32 Helmholtz sweeps at the edges of their regions: one region,
one column or row more, rows that start at multiples of four columns (streamed
regions) and rows that do not, blocks of 12 and of 24 warps (the latter where
every SM gets a region), more regions than resident blocks.  Each cell is
relaxed with the global sweep's arithmetic, so the result of every K equals
that of global sweeps bit for bit.
"""
import numpy as np
import pytest

from swm_gb300.model import GpuHelmholtz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nx,ny', [(4, 3), (48, 32), (52, 33), (56, 40), (60, 41), (63, 47), (64, 48), (65, 49),
                                   (628, 957), (629, 964), (1920, 1281)])
def test_tiles_equal_global_sweeps(nx, ny, monkeypatch):
    rng = np.random.default_rng(nx + 7 * ny)
    H = rng.uniform(50.0, 5000.0, (ny, nx))
    ocean = (rng.random((ny, nx)) < 0.95).astype(np.int8)
    ocean[1, 1] = 1
    rhs = 1e-10 * rng.standard_normal((ny, nx)) * ocean
    want = None
    for k in ('0', '1', '2', '3', '4'):
        monkeypatch.setenv('SWM_GB300_HELM_K', k)
        h = GpuHelmholtz(H, ocean, 5e3, 5e3, 1.6e-12)
        h.autotune(rhs, 1.7, 1.7, 1, 16)
        psi, sweeps, _, _, _ = h.solve(rhs, omega=1.7, rtol=1e-30, max_sweeps=12, mixed=True, raise_on_fail=False)
        h.close()
        if want is None:
            want = psi, sweeps
        assert sweeps == want[1] and np.array_equal(psi, want[0])
