"""swm_gpu_get_field_async into pinned arrays at every offset from a double's
alignment: small fields of the pair state are stored there by a kernel where
the array is aligned, and copied where it is not."""
import ctypes

import numpy as np
import pytest

from harness import run_case
from swm_gb300._lib import FIELD_ID, check
from swm_gb300.host import synthetic
from swm_gb300.model import GpuModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('path', ['plain_fp64', 'fused_fp32c'])
def test_unaligned_pinned_array(path):
    import torch
    case = synthetic.double_gyre((45, 37), biharmonic=False, nsteps=8)
    g = GpuModel(path)
    run_case(case, g, nsteps=8, with_diag=False)
    want = g.field('u')
    raw = torch.empty(want.nbytes + 64, dtype=torch.uint8).pin_memory()
    for offset in (0, 1, 2, 4, 7, 8, 12):
        raw.fill_(0x5a)
        ticket = ctypes.c_int64()
        check(g.L.swm_gpu_get_field_async(g.ctx, FIELD_ID['u'], raw.data_ptr() + offset, ctypes.byref(ticket)))
        g.wait(ticket.value)
        got = raw.numpy().tobytes()
        assert got[offset:offset + want.nbytes] == want.tobytes(), offset
        assert set(got[:offset] + got[offset + want.nbytes:]) == {0x5a}, offset
    g.close()
