"""Evict-last population stores (bit 13 of the launch shapes) follow from the L2 of
the device: set while both buffers of the fluid nodes take at most half of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _l2_bytes():
    import torch
    return torch.cuda.get_device_properties(0).L2_cache_size


@pytest.mark.parametrize("side", [-1, 0, 1])
def test_line_at_half_the_l2(built, side):
    from hemocell_gb300 import _lib as L
    from hemocell_gb300.hemocell import HemoCell
    line = _l2_bytes() // (2 * 152)           # fluid nodes whose two FP32 buffers take half the L2
    nz = -(-(line + 64) // (96 * 80))
    flags = np.ones(96 * 80 * nz, np.uint8)
    flags[:line + side] = 0
    hc = HemoCell(96, 80, nz, form=L.HC_FORM_MIXED_F32, launch=L.HC_LAUNCH_BATCHED)
    hc.set_flags(flags)
    assert bool(hc.tuning()[7] & 0x2000) == (side <= 0)
    hc.close()
