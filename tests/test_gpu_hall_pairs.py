"""Planes just below and just above the line from which an FP32 step smooths the Hall field by fused pairs of passes: the
z-slabs of the same grid always take single passes, and their states are bit for bit the whole grid's."""
import numpy as np
import pytest

from dasha_b200 import capi, harris, slabs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("my", [256, 257])
def test_fused_hall_pairs_equal_single_passes(my):
    cfg = harris.RunConfig("hall-1024x%dx10" % my, 1024, my, 10, True, 0.003, 1.0, 1)
    one = capi.gem_context(cfg, 1)
    grp = slabs.gem_slab_group(cfg, 2, 1)
    try:
        dt = one.setdt(0.0)
        assert dt == grp.setdt(0.0)
        for d in (one, grp):
            d.stepon(0.0, dt, 1)
        assert np.array_equal(one.get_state(), grp.get_state())
    finally:
        grp.close()
        one.close()
