"""The FP32 hydro right-hand side with two nodes a thread (planes of 20 and more 64 x 6 tiles): tiles cut by the
grid's x and y ends, the smallest z range, a plane just below the rule's line, against the FP64 context's right-hand
side and, bit for bit, against the build that checks every global index."""
import numpy as np
import pytest

from dasha_b200 import capi, harris

pytestmark = pytest.mark.gpu

# |rhs FP32 - rhs FP64|: every term is a difference quotient, sum |coefficient| <= 30 on the stretched z axis of these
# grids, of a field below 0.2, or a product of a current and a field of order one.  Rounded to 2^-24 each:
# 30 * 0.2 * 6e-8 = 4e-7 per quotient, three of them, the current's again times |B| = 1, and 1e-7 per product:
# below 3e-6.  A node read from the wrong place changes the quotient by 30 * 1e-2.
TOL = 1e-5


@pytest.mark.parametrize("hall", [1, 0])
@pytest.mark.parametrize("grid", [(124, 66, 9), (128, 61, 7), (192, 42, 13), (256, 31, 8), (128, 54, 8)],
                         ids=lambda g: "x".join(map(str, g)))
def test_rhs_of_node_pairs(grid, hall):
    cfg = harris.RunConfig("pairs", *grid, True, 0.005, 0.5, 1, hall=hall)
    x, y, z = harris.make_grid(*grid, cfg.stretch)
    X = harris.gem_state(x, y, z) + 1e-2 * np.random.default_rng(11).uniform(-1, 1, (8, *grid[::-1]))
    out = []
    for precision, lib in ((0, None), (1, None), (1, capi.bind(capi.BOUNDS_LIB_PATH))):
        d = capi.gem_context(cfg, precision, lib=lib)
        d.set_state(X)
        out.append(d.rhs(0.5))
        d.close()
    hydro = [0, 1, 2, 3, 7]
    assert np.abs(out[1][hydro] - out[0][hydro]).max() <= TOL
    assert np.array_equal(out[1], out[2])
