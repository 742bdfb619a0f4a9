"""The transposed right-hand side on the smallest grids and ragged ones: planes next to both walls at once
(mz = 7), fewer columns than a block, columns that do not fill one.  <W, G' V> by central differences of the
library's own right-hand side against <G'^T W, V>, with the inputs, the step and the tolerance of
the same check on the 32x16x32 grid (tests/test_gpu_adjoint.py)."""
import numpy as np
import pytest

from dasha_b200 import capi, harris

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hall", [1, 0])
@pytest.mark.parametrize("grid", [(8, 5, 7), (36, 5, 8), (44, 6, 9), (132, 7, 13)], ids=lambda g: "x".join(map(str, g)))
def test_adjoint_rhs_dot_product_on_small_grids(grid, hall):
    cfg = harris.RunConfig("adj-edge", *grid, True, 0.005, 0.5, 1, hall=hall)
    x, y, z = harris.make_grid(*grid, cfg.stretch)
    X = harris.gem_state(x, y, z)
    rng = np.random.default_rng(5)
    V = 1e-3 * rng.standard_normal(X.shape)
    W = rng.standard_normal(X.shape)
    d = capi.gem_context(cfg, 0)
    GtW = d.adjoint_rhs(W)
    e = 1e-3
    d.set_state(X + e * V)
    gp = d.rhs(0.5)
    d.set_state(X - e * V)
    gm = d.rhs(0.5)
    d.close()
    lhs, rhs = float(np.sum(W * (gp - gm) / (2 * e))), float(np.sum(GtW * V))
    scale = float(np.linalg.norm(W) * np.linalg.norm((gp - gm) / (2 * e)))   # the products may cancel on a few nodes
    assert abs(lhs - rhs) <= 1e-6 * max(abs(lhs), 1e-3 * scale), (lhs, rhs)
