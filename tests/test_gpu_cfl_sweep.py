"""dasha_setdt's sweep screens nodes by an FP32 bound: the node with the largest rate has to be found wherever it is,
whatever sets it, next to a crowd of nodes within a rounding of it, with a density that nearly cancels, and a NaN has to win.
Against the oracle's sweep of the same state."""
import numpy as np
import pytest

from dasha_b200 import capi, harris

pytestmark = pytest.mark.gpu

GRIDS = [(36, 8, 20), (100, 6, 12), (160, 7, 9), (64, 45, 77)]
# FP64: the tolerance of the other setdt comparisons; FP32: the stored perturbation is rounded to 2^-24 of itself, at most
# 1.5 roundings of rate per rounding of a field, and the quiet nodes stay 1e-3 below the one that counts
TOL = {0: 1e-14, 1: 2e-7}


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("whistler", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
def test_largest_rate_is_found(grid, whistler, precision):
    import dataclasses
    from oracle.oracle import gem_oracle
    cfg = dataclasses.replace(harris.RunConfig("cfl", *grid, True, 0.005, 0.5, 1), dt_whistler=whistler)
    mx, my, mz = grid
    o, d = gem_oracle(cfg), capi.gem_context(cfg, precision)
    X0 = o.get_state()
    rng = np.random.default_rng(3)
    last = (mz - 3, my - 2, mx - 3)
    places = [(0, 0, 0), last, (last[0], 0, 1), (1, last[1], 2)] + [tuple(int(rng.integers(0, n + 1)) for n in last) for _ in range(4)]
    for n, (k, j, i) in enumerate(places):
        X = X0.copy()
        m = (n % 3) + 1
        if n % 2:
            X[m, k, j, i] = -40.0 * X[0, k, j, i]     # a fast node
        else:
            X[0, k, j, i] = 2e-3                      # a nearly empty one: far below the background
            X[m, k, j, i] = 0.5
        X[1:4, :, my - 1, :] = 1e4                    # outside the region
        X[1:4, :, :, mx - 2:] = 1e4
        X[1:4, mz - 2:, :, :] = 1e4
        o.set_state(X)
        d.set_state(X)
        # an FP32 density total of 2e-3 on a background of order one carries 2^-24 of the background
        tol = TOL[precision] + (0 if precision == 0 or n % 2 else 6e-8 * 1.3 / 2e-3)
        assert abs(d.setdt() - o.setdt()) <= tol * o.setdt(), (n, d.setdt(), o.setdt())
    X = X0.copy()
    X[7, last[0], last[1], last[2]] = np.nan
    d.set_state(X)
    with pytest.raises(capi.DashaError, match="not a positive finite"):
        d.setdt()
    d.close()
