"""dasha_setdt's screened sweep returns the largest rate itself: against the FP64 rates of every node, formed in numpy from the
perturbations as the context stores them (FP32 ones rounded, no compensation after a set_state), on evolved states and on
states whose nodes all tie to the rounding of the stored fields; consecutive calls, which take the two rate
words in turn, with larger and smaller rates after one another.  The formula takes a dozen roundings of FP64."""
import numpy as np
import pytest

from dasha_b200 import capi, harris

pytestmark = pytest.mark.gpu

TOL = 1e-14


def _rates(d, X, precision):
    """max over the region of the rate (dasha_setdt's formula) of the state X as stored"""
    rho0, b0, p0, _ = harris.harris_profiles(d.z)
    eq = np.zeros((8, d.mz))
    eq[0], eq[4:7], eq[7] = rho0, b0, p0
    P = X - eq[:, :, None, None]
    if precision:
        P = P.astype(np.float32).astype(np.float64)
    T = P + eq[:, :, None, None]
    p = d.params
    bb = T[4] ** 2 + T[5] ** 2 + T[6] ** 2
    vf = np.sqrt(np.abs((bb + p.gamma * T[7]) / T[0]))
    w = (p.di * np.pi if p.dt_whistler and p.hall else 0.0) * np.sqrt(bb) / T[0]
    best = 0.0
    for m, (c, shape) in enumerate(((d.x, (1, 1, -1)), (d.y, (1, -1, 1)), (d.z, (-1, 1, 1)))):
        h = np.abs(np.append(np.diff(c), c[-1] - c[-2])).reshape(shape)
        r = (np.abs(T[1 + m] / T[0]) + vf + w / h) / (p.cfl * h) + (p.eta + p.mu) / (2 * h * h)
        best = max(best, float(r[:-2, :-1, :-2].max()))
    return best


def _tied(d, X, rng):
    """the state with the x velocity of every node chosen so that all rates are the same number"""
    p = d.params
    X = X.copy()
    bb = X[4] ** 2 + X[5] ** 2 + X[6] ** 2
    vf = np.sqrt(np.abs((bb + p.gamma * X[7]) / X[0]))
    w = (p.di * np.pi if p.dt_whistler and p.hall else 0.0) * np.sqrt(bb) / X[0]
    h = np.abs(np.append(np.diff(d.x), d.x[-1] - d.x[-2])).reshape(1, 1, -1)
    top = 1.2 * (vf + w / h).max() / (p.cfl * h.min())
    X[1] = X[0] * (top * p.cfl * h - vf - w / h) * (1 + 1e-13 * rng.standard_normal(X[0].shape))
    return X


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("whistler", [0, 1])
@pytest.mark.parametrize("grid,stretch", [((36, 8, 20), False), ((100, 45, 77), True), ((160, 7, 9), True)],
                         ids=["36x8x20", "100x45x77", "160x7x9"])
def test_setdt_is_the_largest_rate(grid, stretch, whistler, precision):
    import dataclasses
    cfg = dataclasses.replace(harris.RunConfig("cfl", *grid, stretch, 0.005, 0.5, 1), dt_whistler=whistler)
    d = capi.gem_context(cfg, precision)
    rng = np.random.default_rng(11)
    t, states = 0.0, []
    for n in range(3):
        dt = d.setdt(t)
        d.stepon(t, dt, n)
        t += dt
        states.append(d.get_state())
    tied = _tied(d, states[0], rng)
    for X in (states[0], tied, states[1], states[2], tied, tied, states[0]):
        d.set_state(X)
        want = 1.0 / _rates(d, X, precision)
        got = [d.setdt() for _ in range(2)]
        assert got[0] == got[1]
        assert abs(got[0] - want) <= TOL * want, (got[0] / want - 1)
    d.close()
