"""A bounded context given a new equilibrium runs as a fresh context does, whatever it did before.  The inflow
driver reads rhoi at y index jz; on grids with mz - 1 >= 3 my that position of interior rows lies behind the
last physical plane, where the equilibrium has to hold zeros."""
import numpy as np
import pytest

from dasha_b200 import capi, dipole

pytestmark = pytest.mark.gpu


def _params():
    return capi.ParamsC(gamma=5 / 3, eta=2e-4, di=0.07, cfl=0.5, rcr=1.0, hall=1, viscos=0, diffu=0, total_e=1)


def _steps(d, X):
    d.set_state(X)
    t = 12.0
    for s in range(2):
        dt = d.setdt(t)
        d.stepon(t, dt, s)
        t += dt
    return d.get_state()


@pytest.mark.parametrize("grid", [(12, 7, 24), (33, 5, 40)], ids=lambda g: "x".join(map(str, g)))
def test_a_second_equilibrium_runs_as_the_first(grid):
    mx, my, mz = grid
    x, y, z = np.linspace(-2.1, 5.65, mx), np.linspace(-2.5, 2.5, my), np.linspace(-2.5, 2.5, mz)
    E, X = dipole.dipole_equilibrium(x, y, z), dipole.dipole_state(x, y, z)
    rng = np.random.default_rng(5)
    X[1:4] += 0.01 * rng.standard_normal(X[1:4].shape) * X[0]
    with dipole.bounded_context(x, y, z, _params(), E) as d:
        fresh = _steps(d, X)
    with dipole.bounded_context(x, y, z, _params(), E, X) as d:
        d.rhs(12.0)
        d.set_equilibrium_3d(E)
        again = _steps(d, X)
    assert np.isfinite(fresh).all()
    assert np.array_equal(fresh, again)
