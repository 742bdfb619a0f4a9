"""dasha_stepon of a bounded context enqueues, as its declaration says: the host is free long before the steps are done, and
the calls that follow (time step, state, a new state) take their place behind them."""
import time

import numpy as np
import pytest

from dasha_b200 import capi, dipole

pytestmark = pytest.mark.gpu


def _context(grid):
    mx, my, mz = grid
    x, y, z = np.linspace(-2.1, 5.65, mx), np.linspace(-2.5, 2.5, my), np.linspace(-2.5, 2.5, mz)
    p = capi.ParamsC(gamma=5 / 3, eta=2e-4, di=0.07, cfl=0.5, rcr=1.0, hall=1, viscos=0, diffu=0, total_e=1)
    E, X = dipole.dipole_equilibrium(x, y, z), dipole.dipole_state(x, y, z)
    return dipole.bounded_context(x, y, z, p, E, X), X


def test_steps_are_enqueued():
    d, X = _context((129, 72, 101))
    dt = 0.1 * d.setdt(0.0)
    ratio = []
    for _ in range(4):                       # the first one loads the kernels
        d.timer_start()
        t0 = time.perf_counter()
        for n in range(5):
            d.stepon(1.0 + n * dt, dt, n)
        host = time.perf_counter() - t0
        ratio.append(1e3 * host / d.timer_stop())
    d.close()
    assert min(ratio) < 0.6, ratio


@pytest.mark.parametrize("grid", [(41, 25, 33), (64, 40, 50)], ids=lambda g: "x".join(map(str, g)))
def test_calls_behind_enqueued_steps(grid):
    """a second state and its steps follow enqueued ones: the result is that of a fresh context"""
    a, X = _context(grid)
    b, _ = _context(grid)
    dt = 0.1 * a.setdt(0.0)
    for n in range(3):
        a.stepon(1.0 + n * dt, dt, n)
    a.set_state(X)
    b.set_state(X)
    for d in (a, b):
        for n in range(2):
            d.stepon(2.0 + n * dt, dt, n)
    assert a.setdt(2.0) == b.setdt(2.0)
    assert np.array_equal(a.get_state(), b.get_state())
    a.close()
    b.close()


@pytest.mark.parametrize("grid", [(5, 7, 9), (41, 25, 33), (66, 40, 53), (129, 72, 101)], ids=lambda g: "x".join(map(str, g)))
def test_states_come_back_as_they_went(grid):
    """both ways of gathering the rows, one and several chunks, pageable and pinned: the state of dasha_get_state is that of
    dasha_set_state, and the caller's halo stays as it was"""
    from dasha_b200 import harris
    d, X = _context(grid)
    rng = np.random.default_rng(2)
    for _ in range(2):
        Y = X * (1 + 0.1 * rng.standard_normal(X.shape))
        d.set_state(Y)
        H = harris.to_halo(np.zeros_like(X))
        H[:] = 7.0
        assert d.lib.dasha_get_state(d.h, capi._dp(H), H.shape[3], H.shape[2]) == capi.OK
        assert np.array_equal(harris.from_halo(H, *grid), Y)
        H[:, 2:-2, :, 2:-2] = 7.0
        assert (H == 7.0).all()
    d.close()
