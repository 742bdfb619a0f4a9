"""The bounded engine on the GPU against the host build of the same core (tests/walls_host.cpp), which
tests/test_walls_host.py holds against the reference program: the executor's node mapping, the loops
over all fields (one thread for all or one per field, by grid size), the division by a known
reciprocal and the packed transfers, on the narrowest grids (where the x-min extrapolation reaches the
x-max rows), ragged ones, and one of each side of the loops' size rule.  The two differ by the
rounding of exp and tanh only; the tolerance is that of the comparison with the reference
(tests/test_gpu_dipole.py)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from dasha_b200 import capi, dipole, harris

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
D = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def host_core(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("walls") / "libwalls_host.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-x", "c++",
                    "-I" + os.path.join(ROOT, "dasha_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "walls_host.cpp")], check=True)
    L = C.CDLL(out)
    L.wh_create.restype = C.c_void_p
    L.wh_create.argtypes = [C.c_int] * 3 + [D] * 4 + [C.c_int] * 4
    for fn in ("wh_set_eq", "wh_set_x"):
        getattr(L, fn).argtypes = [C.c_void_p, D]
    L.wh_get.argtypes = [C.c_void_p, C.c_int, D]
    L.wh_setdt.restype = C.c_double
    L.wh_setdt.argtypes = [C.c_void_p]
    L.wh_stepon.argtypes = [C.c_void_p, C.c_double, C.c_double]
    return L


def _p(a):
    return a.ctypes.data_as(D)


@pytest.mark.parametrize("hall,uyz,visc", [(1, 0, 0.0), (0, 1, 1e-3)], ids=["hall", "uyzlimiter-viscous"])
@pytest.mark.parametrize("grid", [(5, 7, 9), (6, 5, 8), (33, 9, 17), (64, 40, 50)], ids=lambda g: "x".join(map(str, g)))
def test_gpu_engine_equals_the_host_build(host_core, grid, hall, uyz, visc):
    mx, my, mz = grid
    x, y, z = np.linspace(-2.1, 5.65, mx), np.linspace(-2.5, 2.5, my), np.linspace(-2.5, 2.5, mz)
    E = dipole.dipole_equilibrium(x, y, z)
    X = dipole.dipole_state(x, y, z)
    rng = np.random.default_rng(7)
    X[1:4] += 0.01 * rng.standard_normal(X[1:4].shape) * X[0]
    X[4:7] *= 1 + 0.01 * rng.standard_normal(X[4:7].shape)
    par = np.array([5 / 3, 2e-4, visc, visc / 2, visc / 3, 0.5, 1.0, 0.07])
    h = host_core.wh_create(mx, my, mz, _p(x), _p(y), _p(z), _p(par), hall, uyz, 0, 0)

    def padded(a):
        return np.nan_to_num(harris.to_halo(a))

    host_core.wh_set_eq(h, _p(padded(E)))
    host_core.wh_set_x(h, _p(padded(X)))
    p = capi.ParamsC(gamma=5 / 3, eta=2e-4, di=0.07, mu=visc, drho=visc / 2, dp=visc / 3, cfl=0.5, rcr=1.0, hall=hall,
                     viscos=1, diffu=1, total_e=1, uyzlimiter=uyz)
    with dipole.bounded_context(x, y, z, p, E, X) as d:
        t = 12.0
        for s in range(3):
            dt = host_core.wh_setdt(h)
            assert abs(d.setdt(t) - dt) <= 1e-13 * dt
            host_core.wh_stepon(h, t, dt)
            d.stepon(t, dt, s)
            t += dt
        H = np.zeros((8, mz + 4, my, mx + 4))
        host_core.wh_get(h, 0, _p(H))
        a, b = d.get_state(), harris.from_halo(H, mx, my, mz)
    for m in range(8):
        assert np.abs(a[m] - b[m]).max() <= 1e-12 * np.abs(b[m]).max(), m
