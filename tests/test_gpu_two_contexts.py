"""Two contexts driven in turn by one host thread with steps in flight (dasha_stepon only enqueues): each gives the states
and time steps of its own run, bit for bit; and a ring wait that ran out (planted on the host through the checking
build's dasha_check_ring_wait, which stores what such a launch stores) is reported by the context whose launch it was,
by that one alone, at its next call that waits."""
import ctypes as C

import numpy as np
import pytest

from dasha_b200 import capi, harris

pytestmark = pytest.mark.gpu

CFGS = [harris.RunConfig("turns-64x32x64", 64, 32, 64, False, 0.005, 0.5, 1),
        harris.RunConfig("turns-100x44x77-sinh", 100, 44, 77, True, 0.003, 1.0, 2, dt_whistler=1)]


def _run_alone(cfg, precision, steps):
    d = capi.gem_context(cfg, precision)
    t, dts = 0.0, []
    for n in range(steps):
        dts.append(d.setdt(t))
        d.stepon(t, dts[-1], n)
        t += dts[-1]
    X = d.get_state()
    d.close()
    return dts, X


@pytest.mark.parametrize("precisions", [(0, 0), (0, 1), (1, 1)], ids=["fp64-fp64", "fp64-fp32", "fp32-fp32"])
def test_contexts_stepped_in_turn_keep_apart(precisions):
    steps = 6
    alone = [_run_alone(c, p, steps) for c, p in zip(CFGS, precisions)]
    ds = [capi.gem_context(c, p) for c, p in zip(CFGS, precisions)]
    t, dts = [0.0, 0.0], [[], []]
    for n in range(steps):
        for q, d in enumerate(ds):
            dts[q].append(d.setdt(t[q]))       # with the other context's step still in flight
        for q, d in enumerate(ds):
            d.stepon(t[q], dts[q][-1], n)
            t[q] += dts[q][-1]
    for q, d in enumerate(ds):
        assert dts[q] == alone[q][0]
        assert np.array_equal(d.get_state(), alone[q][1])
        d.close()


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("call", ["setdt", "get_state", "diagnostics", "timer_stop", "profile_read"])
def test_a_ring_wait_is_reported_by_its_own_context(call, precision):
    lib = capi.bind(capi.BOUNDS_LIB_PATH)
    lib.dasha_check_ring_wait.argtypes = [C.c_void_p]
    a, b = (capi.gem_context(CFGS[0], precision, lib=lib) for _ in range(2))
    dt = a.setdt(0.0)
    a.timer_start()
    a.stepon(0.0, dt, 0)
    assert lib.dasha_check_ring_wait(a.h) == capi.OK
    b.stepon(0.0, b.setdt(0.0), 0)
    b.get_state()
    b.diagnostics()
    assert b.setdt(0.0) > 0
    with pytest.raises(capi.DashaError, match="ring wait") as e:
        getattr(a, call)()
    assert e.value.code == capi.E_CUDA
    with pytest.raises(capi.DashaError):
        a.stepon(0.0, dt, 1)                   # a context that lost a pass stays failed
    a.close()
    b.stepon(0.0, dt, 1)
    assert np.isfinite(b.get_state()).all()
    b.close()


@pytest.mark.parametrize("write", ["checkpoint", "m3d"])
def test_a_failed_step_leaves_the_files_before_it(write, tmp_path):
    """dasha_checkpoint and dasha_m3d_write_ctx look for the step's status before they open their file: the last good
    one stays as it is."""
    lib = capi.bind(capi.BOUNDS_LIB_PATH)
    lib.dasha_check_ring_wait.argtypes = [C.c_void_p]
    d = capi.gem_context(CFGS[0], 0, lib=lib)
    path = str(tmp_path / "file").encode()

    def out():
        if write == "checkpoint":
            return lib.dasha_checkpoint(d.h, path, 1, 2, 0.5, 3, 0)
        return lib.dasha_m3d_write_ctx(d.h, path, 0.5)

    assert out() == capi.OK
    good = {p.name: p.read_bytes() for p in tmp_path.iterdir()}
    d.stepon(0.0, d.setdt(0.0), 0)
    assert lib.dasha_check_ring_wait(d.h) == capi.OK
    assert out() == capi.E_CUDA
    assert {p.name: p.read_bytes() for p in tmp_path.iterdir()} == good
    d.close()
