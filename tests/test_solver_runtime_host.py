"""The solver's host runtime over a stand-in for the CUDA runtime, without a GPU."""
import ctypes

import numpy as np
import pytest

from test_batch_runtime_host import build_over_fake_runtime

NX, NY = 24, 18
OK, ERR_CUDA = 0, 2


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    lib = build_over_fake_runtime(tmp_path_factory.mktemp("solver_runtime"), "solver_runtime_host.cpp",
                                  [("fvm2d_capi.cu", ())])
    lib.sr_device.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    lib.sr_run.argtypes = [ctypes.c_double]
    lib.sr_device.restype = lib.sr_run.restype = lib.sr_seen.restype = None
    lib.sr_device_copies.restype = ctypes.c_long
    lib.fvm2d_set_end_time.argtypes = [ctypes.c_void_p, ctypes.c_double]
    return lib


@pytest.fixture
def handle(lib):
    h = ctypes.c_void_p()
    assert lib.fvm2d_create(ctypes.byref(h), NX, NY) == OK
    yield h
    lib.sr_device(None, 0)
    lib.fvm2d_destroy(h)


CALLS = {
    "set_state": lambda lib, h, p: lib.fvm2d_set_state(h, p, 5),
    "get_state": lambda lib, h, p: lib.fvm2d_get_state(h, p, 5),
    "set_state_planes": lambda lib, h, p: lib.fvm2d_set_state_planes(h, p),
    "get_state_planes": lambda lib, h, p: lib.fvm2d_get_state_planes(h, p),
    "set_rows": lambda lib, h, p: lib.fvm2d_set_rows(h, 3, 7, p),
    "get_rows": lambda lib, h, p: lib.fvm2d_get_rows(h, 3, 7, p),
}
DOUBLES = {"set_state": 5 * NX * NY, "get_state": 5 * NX * NY, "set_state_planes": 4 * NX * NY,
           "get_state_planes": 4 * NX * NY, "set_rows": 4 * 7 * NX, "get_rows": 4 * 7 * NX}


@pytest.mark.parametrize("call", CALLS)
def test_device_buffers_are_used_in_place_only_if_they_are_long_enough(lib, handle, call):
    """A kernel gets the caller's device buffer if all of it is there; one that
    ends before goes through the runtime's copy, which refuses it."""
    state = np.ones((NY, NX, 5))
    assert lib.fvm2d_set_state(handle, ctypes.c_void_p(state.ctypes.data), 5) == OK
    n = DOUBLES[call]
    buffer = np.ones(n + 40)  # (room behind the end that counts, for the copy that must not be made)
    start = buffer.ctypes.data + 16  # not at its allocation's start
    for doubles, code, copies in ((n, OK, 0), (n + 5, OK, 0), (n - 1, ERR_CUDA, 1)):
        lib.sr_device(buffer.ctypes.data, 16 + 8 * doubles)
        assert CALLS[call](lib, handle, ctypes.c_void_p(start)) == code, (doubles, code)
        assert lib.sr_device_copies() == copies
    lib.sr_device(None, 0)
    assert CALLS[call](lib, handle, ctypes.c_void_p(start)) == OK  # host memory


@pytest.mark.parametrize("n,first", [(24, 16), (800, 13), (2100, 1)])  # cells a side; steps before the first look
@pytest.mark.parametrize("call", ["solve", "advance"])
def test_few_steps_are_enqueued_past_the_end(lib, n, first, call):
    """A run that ends early leaves few steps that do nothing: each of them loads
    the array."""
    h = ctypes.c_void_p()
    assert lib.fvm2d_create(ctypes.byref(h), n, n) == OK
    state, out, done = np.ones((n, n, 4)), (ctypes.c_long * 3)(), ctypes.c_int(0)
    for steps in (0, 1, 2, 3, 13, 16, 17, 60, 128, 129, 300):
        lib.sr_run(0.25)  # (exact in binary)
        assert lib.fvm2d_set_end_time(h, 0.25 * steps) == OK
        assert lib.fvm2d_set_state(h, ctypes.c_void_p(state.ctypes.data), 4) == OK
        assert (lib.fvm2d_solve(h) if call == "solve" else lib.fvm2d_advance(h, 1000, ctypes.byref(done))) == OK
        lib.sr_seen(out)
        enqueued, ran, groups = out
        assert ran == steps and (call == "solve" or done.value == steps)
        assert enqueued <= max(first, steps + 1), (steps, list(out))
        assert groups <= 2 + steps // 100
    lib.fvm2d_destroy(h)


def test_a_short_advance_is_one_group(lib, handle):
    state, out, done = np.ones((NY, NX, 4)), (ctypes.c_long * 3)(), ctypes.c_int(0)
    assert lib.fvm2d_set_end_time(handle, 1e9) == OK
    assert lib.fvm2d_set_state(handle, ctypes.c_void_p(state.ctypes.data), 4) == OK
    for n in (1, 2, 16):
        lib.sr_run(0.25)
        assert lib.fvm2d_advance(handle, n, ctypes.byref(done)) == OK and done.value == n
        lib.sr_seen(out)
        assert list(out) == [n, n, 1]
