"""Runs of steps in tiles through the records that hand them on, without a GPU:
bit for bit the oracle's steps, in groups of every parity, to an end time in
the middle of a group or to a step limit; and single-precision tiles bit for
bit the sweeps."""
import ctypes

import numpy as np
import pytest

from test_kernels_host import build_host, sweep_case


@pytest.fixture(scope="module")
def tc(tmp_path_factory):
    lib = build_host(tmp_path_factory, "tile_chain_host.cpp")
    lib.tc_run.argtypes = ([ctypes.c_void_p] + [ctypes.c_int] * 2 + [ctypes.c_double] * 4 + [ctypes.c_int] * 4 +
                           [ctypes.c_void_p] * 2)
    lib.tc_single.argtypes = [ctypes.c_int] * 2 + [ctypes.c_void_p] + [ctypes.c_int] * 2 + [ctypes.c_double] * 3
    lib.tc_single.restype = ctypes.c_long
    return lib


@pytest.mark.parametrize("strategy,group,limit", [(0, 1, 9), (1, 2, 9), (2, 3, 7), (3, 4, 8), (4, 5, 9), (5, 16, 9),
                                                  (6, 3, 1 << 30), (0, 4, 1 << 30), (4, 1, 1 << 30)])
def test_runs_equal_the_oracles(tc, oracle, pkg, strategy, group, limit):
    nx, ny, width, height = 37, 21, 1.0, 0.6
    U = oracle.ghost(pkg.scenarios.seeded_four_quadrant(nx, ny, 11 + strategy), strategy, width=width, height=height)
    kw = dict(width=width, height=height, cfl=0.4, alpha=1.9, gamma=1.4, strategy=strategy)
    _, t, dt = oracle.step(U, t=0.0, t_end=1e9, **kw)
    t_end = 6.3 * dt if limit > 1000 else 1e9
    V, t, steps, done = U, 0.0, 0, 0
    while steps < limit:
        r = oracle.step(V, t=t, t_end=t_end, **kw)
        if r is None:
            done = 1
            break
        V, t, dt = r
        steps += 1
    out, rec = np.empty_like(U), np.empty(5)
    C = np.ascontiguousarray(U)
    active = tc.tc_run(C.ctypes.data, nx, ny, width, height, t_end, 0.4, min(limit, 2**31 - 1), strategy, group, 40,
                       out.ctypes.data, rec.ctypes.data)
    assert active == 0 and steps > 5
    assert np.array_equal(out, V)
    assert (rec[0], rec[2], rec[3], rec[4]) == (t, steps, done, 0)


def test_a_bad_cell_is_noted_with_its_step(tc, oracle, pkg):
    U, width, height, _ = sweep_case(pkg, oracle, 37, 21, 3)
    U = np.ascontiguousarray(U)
    U[10, 20, 1] = np.nan
    out, rec = np.empty_like(U), np.empty(5)
    tc.tc_run(U.ctypes.data, 37, 21, width, height, 1e9, 0.4, 4, 0, 2, 4, out.ctypes.data, rec.ctypes.data)
    assert rec[2] == 4 and rec[4] == 1


@pytest.mark.parametrize("physics", [0, 1, 2])
@pytest.mark.parametrize("shape", [0, 1])
@pytest.mark.parametrize("nx,ny", [(6, 6), (35, 33), (70, 47)])
def test_single_precision_tiles_equal_the_sweeps(tc, oracle, pkg, nx, ny, shape, physics):
    U, width, height, dt = sweep_case(pkg, oracle, nx, ny, 8)
    U = np.ascontiguousarray(U * (1 + 1e-3 * np.random.default_rng(2).uniform(-1, 1, U.shape)))
    assert tc.tc_single(physics, shape, U.ctypes.data, nx, ny, width, height, dt) == 0
