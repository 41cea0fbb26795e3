"""The reverse step's own kernels, without a GPU: the ring's transpose as it
gathers, bit for bit the scatter, for every preset and on arrays whose corners
meet; the two transposes side by side, bit for bit each alone; their sum."""
import ctypes

import numpy as np
import pytest

from test_kernels_host import build_host, sweep_case


@pytest.fixture(scope="module")
def rs(tmp_path_factory):
    lib = build_host(tmp_path_factory, "reverse_step_host.cpp")
    lib.rs_ring.argtypes = [ctypes.c_void_p] * 2 + [ctypes.c_int] * 3
    lib.rs_pair.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 2 + [ctypes.c_double] * 2
    lib.rs_ring.restype = lib.rs_pair.restype = ctypes.c_long
    return lib


@pytest.mark.parametrize("strategy", range(7))
@pytest.mark.parametrize("nx,ny", [(6, 6), (7, 6), (6, 7), (7, 9), (8, 8), (9, 23), (50, 11), (61, 40)])
def test_ring_transpose_gathers_what_a_scatter_adds(rs, nx, ny, strategy):
    r = np.random.default_rng([nx, ny, strategy])
    p, q = r.integers(-1000, 1000, (2, ny, nx, 4)).astype(float)
    assert rs.rs_ring(p.ctypes.data, q.ctypes.data, nx, ny, strategy) == 0


@pytest.mark.parametrize("nx,ny", [(6, 6), (7, 9), (26, 26), (27, 31), (60, 53)])
def test_pair_of_transposes_equals_each_alone(rs, oracle, pkg, nx, ny):
    U, width, height, dt = sweep_case(pkg, oracle, nx, ny, 5)
    r = np.random.default_rng([nx, ny])
    bx, by = r.uniform(-1, 1, (2, ny, nx, 4))
    assert rs.rs_pair(U.ctypes.data, bx.ctypes.data, by.ctypes.data, nx, ny, width / nx, dt) == 0
