"""The step in tiles (2d_fvm_cuda_b200/csrc/fvm2d_tile.cuh) compiled for the
host (tests/tile_host.cpp), without a GPU: with the reference's operation
order the interior cells of one step equal the oracle's bit for bit, for
every tile shape, on arrays smaller than a tile, of exactly one or two tiles
and one cell more or less; with shared reciprocals they agree to rounding."""
import ctypes

import numpy as np
import pytest

from test_kernels_host import build_host, sweep_case

SHAPES = [(30, 30), (30, 14), (14, 14), (14, 6)]


@pytest.fixture(scope="module")
def th(tmp_path_factory):
    lib = build_host(tmp_path_factory, "tile_host.cpp")
    lib.th_step.argtypes = ([ctypes.c_int] * 2 + [ctypes.c_void_p] * 2 + [ctypes.c_int] * 2 + [ctypes.c_double] * 5 +
                            [ctypes.c_void_p] * 2)
    lib.th_tape.argtypes = [ctypes.c_int, ctypes.c_void_p] + [ctypes.c_int] * 3 + [ctypes.c_double] * 4 + [ctypes.c_int]
    lib.th_tape.restype = ctypes.c_long
    return lib


def sizes(tx, ty):
    return [(6, 6), (tx + 4, ty + 4), (tx + 5, ty + 3), (2 * tx + 3, ty + 5), (7, 2 * ty + 5)]


@pytest.mark.parametrize("shape", range(4))
def test_interior_of_a_step_equals_the_oracle(th, oracle, pkg, shape):
    for k, (nx, ny) in enumerate(sizes(*SHAPES[shape])):
        U, width, height, dt = sweep_case(pkg, oracle, nx, ny, 40 + k)
        O = 0.5 * (oracle.sweep_y(oracle.sweep_x(U, width, dt), height, dt) +
                   oracle.sweep_x(oracle.sweep_y(U, height, dt), width, dt))
        P = np.ascontiguousarray(U.transpose(2, 0, 1))
        for policy in (0, 1):
            out = np.full_like(P, np.nan)
            vmax, bad = ctypes.c_double(0), ctypes.c_int(0)
            assert th.th_step(policy, shape, P.ctypes.data, out.ctypes.data, nx, ny, width, height, dt, 1.9, 1.4,
                              ctypes.byref(vmax), ctypes.byref(bad)) == 0
            G = out.transpose(1, 2, 0)
            ring = np.ones((ny, nx), bool)
            ring[2:-2, 2:-2] = False
            assert np.isnan(G[ring]).all()  # the ring is the ghost fill's
            A, B = G[~ring], O[~ring]
            assert bad.value == 0
            if policy == 0:
                assert np.array_equal(A, B), (nx, ny)
                speed = np.sqrt(B[:, 2] ** 2 + B[:, 3] ** 2) + np.sqrt(1.4 * B[:, 1] / B[:, 0])
                assert vmax.value == pytest.approx(speed.max(), rel=1e-15)
            else:
                # two sweeps of relative rounding, as the walkers' items (1e-13 each)
                assert np.abs(A - B).max() <= 2e-13 * np.abs(B).max(), (nx, ny)


@pytest.mark.parametrize("strategy", range(7))
@pytest.mark.parametrize("shape", range(4))
def test_tape_equals_the_sweeps(th, oracle, pkg, shape, strategy):
    """What a taped step in tiles keeps (X(U), Y(U), the sweeps' fluxes, and
    the ring it fills in its input) against the taped sweeps, bit for bit."""
    tx, ty = SHAPES[shape]
    for k, (nx, ny) in enumerate([(6, 6), (tx + 4, ty + 4), (tx + 5, 2 * ty + 3)]):
        U, width, height, _ = sweep_case(pkg, oracle, nx, ny, 60 + k)
        t = 0.01 * k
        U = np.ascontiguousarray(oracle.ghost(U, strategy, t=t, width=width, height=height))
        dt = 0.3 * min(width / nx, height / ny) / oracle.max_speed(U)  # the presets' inflows are in the ring
        for fill in (0, 1):
            assert th.th_tape(shape, U.ctypes.data, nx, ny, strategy, t, dt, width, height, fill) == 0, (nx, ny, fill)
