"""Steps in tiles give the bits of the same steps sweep by sweep, in every build
that leaves the compiler no contraction: tests/test_tile_gpu.py's comparison
for the single-precision builds, exactly, and at a size whose 30 x 30 tiles
fill the device in all builds."""
import numpy as np
import pytest

from test_tile_gpu import PRESETS, start, sweeps

pytestmark = pytest.mark.gpu

SMALL = [(6, 6), (17, 11), (34, 34), (35, 33), (130, 129), (257, 131), (400, 402), (611, 500)]
LARGE = (1003, 1021)  # 34 x 34 tiles of 30 x 30


def same(pkg, nx, ny, preset, precision, n):
    a, b = (start(pkg, nx, ny, preset, precision, 1) for _ in range(2))
    S = a.get_state(4)
    a.set_state(S)  # a run of its own from t = 0, as slab_begin starts one
    assert a.advance(n) == n
    t = sweeps(b, n)
    A, B = a.get_state(4), b.get_state(4)
    assert np.isfinite(A).all() and not np.array_equal(A, S)
    assert np.array_equal(A, B), (preset, n)
    assert a.time()[0] == t
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [3, 4])
@pytest.mark.parametrize("nx,ny", SMALL)
def test_single_precision_tiles_equal_sweeps(pkg, nx, ny, precision):
    for preset in (PRESETS if nx == 35 else [PRESETS[(nx + ny) % len(PRESETS)]]):
        same(pkg, nx, ny, preset, precision, 3)


@pytest.mark.parametrize("precision", [0, 1, 3, 4])
@pytest.mark.parametrize("preset", [0, 4, 5, 6])
def test_large_tiles_equal_sweeps(pkg, preset, precision):
    same(pkg, *LARGE, preset, precision, 2)


def test_large_tiles_of_the_contracting_build(pkg):
    """FP64_REFORDER, whose kernels the compiler contracts: to rounding."""
    a, b = (start(pkg, *LARGE, 0, 2, 1) for _ in range(2))
    a.set_state(a.get_state(4))
    assert a.advance(2) == 2
    sweeps(b, 2)
    A, B = a.get_state(4), b.get_state(4)
    assert np.abs(A - B).max() <= 1e-12 * np.abs(B).max()
    a.close()
    b.close()
