"""Steps in tiles of very tall and very wide arrays are launches the device can
take (a grid's second dimension ends at 65535), without a GPU."""
import ctypes

import pytest

from test_batch_runtime_host import build_over_fake_runtime


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return build_over_fake_runtime(tmp_path_factory.mktemp("tall_grid"), "tall_grid_host.cpp",
                                   [("fvm2d_fp64.cu", ("-fmad=false",))])


@pytest.mark.parametrize("taped", [0, 1])
@pytest.mark.parametrize("nx,ny", [(6, 6), (100, 90), (6, 393_224), (6, 1_966_055), (32, 60_000_000), (2_000_000, 6),
                                   (45_000, 45_000)])
def test_steps_of_any_shape_can_be_launched(lib, nx, ny, taped):
    blocks = (ctypes.c_longlong * 2)()
    assert lib.tg_step(nx, ny, taped, blocks) == 0
    # some tile of 30, 14 or 6 cells a side covers the interior
    shapes = [(30, 30), (14, 14), (14, 6)]
    tiles = [-(-(nx - 4) // x) * -(-(ny - 4) // y) for x, y in shapes]
    assert any(n <= blocks[0] <= n + 65535 * -(-(nx - 4) // 6) for n in tiles)
    assert blocks[0] in tiles or ny > 65535 * 6
    assert blocks[1] * 256 >= 4 * nx + 4 * (ny - 4)
