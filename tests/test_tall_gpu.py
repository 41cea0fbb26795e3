"""Very tall arrays step in tiles as they do sweep by sweep: more tile rows than
a grid's second dimension holds."""
import numpy as np
import pytest

from test_tile_gpu import sweeps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 3])
def test_two_million_rows(pkg, precision):
    nx, ny = 6, 2_000_000
    r = np.random.default_rng(9)
    P = np.empty((4, ny, nx))
    for f, (lo, hi) in enumerate(((0.5, 2.0), (0.5, 2.0), (-0.5, 0.5), (-0.5, 0.5))):
        P[f] = r.uniform(lo, hi, (ny, nx))
    got = []
    for tiles in (True, False):
        h = pkg.Handle(nx, ny)
        h.configure(6.0, float(ny), 1e9, 0.4, 1.9, 1.4, 0, precision)
        h.set_state_planes(P)
        if tiles:
            assert h.advance(2) == 2
            t = h.time()[0]
        else:
            t = sweeps(h, 2)
        got.append((t, h.get_state_planes()))
        h.close()
    assert got[0][0] == got[1][0] > 0
    assert np.isfinite(got[0][1]).all() and not np.array_equal(got[0][1], P)
    assert np.array_equal(got[0][1], got[1][1])
