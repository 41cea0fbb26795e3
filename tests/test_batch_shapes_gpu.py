"""A batch whose large problems end early: the small ones go on with tiles of
another shape, and every problem equals its single solve."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# interior cells of 30 x 30 tiles enough for any build at first, then of few small ones
SIZES = [(420, 400)] * 10 + [(61, 47), (40, 73), (90, 33)]


@pytest.mark.parametrize("precision", [0, 1, 3])
def test_tiles_of_another_shape_after_some_problems_end(pkg, precision):
    b = pkg.Batch(SIZES)
    b.set_precision(precision)
    probs = []
    for p, (nx, ny) in enumerate(SIZES):
        U = pkg.scenarios.seeded_four_quadrant(nx, ny, 70 + p)
        kw = dict(width=1.0, height=ny / nx, t_end=0.004 + 0.0002 * p if nx == 420 else 0.12 + 0.01 * p, cfl=0.45,
                  alpha=1.9, gamma=1.4, strategy=(0, 6, 5)[p % 3] if nx < 420 else 0)
        b.set_problem(p, **kw)
        b.set_state(p, U)
        probs.append((U, kw))
    b.solve()
    large, small = [], []
    for p, (U, kw) in enumerate(probs):
        h = pkg.Handle(U.shape[1], U.shape[0])
        h.configure(*kw.values(), precision)
        h.set_state(U)
        h.solve()
        A, B = b.get_state(p), h.get_state(4)
        (large if U.shape[1] == 420 else small).append(b.time(p)[1])
        if precision == 3:  # one rounding along y is the batch's own
            assert np.abs(A - B).sum() <= 2e-4 * np.abs(B).sum(), p
        else:
            assert b.time(p) == h.time()[:2] and np.array_equal(A, B), p
        h.close()
    b.close()
    assert max(large) + 16 < min(small)  # whole groups of steps were theirs alone
