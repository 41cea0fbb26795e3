"""A batch that changes its precision between solves steps every tile of every
problem: each solve equals that of a batch made with its precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_precision_changed_between_solves(pkg):
    sizes = [(200, 200)] * 4  # (the FP64 build's 14 x 14 tiles, 30 x 14 in others)
    # (one state: problems that end together leave no list to be made again)
    U = [pkg.scenarios.seeded_four_quadrant(nx, ny, 40) for nx, ny in sizes]

    def batch(precision):
        b = pkg.Batch(sizes)
        b.set_precision(precision)
        for p in range(len(sizes)):
            b.set_problem(p, width=1.0, height=1.0, t_end=0.01, cfl=0.4, alpha=1.9, gamma=1.4, strategy=0)
        return b

    def solve(b):
        for p, u in enumerate(U):
            b.set_state(p, u)
        b.solve()
        return [b.get_state(p) for p in range(len(sizes))]

    changing = batch(pkg.FP64_STRICT)
    for precision in (pkg.FP64_STRICT, pkg.FP64, pkg.FP64_REFORDER, pkg.FP32, pkg.FP64, pkg.FP64_STRICT):
        changing.set_precision(precision)
        b = batch(precision)
        for A, B in zip(solve(changing), solve(b)):
            assert np.array_equal(A, B), precision
        b.close()
    changing.close()
