"""The single-precision builds give the bits they have always given (on a
B200): the midpoint flux jumps where a wave speed crosses zero, so a
rearranged sum can move isolated cells by 1e-4, far beyond rounding."""
import importlib.util
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def test_cells_are_the_recorded_ones(pkg):
    spec = importlib.util.spec_from_file_location("make_fp32_cells", os.path.join(GOLDEN, "make_fp32_cells.py"))
    make = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(make)
    got = make.run(pkg)
    with np.load(os.path.join(GOLDEN, "fp32_cells.npz")) as want:
        assert sorted(want.files) == sorted(got)
        for k in want.files:
            assert np.isfinite(want[k]).all(), k
            assert np.array_equal(got[k], want[k]), k
