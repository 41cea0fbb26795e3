"""The single-precision adjoint takes the forward's side of the contact, without
a GPU: the midpoint flux jumps where the contact speed crosses zero, so a
reverse that rounds the speed otherwise differentiates the wrong side.  The
interfaces here have contact speeds of a few rounding units around zero."""
import ctypes

import numpy as np
import pytest

from test_kernels_host import build_host


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_adjoint_takes_the_forwards_side(tmp_path_factory, seed):
    lib = build_host(tmp_path_factory, "fp32_sides_host.cpp")
    lib.fs_sides.argtypes = [ctypes.c_void_p, ctypes.c_long] + [ctypes.c_double] * 4 + [ctypes.c_void_p] * 2
    lib.fs_sides.restype = None
    r = np.random.default_rng(seed)
    n, h = 100_000, 1 / 400
    v = np.empty((n, 4, 4), np.float32)
    v[:, 0, 0], v[:, 1, 0] = r.uniform(0.5, 2, (2, n))
    v[:, 0, 1] = r.uniform(0.5, 2, n)
    v[:, 1, 1] = v[:, 0, 1] * (1 + r.integers(-2, 3, n) * 2.0 ** -23)
    v[:, :2, 2] = r.uniform(-1, 1, (n, 2)) * 2.0 ** -23
    v[:, :2, 3] = r.uniform(-1, 1, (n, 2))
    v[:, 2:] = r.uniform(-1, 1, (n, 2, 4))
    v[:, 2:, 0:3] *= 2.0 ** -14  # faces that differ from the cells by about a rounding unit
    taken, wrong = np.zeros(2, np.int64), ctypes.c_long(0)
    lib.fs_sides(v.ctypes.data, n, h, 1e-3, 1.9, 1.4, taken.ctypes.data, ctypes.byref(wrong))
    assert taken.sum() == n and taken.min() > n // 4
    assert wrong.value == 0
