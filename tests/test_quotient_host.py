"""Quotients from shared reciprocals (2d_fvm_cuda_b200/csrc/fvm2d_quotient.cuh)
compiled for the host, without a GPU: bit for bit those of division, alone and
in the interface flux and update that take them, on ordinary states of every
wave case and on ones out of the quotients' range, which divide."""
import ctypes

import numpy as np
import pytest

from test_kernels_host import build_host


@pytest.fixture(scope="module")
def qh(tmp_path_factory):
    lib = build_host(tmp_path_factory, "quotient_host.cpp")
    lib.qh_quotients.argtypes = [ctypes.c_void_p] * 2 + [ctypes.c_long] + [ctypes.c_void_p] * 2
    lib.qh_physics.argtypes = [ctypes.c_void_p, ctypes.c_long] + [ctypes.c_double] * 3 + [ctypes.c_void_p] * 2
    lib.qh_quotients.restype = lib.qh_physics.restype = None
    return lib


@pytest.mark.parametrize("spread", [0, 50, 1070])
def test_quotients_are_divisions(qh, spread):
    r = np.random.default_rng(spread)
    n = 400_000
    a = r.uniform(1, 2, n) * 2.0 ** r.integers(-spread, min(spread, 1020) + 1, n) * r.choice([-1.0, 1.0], n)
    b = r.uniform(1, 2, n) * 2.0 ** r.integers(-min(spread, 62), min(spread, 62) + 1, n)
    # mantissas near a power of two and quotients next to a rounding boundary
    b[::7] = np.nextafter(2.0 ** np.floor(np.log2(b[::7]) + 1), 0)
    k = slice(1, n, 5)
    m = np.round(r.uniform(2 ** 52, 2 ** 53, len(a[k]))) * 2 + 1  # a midpoint of two quotients, rounded
    a[k] = (m * 2.0 ** -53) * b[k]
    a[::11] = r.choice([0.0, -0.0], len(a[::11]))
    a[:6], b[:6] = [np.inf, np.nan, 5e-324, 1.0, 1.0, 1.0], [1.0, 1.0, 1.0, 0.0, np.nan, -2.0]
    taken, wrong = ctypes.c_long(0), ctypes.c_long(0)
    qh.qh_quotients(a.ctypes.data, b.ctypes.data, n, ctypes.byref(taken), ctypes.byref(wrong))
    assert wrong.value == 0
    assert taken.value >= (0.99 if spread < 60 else 0.5) * n
    assert taken.value <= n - 6  # the planted ones divide


@pytest.mark.parametrize("kind", ["smooth", "jumps", "supersonic", "vanishing", "broken"])
def test_interface_and_update_give_the_reference_order(qh, kind):
    r = np.random.default_rng(len(kind))
    n = 20_000
    h, dt = 1 / 400, 3e-4
    v = np.empty((n, 4, 4))
    v[:, :2, 0] = r.uniform(0.1, 2, (n, 2))
    v[:, :2, 1] = r.uniform(0.02, 2, (n, 2))
    v[:, :2, 2:] = r.uniform(-1.5, 1.5, (n, 2, 2))
    v[:, 2:] = r.uniform(-1, 1, (n, 2, 4)) * (0.05 / h)
    if kind == "smooth":
        v[:, 1] = v[:, 0] * (1 + 1e-3 * r.uniform(-1, 1, (n, 4)))
        v[::3, 2:] = 0.0
        v[::4, :2, 2] = 0.0
    elif kind == "supersonic":
        v[:, :2, 2] += r.choice([-800.0, -6.0, 6.0, 800.0], (n, 1))
    elif kind == "vanishing":
        v[:, :, 2:] *= 10.0 ** r.uniform(-320, -280, (n, 4, 1))
    elif kind == "broken":
        bad = r.choice([0.0, -1.0, np.nan, np.inf, -np.inf, 1e300, 1e-300, 5e-324], n)
        v.reshape(n, 16)[np.arange(n), r.integers(0, 16, n)] = bad
    wrong, shared = ctypes.c_long(0), ctypes.c_long(0)
    v = np.ascontiguousarray(v)
    qh.qh_physics(v.ctypes.data, n, 1.4, h, dt, ctypes.byref(wrong), ctypes.byref(shared))
    assert wrong.value == 0
    assert shared.value >= 0.99 * n if kind in ("smooth", "jumps", "supersonic") else shared.value < n
