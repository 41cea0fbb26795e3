"""Steps in tiles on the GPU against the same steps taken sweep by sweep.

A solver of a whole problem steps in tiles; fvm2d_slab_step steps the same
state in place with the four sweep kernels.  Both inline the same arithmetic,
so the FP64 builds that leave the compiler no contraction give the same bits;
the others agree to rounding.  Sizes: smaller than a tile, one cell more or
less than a tile of each shape, several tiles; odd and even step counts (the
state ends in either buffer)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(6, 6), (7, 40), (17, 11), (34, 34), (35, 33), (48, 32), (65, 19), (130, 129), (257, 131), (400, 402),
         (611, 500)]
PRESETS = [0, 2, 3, 4, 5, 6]


def start(pkg, nx, ny, preset, precision, steps):
    """A solver with a seeded state, every field varying, and `steps` done."""
    rng = np.random.default_rng([nx, ny, preset])
    U = pkg.scenarios.seeded_four_quadrant(nx, ny, 3 + preset)
    U *= 1 + 0.1 * rng.uniform(-1, 1, U.shape)
    h = pkg.Handle(nx, ny)
    h.configure(1.0, ny / nx, 1e9, 0.4, 1.9, 1.4, preset, precision)
    h.set_state(U)
    assert h.advance(steps) == steps
    return h


def sweeps(h, n):
    """n steps in place, sweep by sweep; returns the time."""
    import torch

    a = torch.zeros(2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    h.slab_begin(a[0].data_ptr())
    for _ in range(n):
        h.slab_step(a[0].data_ptr(), a[0].data_ptr())
    return h.slab_sync()[0]


@pytest.mark.parametrize("precision", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_tiles_equal_sweeps(pkg, nx, ny, precision):
    presets = PRESETS if (nx, ny) in ((48, 32), (35, 33)) else [PRESETS[(nx + ny) % len(PRESETS)]]
    for preset in presets:
        for lead, n in ((1, 1), (2, 3)):
            a, b = (start(pkg, nx, ny, preset, precision, lead) for _ in range(2))
            S = a.get_state(4)
            assert np.array_equal(S, b.get_state(4), equal_nan=True)
            a.set_state(S)  # a run of its own from t = 0, as slab_begin starts one
            assert a.advance(n) == n
            t = sweeps(b, n)
            A, B = a.get_state(4), b.get_state(4)
            if precision in (0, 1):
                assert np.array_equal(A, B, equal_nan=True), (preset, n)
                assert a.time()[0] == t
            else:
                tol = 1e-12 if precision == 2 else 2e-5
                for f in range(4):
                    scale = np.nanmax(np.abs(B[..., f]))
                    assert np.nanmax(np.abs(A[..., f] - B[..., f])) <= tol * scale, (preset, n, f)
                assert a.time()[0] == pytest.approx(t, rel=1e-6)
            a.close()
            b.close()


@pytest.mark.parametrize("steps", [1, 2, 3, 5, 16, 21, 37, 150])
def test_any_step_count_and_restart(pkg, steps):
    """One advance equals the same steps one by one, and a solve, which ends
    within a group of enqueued steps, equals single steps up to its end time."""
    a, b = start(pkg, 97, 61, 0, pkg.FP64, steps), start(pkg, 97, 61, 0, pkg.FP64, 0)
    for _ in range(steps):
        assert b.advance(1) == 1
    assert a.time() == b.time()
    assert np.array_equal(a.get_state(4), b.get_state(4))
    t, _, dt = a.time()
    c, d = start(pkg, 97, 61, 0, pkg.FP64, 0), start(pkg, 97, 61, 0, pkg.FP64, 0)
    for h in (c, d):
        h.configure(1.0, 61 / 97, t + 0.4 * dt, 0.4, 1.9, 1.4, 0, pkg.FP64)  # ends in the middle of a step
    c.solve()
    while d.advance(1):
        pass
    assert c.time() == d.time() and c.time()[0] == t + 0.4 * dt
    assert np.array_equal(c.get_state(4), d.get_state(4))
    for h in (a, b, c, d):
        h.close()
