"""Writes fp32_cells.npz: cells of the single-precision builds on a B200, as the
tree whose root is the working folder computes them.  Recorded from the
package's first single-precision and batched builds, before steps were taken
in tiles; tests/test_fp32_bits_gpu.py holds every later build to them."""
import importlib
import os
import sys

import numpy as np

sys.path[:0] = [os.getcwd()]
CASES = [(31, 27, 0, 14), (34, 41, 4, 9), (29, 33, 6, 12)]  # nx, ny, preset, steps


def cells(pkg, nx, ny, preset):
    """A seeded four-quadrant state with every field varying."""
    r = np.random.default_rng([nx, ny, preset])
    U = pkg.scenarios.seeded_four_quadrant(nx, ny, 3 + preset)
    return U * (1 + 0.1 * r.uniform(-1, 1, U.shape))


def run(pkg):
    out = {}
    for nx, ny, preset, steps in CASES:
        U = cells(pkg, nx, ny, preset)
        for name, precision in (("fp32", pkg.FP32), ("residual", pkg.FP32_RESIDUAL)):
            h = pkg.Handle(nx, ny)
            h.configure(1.0, ny / nx, 1e9, 0.4, 1.9, 1.4, preset, precision)
            h.set_state(U)
            assert h.advance(steps) == steps
            out[f"{name}_{nx}x{ny}"] = h.get_state(4)
            out[f"{name}_{nx}x{ny}_t"] = h.time()[0]
            h.close()
    b = pkg.Batch([(nx, ny) for nx, ny, _, _ in CASES])
    b.set_precision(pkg.FP32)
    for p, (nx, ny, preset, steps) in enumerate(CASES):
        b.set_problem(p, width=1.0, height=ny / nx, t_end=0.9 * float(out[f"fp32_{nx}x{ny}_t"]), cfl=0.4, alpha=1.9,
                      gamma=1.4, strategy=preset)
        b.set_state(p, cells(pkg, nx, ny, preset))
    b.solve()
    for p, (nx, ny, _, _) in enumerate(CASES):
        out[f"batch_{nx}x{ny}"] = b.get_state(p)
        out[f"batch_{nx}x{ny}_t"] = b.time(p)[0]
    b.close()
    return out


if __name__ == "__main__":
    got = run(importlib.import_module("2d_fvm_cuda_b200"))
    # (single-precision values are kept as such)
    np.savez_compressed(sys.argv[1], **{k: np.float32(v) if not k.startswith("residual") and np.ndim(v) else v
                                        for k, v in got.items()})
