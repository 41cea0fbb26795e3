"""The batch's host runtime over a stand-in for the CUDA runtime, without a GPU:
which plan its steps get, what the autotuner keeps, and what an error leaves."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "2d_fvm_cuda_b200", "csrc")


def build_over_fake_runtime(tmp, harness, sources):
    """A library of nvcc-compiled `sources` linked with `harness` in place of the
    CUDA runtime."""
    nvcc = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    cc = [nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC"]
    objs = []
    for s, flags in sources:
        objs.append(str(tmp / (os.path.basename(s) + ".o")))
        subprocess.run([*cc, *flags, "-c", os.path.join(CSRC, s), "-o", objs[-1]], check=True)
    so = str(tmp / (harness + ".so"))
    # (its own definitions first: another CUDA runtime may be loaded here)
    subprocess.run([*cc, "-shared", "-cudart", "none", "-Xlinker", "-Bsymbolic", os.path.join(HERE, harness), *objs,
                    "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    lib = build_over_fake_runtime(tmp_path_factory.mktemp("batch_runtime"), "batch_runtime_host.cpp",
                                  [("fvm2d_batch_host.cu", ())])
    lib.br_set.argtypes = [ctypes.c_double] * 3 + [ctypes.c_long, ctypes.c_int]
    lib.br_set.restype = lib.br_seen.restype = None
    lib.fvm2d_batch_set_problem.argtypes = [ctypes.c_void_p, ctypes.c_int] + [ctypes.c_double] * 6 + [ctypes.c_int]
    return lib


def seen(lib):
    out = (ctypes.c_long * 4)()
    lib.br_seen(out)
    return dict(zip(("tiles", "sweeps", "wrong_plan", "mixed"), out))


@pytest.fixture
def batch(lib):
    b = ctypes.c_void_p()
    sizes = (ctypes.c_int * 3)(40, 50, 60)
    assert lib.fvm2d_batch_create(ctypes.byref(b), 3, sizes, sizes) == 0
    for p, n in enumerate(sizes):
        cells = np.ones((n, n, 4))
        assert lib.fvm2d_batch_set_problem(b, p, 1.0, 1.0, 1.0, 0.4, 1.9, 1.4, 0) == 0
        assert lib.fvm2d_batch_set_state(b, p, ctypes.c_void_p(cells.ctypes.data), 4) == 0
    yield b
    lib.fvm2d_batch_destroy(b)


@pytest.mark.parametrize("apart", [0, 7])  # problems that end together, or one by one
def test_steps_follow_the_precision_set_last(lib, batch, apart):
    """Another precision of the same storage type has other tiles: its first step
    takes a plan of its own."""
    for precision in (0, 1, 0, 2, 3, 0):
        lib.br_set(2.0, 1.0, 0.0, -1, apart)
        assert lib.fvm2d_batch_set_precision(batch, precision) == 0
        assert lib.fvm2d_batch_solve(batch) == 0
        got = seen(lib)
        assert got["tiles"] > 0 and got["wrong_plan"] == 0 and got["mixed"] == 0, (precision, got)


def test_autotuning_times_no_first_run(lib, batch):
    """Tiles that are faster are kept although the process's first run, which is
    in tiles, costs more than any sweep."""
    lib.br_set(2.0, 1.0, 500.0, -1, 0)
    assert lib.fvm2d_batch_autotune(batch, 2, None, None) == 0
    lib.br_set(2.0, 1.0, 0.0, -1, 0)
    assert lib.fvm2d_batch_solve(batch) == 0
    assert seen(lib) == {"tiles": 20, "sweeps": 0, "wrong_plan": 0, "mixed": 0}
    lib.br_set(1.0, 2.0, 0.0, -1, 0)
    assert lib.fvm2d_batch_autotune(batch, 2, None, None) == 0
    lib.br_set(1.0, 2.0, 0.0, -1, 0)
    assert lib.fvm2d_batch_solve(batch) == 0
    assert seen(lib) == {"tiles": 0, "sweeps": 32, "wrong_plan": 0, "mixed": 0}


@pytest.mark.parametrize("trial", [0, 4, 17])
def test_a_failed_autotuning_leaves_the_batch_as_it_was(lib, batch, trial):
    """An error in any of the sweeps' trials is returned, and the next solve steps
    as the ones before."""
    lib.br_set(2.0, 1.0, 0.0, trial, 0)
    assert lib.fvm2d_batch_autotune(batch, 2, None, None) != 0
    lib.br_set(2.0, 1.0, 0.0, -1, 0)
    assert lib.fvm2d_batch_solve(batch) == 0
    assert seen(lib) == {"tiles": 20, "sweeps": 0, "wrong_plan": 0, "mixed": 0}


@pytest.mark.parametrize("n", [40, 2100])
def test_few_steps_are_enqueued_past_the_end(lib, n):
    b = ctypes.c_void_p()
    sizes = (ctypes.c_int * 1)(n)
    assert lib.fvm2d_batch_create(ctypes.byref(b), 1, sizes, sizes) == 0
    cells = np.ones((n, n, 4))
    assert lib.fvm2d_batch_set_problem(b, 0, 1.0, 1.0, 1.0, 0.4, 1.9, 1.4, 0) == 0
    assert lib.fvm2d_batch_set_state(b, 0, ctypes.c_void_p(cells.ctypes.data), 4) == 0
    for ends in (20, 3):  # steps to the end; a first group of 16 where steps are cheap
        lib.br_set(2.0, 1.0, 0.0, -1, 0)
        lib.br_ends(ends)
        assert lib.fvm2d_batch_solve(b) == 0
        assert ends <= seen(lib)["tiles"] <= (ends + 1 if n > 2000 else max(16, ends + 1))
    lib.br_ends(20)
    lib.fvm2d_batch_destroy(b)
