// tall_grid_host.cpp -- the launches of the FP64 build's steps in tiles over a
// stand-in for the CUDA runtime (tests/test_tall_grid_host.py).
#include "fake_cudart.h"

#include "../2d_fvm_cuda_b200/csrc/fvm2d_control.h"

extern "C" {
// Enqueues a step (taped: a taped one) of an nx x ny array and its end; returns
// the first error.  blocks[0], blocks[1]: their blocks.
int tg_step(int nx, int ny, int taped, long long *blocks)
{
    fvm2d::LaunchConfig c{};
    c.nx = nx;
    c.ny = ny;
    c.pitch = (nx + 31) / 32 * 32;
    c.plane = (long long)c.pitch * ny;
    void *flux[4] = {};
    fake::launches.clear();
    if (cudaError_t e = fvm2d::fp64::prepare()) return e;
    if (cudaError_t e = taped ? fvm2d::fp64::enqueue_tile_step_taped(c, nullptr, flux, nullptr)
                              : fvm2d::fp64::enqueue_tile_step(c, nullptr))
        return e;
    if (cudaError_t e = fvm2d::fp64::enqueue_end_steps(c, nullptr)) return e;
    if (fake::launches.size() != 2) return -1;
    for (int k = 0; k < 2; ++k) {
        const dim3 g = fake::launches[k].grid;
        blocks[k] = (long long)g.x * g.y * g.z;
    }
    return 0;
}
}
