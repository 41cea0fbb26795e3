// tile_host.cpp -- the step in tiles (2d_fvm_cuda_b200/csrc/fvm2d_tile.cuh)
// compiled for the host with g++ (built-ins emulated by cuda_host_emu.h), for
// tests/test_tile_host.py.
#include "cuda_host_emu.h"

#define FVM2D_VARIANT host
#define FVM2D_REAL double
#include "../2d_fvm_cuda_b200/csrc/fvm2d_tile.cuh"

using namespace fvm2d::host;

namespace {

// The interior cells of one step of a (4, ny, nx) state, tile by tile; NaN
// stays where no tile writes.  *vmax: the written cells' largest wave speed.
template <class Phys, class T>
int step(const double *in, double *out, int nx, int ny, double width, double height, double dt, double alpha,
         double gamma, double *vmax, int *bad)
{
    const long long plane = (long long)nx * ny;
    TileArgs<double> a;
    a.src = Field<double>{const_cast<double *>(in), plane, nx};
    a.dst = Field<double>{out, plane, nx};
    a.nx = nx;
    a.ny = ny;
    a.hx = width / nx;
    a.hy = height / ny;
    a.rhx = 1.0 / a.hx;
    a.rhy = 1.0 / a.hy;
    a.alpha = alpha;
    a.gamma = gamma;
    a.ctl = nullptr;
    std::vector<double> smem((T::template bytes<double, Phys>() + 7) / 8, NAN);
    std::vector<double> v(T::NT, 0.0);
    std::vector<int> b(T::NT, 0);
    emu::launch(dim3((nx - 4 + T::TX - 1) / T::TX, (ny - 4 + T::TY - 1) / T::TY), dim3(T::NT), true, [&] {
        tile_step<double, Phys, T>(a, dt, int(blockIdx.x), int(blockIdx.y),
                                   reinterpret_cast<unsigned char *>(smem.data()), v[threadIdx.x], b[threadIdx.x]);
    });
    *vmax = 0.0;
    *bad = 0;
    for (int t = 0; t < T::NT; ++t) {
        *vmax = std::fmax(*vmax, v[t]);
        *bad |= b[t];
    }
    return 0;
}

} // namespace

extern "C" int th_step(int policy, int shape, const double *in, double *out, int nx, int ny, double width,
                       double height, double dt, double alpha, double gamma, double *vmax, int *bad)
{
    if (nx < 6 || ny < 6) return 1;
#define SHAPE(k, ...)                                                                                            \
    if (shape == k)                                                                                              \
        return policy == 0                                                                                       \
                   ? step<RefOrder, Tile<__VA_ARGS__>>(in, out, nx, ny, width, height, dt, alpha, gamma, vmax, bad) \
                   : step<Hoisted, Tile<__VA_ARGS__>>(in, out, nx, ny, width, height, dt, alpha, gamma, vmax, bad);
    SHAPE(0, 30, 30, 5)
    SHAPE(1, 30, 14, 3)
    SHAPE(2, 14, 14, 4)
    SHAPE(3, 14, 6, 2)
    return 2;
}
