// tile_host.cpp -- the step in tiles (2d_fvm_cuda_b200/csrc/fvm2d_tile.cuh)
// compiled for the host with g++ (built-ins emulated by cuda_host_emu.h), for
// tests/test_tile_host.py.
#include "cuda_host_emu.h"

#define FVM2D_VARIANT host
#define FVM2D_REAL double
#include "../2d_fvm_cuda_b200/csrc/fvm2d_tile.cuh"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_dual.cuh"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_adjoint.inc"

using namespace fvm2d::host;
using fvm2d::ad::Dual;

#include "kernels_host_steps.h"

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
        tile_step<double, Phys, T>(a, int(blockIdx.x), int(blockIdx.y), reinterpret_cast<unsigned char *>(smem.data()),
                                   [&] { return TileStep{0.0, dt, 1, 0}; }, false, v[threadIdx.x], b[threadIdx.x]);
    });
    *vmax = 0.0;
    *bad = 0;
    for (int t = 0; t < T::NT; ++t) {
        *vmax = std::fmax(*vmax, v[t]);
        *bad |= b[t];
    }
    return 0;
}

// A taped step in tiles against the taped sweeps, in the reference's order:
// returns the number of values that differ (bitwise) in X(U), Y(U), the four
// sweeps' fluxes where they are interfaces, the result's interior and the
// input's ring.  fill: the tiles get the input with its ring poisoned.
template <class T>
long tape(const double *cells, int nx, int ny, int strategy, double t, double dt, double width, double height, int fill)
{
    Planes<double> U(nx, ny), A1(nx, ny), B1(nx, ny), V(nx, ny), F[4] = {{nx, ny}, {nx, ny}, {nx, ny}, {nx, ny}};
    cells_to(U, cells, static_cast<const double *>(nullptr));
    forward_step<double, true, RefOrder>(U, A1, B1, V, F, strategy, t, dt, width / nx, height / ny, 1.9, 1.4, 16);
    auto poisoned = [&] {
        Planes<double> P(nx, ny);
        for (auto &x : P.v) x = NAN;
        return P;
    };
    Planes<double> S = U, a1 = poisoned(), b1 = poisoned(), v = poisoned(),
                   f[4] = {poisoned(), poisoned(), poisoned(), poisoned()};
    auto ring = [&](int i, int j) { return i < 2 || i >= nx - 2 || j < 2 || j >= ny - 2; };
    auto at = [&](const Planes<double> &P, int k, int i, int j) { return P.v[k * P.plane + (long long)j * nx + i]; };
    if (fill)
        for (int k = 0; k < 4; ++k)
            for (int j = 0; j < ny; ++j)
                for (int i = 0; i < nx; ++i)
                    if (ring(i, j)) S.v[k * S.plane + (long long)j * nx + i] = NAN;
    TileArgs<double> a;
    a.src = S.field();
    a.dst = v.field();
    a.nx = nx;
    a.ny = ny;
    a.hx = width / nx;
    a.hy = height / ny;
    a.rhx = 1.0 / a.hx;
    a.rhy = 1.0 / a.hy;
    a.alpha = 1.9;
    a.gamma = 1.4;
    a.ctl = nullptr;
    a.strategy = strategy;
    TapeArgs<double> tp{a1.field(), b1.field(), {f[0].field(), f[1].field(), f[2].field(), f[3].field()}};
    std::vector<double> smem((T::template bytes<double, RefOrder>() + 7) / 8, NAN);
    emu::launch(dim3((nx - 4 + T::TX - 1) / T::TX, (ny - 4 + T::TY - 1) / T::TY), dim3(T::NT), true, [&] {
        double vm = 0.0;
        int bad = 0;
        tile_step<double, RefOrder, T, true>(a, int(blockIdx.x), int(blockIdx.y),
                                             reinterpret_cast<unsigned char *>(smem.data()),
                                             [&] { return TileStep{t, dt, 1, 0}; }, fill != 0, vm, bad, &tp);
    });
    long diff = 0;
    auto same = [&](double x, double y) { diff += !(x == y); };
    for (int k = 0; k < 4; ++k)
        for (int j = 0; j < ny; ++j)
            for (int i = 0; i < nx; ++i) {
                same(at(S, k, i, j), at(U, k, i, j));
                same(at(a1, k, i, j), at(A1, k, i, j));
                same(at(b1, k, i, j), at(B1, k, i, j));
                if (!ring(i, j)) same(at(v, k, i, j), at(V, k, i, j));
                const bool col = i < 2 || i >= nx - 2, row = j < 2 || j >= ny - 2;
                const bool xi = i >= 2 && i <= nx - 2, yi = j >= 1 && j <= ny - 3;
                if (xi) same(at(f[0], k, i, j), at(F[0], k, i, j));
                if (yi) same(at(f[1], k, i, j), at(F[1], k, i, j));
                if (yi) same(at(f[2], k, i, j), col ? 0.0 : at(F[2], k, i, j));
                if (xi) same(at(f[3], k, i, j), row ? 0.0 : at(F[3], k, i, j));
            }
    return diff;
}

} // namespace

extern "C" long th_tape(int shape, const double *cells, int nx, int ny, int strategy, double t, double dt, double width,
                        double height, int fill)
{
    if (shape == 0) return tape<Tile<30, 30, 5>>(cells, nx, ny, strategy, t, dt, width, height, fill);
    if (shape == 1) return tape<Tile<30, 14, 3>>(cells, nx, ny, strategy, t, dt, width, height, fill);
    if (shape == 2) return tape<Tile<14, 14, 4>>(cells, nx, ny, strategy, t, dt, width, height, fill);
    return tape<Tile<14, 6, 2>>(cells, nx, ny, strategy, t, dt, width, height, fill);
}

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
