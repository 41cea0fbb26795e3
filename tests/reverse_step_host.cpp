// reverse_step_host.cpp -- the kernels the reverse step launches
// (ghost_adjoint_gather, adjoint_pair_kernel, adjoint_add in
// 2d_fvm_cuda_b200/csrc/fvm2d_adjoint.inc) compiled for the host, against the
// ring's transpose as a scatter and one transpose at a time, for
// tests/test_reverse_step_host.py.
#include "cuda_host_emu.h"

#define FVM2D_VARIANT host
#define FVM2D_REAL double
#include "../2d_fvm_cuda_b200/csrc/fvm2d_kernels.cuh"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_dual.cuh"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_adjoint.inc"

using namespace fvm2d::host;
using fvm2d::ad::Dual;

#include "kernels_host_steps.h"

namespace {
long differ(const Planes<A> &a, const Planes<A> &b)
{
    long n = 0;
    for (size_t k = 0; k < a.v.size(); ++k) n += !(a.v[k] == b.v[k]);
    return n;
}
SweepT sweep(Planes<A> &U, Planes<A> &F, Planes<A> &ub, Planes<A> &out, double h, double dt)
{
    SweepT g;
    g.U = U.field();
    g.F = F.field();
    g.ub = ub.field();
    g.out = out.field();
    g.addend = Field<A>{nullptr, U.plane, U.nx};
    g.nx = U.nx;
    g.ny = U.ny;
    g.K = adjoint_consts(h, dt, 1.9, 1.4);
    return g;
}
} // namespace

extern "C" {
// Values in which ghost^T (p + q) / 2 by gathering and by scattering differ
// (whole p and q: every sum is exact).
long rs_ring(const double *p, const double *q, int nx, int ny, int strategy)
{
    Planes<A> P(nx, ny), Q(nx, ny), S(nx, ny), H(nx, ny), G(nx, ny);
    cells_to(P, p, nullptr);
    cells_to(Q, q, nullptr);
    for (size_t k = 0; k < P.v.size(); ++k) S.v[k] = P.v[k] + Q.v[k];
    for (auto &x : G.v) x = NAN;
    const GhostGeom g{nx, ny, strategy};
    const dim3 grid((nx + 31) / 32, (ny + 7) / 8), block(32, 8);
    emu::launch(grid, block, false, [&] { ghost_adjoint_gather(P.field(), Q.field(), G.field(), g, 0.5); });
    emu::launch(grid, block, false, [&] { ghost_adjoint_copy(S.field(), H.field(), g, 0.5); });
    const int ring = 4 * nx + 4 * (ny - 4);
    emu::launch(dim3((ring + 255) / 256), dim3(256), false, [&] { ghost_adjoint_scatter(S.field(), H.field(), g, 0.5); });
    return differ(G, H);
}

// Values in which the pair kernel's two transposes at one state differ from
// each alone, and adjoint_add's sum from the values'.
long rs_pair(const double *cells, const double *bx, const double *by, int nx, int ny, double h, double dt)
{
    Planes<A> U(nx, ny), A1(nx, ny), B1(nx, ny), V(nx, ny), F[4] = {{nx, ny}, {nx, ny}, {nx, ny}, {nx, ny}};
    cells_to(U, cells, nullptr);
    forward_step<A, true>(U, A1, B1, V, F, PERIODIC, 0.0, dt, h, h, 1.9, 1.4, 16);
    Planes<A> X(nx, ny), Y(nx, ny), ox(nx, ny), oy(nx, ny), px(nx, ny), py(nx, ny);
    cells_to(X, bx, nullptr);
    cells_to(Y, by, nullptr);
    for (auto &x : px.v) x = NAN;
    for (auto &x : py.v) x = NAN;
    transpose(0, U, F[0], X, ox, nullptr, h, dt, 1.9, 1.4);
    transpose(1, U, F[1], Y, oy, nullptr, h, dt, 1.9, 1.4);
    const SweepT gx = sweep(U, F[0], X, px, h, dt), gy = sweep(U, F[1], Y, py, h, dt);
    emu::launch(dim3(adjoint_x_blocks(nx, ny) + adjoint_y_blocks(nx, ny)), dim3(ANT), true,
                [&] { adjoint_pair_kernel(gx, gy); });
    long n = differ(px, ox) + differ(py, oy);
    for (size_t k = 0; k < ox.v.size(); ++k) ox.v[k] += oy.v[k];
    emu::launch(dim3((nx + 31) / 32, (ny + 7) / 8), dim3(32, 8), false,
                [&] { adjoint_add(px.field(), py.field(), nx, ny); });
    return n + differ(px, ox);
}
}
