// tile_chain_host.cpp -- steps in tiles with the records that hand them on
// (begin_tile, fold_record, end_tile, commit_record in
// 2d_fvm_cuda_b200/csrc/fvm2d_tile.cuh), and single-precision tiles, compiled
// for the host, for tests/test_tile_chain_host.py.
#include "cuda_host_emu.h"

#define FVM2D_VARIANT host
#define FVM2D_REAL double
#include "../2d_fvm_cuda_b200/csrc/fvm2d_tile.cuh"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_dual.cuh"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_adjoint.inc"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_packed.cuh"

using namespace fvm2d::host;
using fvm2d::StepControl;
using fvm2d::TileRecord;
using fvm2d::ad::Dual;

#include "kernels_host_steps.h"

namespace {
using T = Tile<14, 6, 3>;

template <typename R>
TileArgs<R> args(R *src, R *dst, int nx, int ny, double width, double height, int strategy)
{
    const long long plane = (long long)nx * ny;
    TileArgs<R> a;
    a.src = Field<R>{src, plane, nx};
    a.dst = Field<R>{dst, plane, nx};
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
    return a;
}
template <class S>
dim3 tiles(int nx, int ny)
{
    return dim3((nx - 4 + S::TX - 1) / S::TX, (ny - 4 + S::TY - 1) / S::TY);
}

// One step of FP32 planes (SPLIT: with residuals), by sweeps and by tiles of
// shape S: the interior values that differ bitwise.
template <class Phys, class S, bool SPLIT>
long single(const double *cells, int nx, int ny, double width, double height, double dt)
{
    const long long plane = (long long)nx * ny;
    const size_t n = (SPLIT ? 6 : 4) * plane;
    std::vector<float> U(n), A(n), B(n), V(n), W(n, NAN);
    for (long long c = 0; c < plane; ++c)
        for (int f = 0; f < 4; ++f) {
            if (SPLIT)
                fvm2d::split_value(cells[4 * c + f], U[f * plane + c],
                                   reinterpret_cast<unsigned short *>(U.data() + 4 * plane)[4 * c + f]);
            else
                U[f * plane + c] = float(cells[4 * c + f]);
        }
    auto sweep = [&](std::vector<float> &s, std::vector<float> &d, double h) {
        SweepArgs<float> a;
        a.src = Field<float>{s.data(), plane, nx};
        a.dst = a.comb = Field<float>{d.data(), plane, nx};
        a.flux = Field<float>{nullptr, plane, nx};
        a.nx = nx;
        a.ny = ny;
        a.h = h;
        a.rh = 1.0 / h;
        a.alpha = 1.9;
        a.gamma = 1.4;
        a.ctl = nullptr;
        a.xchunks = 2;
        return a;
    };
    auto x = [&](std::vector<float> &s, std::vector<float> &d, auto last) {
        const SweepArgs<float> a = sweep(s, d, width / nx);
        const SweepConsts<float> K = sweep_consts(a, dt);
        const int nseg = fvm2d::x_items_per_row(nx, a.xchunks);
        emu::launch(dim3(1), dim3(32), true, [&] {
            double vmax = 0.0;
            int bad = 0;
            for (int w = 0; w < nseg * ny; ++w)
                x_item<float, Phys, decltype(last)::value>(a, K, w / nseg, w % nseg, nseg, int(threadIdx.x), vmax, bad);
        });
    };
    auto y = [&](std::vector<float> &s, std::vector<float> &d) {
        const SweepArgs<float> a = sweep(s, d, height / ny);
        const SweepConsts<float> K = sweep_consts(a, dt);
        for (int seg = 0; seg < y_segments(ny, 16); ++seg)
            for (int cw = 0; cw < (nx + 31) / 32; ++cw)
                for (int lane = 0; lane < 32; ++lane) y_item<float, Phys>(a, K, seg, y_segments(ny, 16), cw, lane, 16);
    };
    x(U, A, std::false_type());
    y(U, B);
    y(A, V);
    x(B, V, std::true_type());
    const TileArgs<float> a = args(U.data(), W.data(), nx, ny, width, height, 0);
    std::vector<double> smem((S::template bytes<float, Phys>() + 7) / 8, NAN);
    emu::launch(tiles<S>(nx, ny), dim3(S::NT), true, [&] {
        double vmax = 0.0;
        int bad = 0;
        tile_step<float, Phys, S>(a, int(blockIdx.x), int(blockIdx.y), reinterpret_cast<unsigned char *>(smem.data()),
                                  [&] { return TileStep{0.0, dt, 1, 0}; }, false, vmax, bad);
    });
    long diff = 0;
    for (int j = 2; j < ny - 2; ++j)
        for (int i = 2; i < nx - 2; ++i) {
            const long long c = (long long)j * nx + i;
            for (int f = 0; f < 4; ++f) diff += !(V[f * plane + c] == W[f * plane + c]);
            if (SPLIT)
                diff += reinterpret_cast<unsigned long long *>(V.data() + 4 * plane)[c] !=
                        reinterpret_cast<unsigned long long *>(W.data() + 4 * plane)[c];
        }
    return diff;
}
} // namespace

extern "C" {
// A run from t = 0 as the solver enqueues it: the first plan, then groups of
// `group` steps in tiles, each ended as end_steps_kernel ends it, until no step
// is in flight or `groups` have run.  out: the state; record: t, dt, steps,
// done, first bad step.
int tc_run(const double *cells, int nx, int ny, double width, double height, double t_end, double cfl, int limit,
           int strategy, int group, int groups, double *out, double *record)
{
    Planes<double> P[2] = {{nx, ny}, {nx, ny}};
    cells_to(P[0], cells, nullptr);
    for (auto &x : P[1].v) x = NAN;
    StepControl ctl{};
    ctl.step_limit = limit;
    fvm2d::PlanParams plan{t_end, cfl, std::fmin(width / nx, height / ny), 0.0};
    for (long long k = 0; k < P[0].plane; ++k) {
        const double *v = P[0].v.data();
        ctl.smax_last = std::fmax(ctl.smax_last, wave_speed(v[k], v[P[0].plane + k], v[2 * P[0].plane + k],
                                                            v[3 * P[0].plane + k], 1.4));
    }
    plan_step(&ctl, plan);
    open_record(&ctl);
    std::vector<double> smem((T::bytes<double, RefOrder>() + 7) / 8, NAN);
    for (int g = 0; g < groups && ctl.active; ++g) {
        const int parity = ctl.parity;
        for (int k = 0; k < group; ++k) {
            const int now = (parity + k) & 1;
            TileArgs<double> a =
                args(P[now].v.data(), P[now ^ 1].v.data(), nx, ny, width, height, strategy);
            a.ctl = &ctl;
            a.plan = plan;
            emu::launch(tiles<T>(nx, ny), dim3(T::NT), true, [&] {
                const bool first = blockIdx.x == 0 && blockIdx.y == 0;
                double vmax = first && threadIdx.x == 0 ? ring_speed<double>(strategy, 1.4) : 0.0;
                int bad = 0;
                unsigned char *const s = reinterpret_cast<unsigned char *>(smem.data());
                if (tile_step<double, RefOrder, T>(a, int(blockIdx.x), int(blockIdx.y), s,
                                                   [&] { return begin_tile(a.ctl, k & 1, plan, first); }, k > 0, vmax, bad))
                    end_tile<T::NT>(vmax, bad, &ctl, reinterpret_cast<TileHead<double, RefOrder> *>(s)->step.steps);
            });
        }
        const TileRecord r = fold_record(&ctl, group & 1, plan);
        if (r.ring_due) {
            TileArgs<double> a = args(P[r.parity].v.data(), P[r.parity].v.data(), nx, ny, width, height, strategy);
            a.ctl = &ctl;
            a.plan = plan;
            for (int k = 0; k < 4 * nx + 4 * (ny - 4); ++k) ghost_cell(ring_args(a), k, r.t);
        }
        commit_record(&ctl, r);
    }
    const Planes<double> &S = P[ctl.parity];
    for (long long c = 0; c < S.plane; ++c)
        for (int f = 0; f < 4; ++f) out[4 * c + f] = S.v[f * S.plane + c];
    record[0] = ctl.t;
    record[1] = ctl.dt;
    record[2] = ctl.steps;
    record[3] = ctl.done;
    record[4] = ctl.first_bad;
    return ctl.active;
}

// physics 0 the FP32 build's, 1 the batch's, 2 the residual build's
long tc_single(int physics, int shape, const double *cells, int nx, int ny, double width, double height, double dt)
{
    using S0 = Tile<30, 30, 5>;
    using S1 = Tile<14, 14, 4>;
#define ON(P, SPLIT) \
    (shape ? single<P, S1, SPLIT>(cells, nx, ny, width, height, dt) : single<P, S0, SPLIT>(cells, nx, ny, width, height, dt))
    return physics == 0 ? ON(PackedCompensated, false) : physics == 1 ? ON(PackedBatch, false) : ON(PackedResidual, true);
}
}
