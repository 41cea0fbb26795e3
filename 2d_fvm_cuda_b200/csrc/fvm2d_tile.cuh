// fvm2d_tile.cuh -- a whole split step of one tile of the array per block.
//
// A block takes a tile of TX x TY cells it will write, loads it with two
// cells around it (the reach of a sweep) into shared memory, and runs both
// split orders there:
//
//   phase 0   X(U) on the tile's columns of every loaded row -> A1, and
//             Y(U) on the tile's rows of every loaded column -> B1
//   phase 1   Y(A1) on the tile -> RA (over U, which is dead)
//   phase 2   X(B1) on the tile, averaged with RA, wave-speed maximum and
//             health test, result to global memory
//
// The smaller shapes, which serve arrays whose steps are a chain of latencies,
// take the tasks of phases 1 and 2 together (X(B1) -> RB) and average after
// one more barrier: 14 x 6 tiles then run two rounds of tasks instead of
// three.
//
// A step leaves its wave-speed maximum; the blocks of the next one each
// commit it and plan for themselves (fold_record) while their tiles are on
// the way, and the end of a group of steps does so once more
// (end_steps_kernel).  A fence, a ticket and the plan in a step's last block,
// with the record read before the tile by the next step, measured 8.1 us per
// step at 100^2 against 6.8, 6.9 against 5.4 at 48^2.  The ghost ring is not
// stored between steps: a tile that loads ring cells of a state stepped to in
// tiles computes them from their interior sources (ring_value);
// end_steps_kernel stores the ring.  A ring cell's wave speed is its source's,
// which is in the maximum, or an inflow constant's (ring_speed).
//
// So the four sweeps' intermediate states never leave the SM: 64 bytes per
// FP64 cell and step in place of 288, one launch in place of five.  Work on
// the two halo cells is done again by the neighbouring tiles (30 x 30: 128 warp
// tasks where four sweeps of 900 cells fill 112.5: 14%), which the shorter
// instruction stream (no global addresses, clamps, carries or ring copies per
// sweep: 433 slots per task of 32 interfaces, in the quadrants at 2048^2,
// against 460-650 per 32 cells of a sweep kernel) repays even where the array is
// large.  What bounds a tile is FP64 latency and issue: FP64 pipe 57%, issue
// slots 61% busy at 20 warps per SM.
//
// Against the sweep kernels with the same arithmetic (FP64,
// us per step of a varied four-quadrant flow): 400^2 58 -> 27, 131 x 517
// 48 -> 16, 1003^2 164 -> 111, 4096^2 1810 -> 1600; FP32 4096^2 1270 -> 1200.
//
// A warp task is 32 interfaces, one per lane: a lane holds cell c of a line,
// computes its limited slope, takes the slope of c-1 from its neighbour by
// shuffle, computes the interface c-1/2, takes the flux of c-3/2 by shuffle
// and updates c-1.  A line of T updated cells takes T + 2 lanes, so T is 30,
// 14 or 6 (1, 2 or 4 lines per warp).  Lines along x and along y run the same
// code with another stride between cells.
//
// Shared memory holds rows of four fields (RS elements apart, an odd number,
// so that lanes along a column meet no bank conflict).
#pragma once

#include "fvm2d_kernels.cuh"

namespace fvm2d {
namespace FVM2D_VARIANT {

// A direction's constants with the products its tasks use, in shared memory.
template <typename Real>
struct TileConsts : SweepConsts<Real> {
    Real hh, hrh, rha, hk;
};
// and dt/h, 1/(gamma-1) and gamma-1 joined, for the FP64 update of a residual
// build: six conversions a task less.  (Padded so that each direction's
// constants start on 16 bytes: FP64 and FP32 steps measured 1% slower where
// they do not.)
template <typename Real>
struct JoinedConsts : TileConsts<Real> {
    double lambda, igm1, gm1, pad;
};
template <typename Real>
__device__ __forceinline__ Real half_h(const TileConsts<Real> &K) { return K.hh; }
template <typename Real>
__device__ __forceinline__ Real half_rh(const TileConsts<Real> &K) { return K.hrh; }
template <typename Real>
__device__ __forceinline__ Real alpha_rh(const TileConsts<Real> &K) { return K.rha; }
template <typename Real>
__device__ __forceinline__ Real half_k(const TileConsts<Real> &K) { return K.hk; }
template <typename Real>
__device__ __forceinline__ double joined_lambda(const JoinedConsts<Real> &K) { return K.lambda; }
template <typename Real>
__device__ __forceinline__ double joined_igm1(const JoinedConsts<Real> &K) { return K.igm1; }
template <typename Real>
__device__ __forceinline__ double joined_gm1(const JoinedConsts<Real> &K) { return K.gm1; }

// The step a block runs, from its control record.
struct TileStep {
    double t, dt;
    int active, steps;  // steps committed before it
};

// What comes first in a block's shared memory.
template <typename Real, class Phys>
struct TileHead {
    using Consts = std::conditional_t<split_storage<Phys>::value, JoinedConsts<Real>, TileConsts<Real>>;
    Consts K[2];  // along x, along y
    TileStep step;
    double pad;
};

template <typename Real>
struct TileArgs {
    Field<Real> src, dst;  // state read and state written (different buffers)
    int nx, ny;
    double hx, hy, rhx, rhy;
    double alpha, gamma;
    StepControl *ctl;
    int strategy;
    PlanParams plan;
};

// What a taped step keeps for its adjoint besides its input state: X(U), Y(U)
// and the interface fluxes of X(U), Y(U), Y(A1) and X(B1), each at the
// interface's right cell in planes mass, normal momentum, energy, tangential
// momentum.  The second sweeps' fluxes on the ring, where nothing is updated,
// are stored as 0.
template <typename Real>
struct TapeArgs {
    Field<Real> A1, B1, F[4];
};

template <typename Real>
__device__ __forceinline__ GhostArgs<Real> ring_args(const TileArgs<Real> &a)
{
    GhostArgs<Real> g;
    g.U = a.src;
    g.nx = a.nx;
    g.ny = a.ny;
    g.strategy = a.strategy;
    g.gamma = a.gamma;
    g.ctl = a.ctl;
    g.plan = a.plan;
    g.row0 = 0;
    g.gny = a.ny;
    g.fill_top = g.fill_bottom = 1;
    return g;
}

// Ring cell (i, j) of a state at time t, from the state's interior.
template <typename Real>
__device__ __forceinline__ Cell<Real> ring_value(const GhostArgs<Real> &g, int i, int j, double t)
{
    return i < 2 || i >= g.nx - 2 ? col_rule(g, i, j, t) : row_rule(g, i, j, t);
}

// The largest wave speed of the ring cells that copy no interior cell: the
// inflow states of the presets that have them, each of which is on the ring
// of any array (the left columns' at least).
template <typename Real>
__device__ __forceinline__ double ring_speed(int strategy, double gamma)
{
    auto speed = [&](double r, double p, double u, double v) {
        const Cell<Real> c = mk<Real>(r, p, u, v);
        return wave_speed(c.rho, c.p, c.un, c.ut, gamma);
    };
    switch (strategy) {
    case OUTFLOW:
    case PERIODIC:
    case REFLECTIVE_TB:
        return 0.0;
    case JET:
        return fmax(speed(5.0, 0.4127, 800.0, 0.0), speed(0.5, 0.4127, 0.0, 0.0));
    case JET800:
        return fmax(speed(1.4, 1, 800, 0), speed(0.14, 1, 0, 0));
    default:
        return fmax(speed(8, 116.5, 4.125 * sqrt(3.0), -4.125), speed(1.4, 1, 0, 0));
    }
}

// Geometry of a tile: TX x TY written cells, NW warps.
template <int TX_, int TY_, int NW_>
struct Tile {
    static constexpr int TX = TX_, TY = TY_, NW = NW_, NT = 32 * NW_;
    static constexpr int SX = TX + 2, SY = TY + 2;    // lanes per line
    static constexpr int RX = 32 / SX, CY = 32 / SY;  // lines per warp task
    static constexpr int NC = TX + 4, NR = TY + 4;    // loaded columns, rows
    static constexpr int RS = 4 * NC + 1;             // elements between rows
    static_assert(32 % SX == 0 && 32 % SY == 0, "a line takes 8, 16 or 32 lanes");
    // phases 1 and 2 together (30 x 30 has no shared memory left for RB)
    static constexpr bool kMerge = TX * TY < 900;
    // U, A1: NR rows; B1, RB: TY rows
    static constexpr int kRows = 2 * NR + TY + (kMerge ? TY : 0);
    static constexpr int kElems = kRows * RS;
    static constexpr int kLo = NC | 1;                // residual words per row
    static constexpr int kLoWords = (2 * NR + TY) * kLo;
    template <typename Real, class Phys>
    static constexpr size_t bytes()
    {
        return sizeof(TileHead<Real, Phys>) + (kElems + 1) / 2 * 2 * sizeof(Real) +
               (split_storage<Phys>::value ? kLoWords * sizeof(unsigned long long) : 0);
    }
};

template <typename Real>
__device__ __forceinline__ void tile_copy(Real *dst_shared, const Real *src)
{
    if constexpr (sizeof(Real) == 4 || sizeof(Real) == 8)
        async_copy(dst_shared, src);
    else
        *dst_shared = *src;
}

// Do the presets' ring values depend on time?  (row_rule: the rows above a
// double Mach reflection)
__device__ __forceinline__ bool ring_timed(int strategy)
{
    return !(strategy == OUTFLOW || strategy == PERIODIC || strategy == REFLECTIVE_TB || strategy == JET ||
             strategy == JET800);
}

// One step of tile (bx, by), by the Tile::NT threads of a block; false, and
// nothing written, if there is none to run.  begin(): the step, called by the
// last warp while the copies of the tile are under way (the record's loads
// and the plan's divisions then cost a step nothing), or before them where
// ring cells depend on its time.  fill: the state's ring cells are computed,
// else read.  TAPE: the step also writes its tape (and the ring it fills,
// into the state it reads).
template <typename Real, class Phys, class T, bool TAPE = false, class Begin>
__device__ __forceinline__ bool tile_step(const TileArgs<Real> &a, int bx, int by, unsigned char *smem, Begin &&begin,
                                          bool fill, double &vmax, int &bad, const TapeArgs<Real> *tape = nullptr)
{
    constexpr bool kResidual = split_storage<Phys>::value;
    using Word = unsigned long long;
    constexpr int NC = T::NC, RS = T::RS;
    // (a residual build's branch B is averaged before it is split)
    constexpr bool MERGE = T::kMerge && !kResidual;
    using Head = TileHead<Real, Phys>;
    using Consts = typename Head::Consts;
    Head *const head = reinterpret_cast<Head *>(smem);
    Consts *const KK = head->K;
    Real *const sU = reinterpret_cast<Real *>(head + 1);
    Real *const sA = sU + T::NR * RS;
    Real *const sB = sA + (T::NR - 2) * RS;  // rows 2 .. TY+1 of B1 (rows 0, 1 are not kept)
    Real *const sR = sB + T::TY * RS;        // the same rows of RB
    Word *const lU = reinterpret_cast<Word *>(sU + (T::kElems + 1) / 2 * 2);
    Word *const lA = lU + T::NR * T::kLo, *const lB = lA + (T::NR - 2) * T::kLo;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid & 31;
    const int x0 = 2 + bx * T::TX, y0 = 2 + by * T::TY;  // first written cell
    const int ncol = min(NC, a.nx - x0 + 2), nrow = min(T::NR, a.ny - y0 + 2);  // loaded columns and rows in the array

    // TAPE: the cells whose tape this tile writes -- its own and, at an edge of
    // the array, the ring's beside them
    const bool last_x = x0 + T::TX > a.nx - 3, last_y = y0 + T::TY > a.ny - 3;
    auto owns_x = [&](int x) { return (x >= x0 || bx == 0) && (x < x0 + T::TX || last_x); };
    auto owns_y = [&](int y) { return (y >= y0 || by == 0) && (y < y0 + T::TY || last_y); };
    const Cell<Real> none = {Real(0), Real(0), Real(0), Real(0)};
    auto start = [&] {
        const TileStep now = begin();
        if (lane == 0) head->step = now;
        if (lane >= 2) return;
        Consts C;
        TileConsts<Real> &K = C;
        const double h = lane == 0 ? a.hx : a.hy;
        K.h = Real(h);
        K.rh = Real(lane == 0 ? a.rhx : a.rhy);
        K.alpha = Real(a.alpha);
        set_gamma_consts(K, a.gamma);
        K.k = Real(now.dt);
        K.lambda = Real(now.dt / h);
        K.lambda_lo = Real(lo_part<Real>(now.dt / h));
        K.hh = K.h * Real(0.5);
        K.hrh = K.rh * Real(0.5);
        K.rha = K.rh * K.alpha;
        K.hk = K.k * Real(0.5);
        if constexpr (kResidual) {
            C.lambda = joined_lambda(K);
            C.igm1 = joined_igm1(K);
            C.gm1 = joined_gm1(K);
        }
        KK[lane] = C;
    };
    const bool timed = fill && by == 0 && ring_timed(a.strategy);
    if (timed) {
        if (warp == T::NW - 1) start();
        __syncthreads();
    }
    const double t = timed ? head->step.t : 0.0;
    // does the loaded tile reach the ring?
    const bool edge = fill && (bx == 0 || by == 0 || x0 - 2 + NC > a.nx - 2 || y0 - 2 + T::NR > a.ny - 2);
    for (int i = tid; i < T::NR * NC; i += T::NT) {
        const int r = i / NC, c = i - r * NC;
        if (r >= nrow) break;
        const int x = min(x0 - 2 + c, a.nx - 1), y = y0 - 2 + r;
        Real *const q = sU + r * RS + c;
        if (edge && (x < 2 || x >= a.nx - 2 || y < 2 || y >= a.ny - 2)) {
            const Cell<Real> v = ring_value(ring_args(a), x, y, t);
            q[0] = v.rho;
            q[NC] = v.p;
            q[2 * NC] = v.un;
            q[3 * NC] = v.ut;
            if constexpr (kResidual) lU[r * T::kLo + c] = 0ull;  // a ring cell holds its FP32 value exactly
            if (TAPE && x0 - 2 + c < a.nx && owns_x(x) && owns_y(y)) store_cell(a.src, x, y, 2, 3, v);
            continue;
        }
        tile_copy(q, &a.src.at(0, x, y));
        tile_copy(q + NC, &a.src.at(1, x, y));
        tile_copy(q + 2 * NC, &a.src.at(2, x, y));
        tile_copy(q + 3 * NC, &a.src.at(3, x, y));
        if constexpr (kResidual) async_copy(lU + r * T::kLo + c, &lo_cell(a.src, x, y));
    }
    async_commit();
    if (!timed && warp == T::NW - 1) start();
    async_wait<0>();
    __syncthreads();
    if (!head->step.active) return false;
    if constexpr (TAPE) {  // the ring's part: sweeps across it pass its cells through
        for (int i = tid; i < T::NR * NC; i += T::NT) {
            const int r = i / NC, c = i - r * NC, x = x0 - 2 + c, y = y0 - 2 + r;
            const bool col = x < 2 || x >= a.nx - 2, row = y < 2 || y >= a.ny - 2;
            if (!(col || row) || x >= a.nx || y >= a.ny || !owns_x(x) || !owns_y(y)) continue;
            const Real *const q = sU + r * RS + c;
            const Cell<Real> v = {q[0], q[NC], q[2 * NC], q[3 * NC]};
            if (col) {
                store_cell(tape->A1, x, y, 2, 3, v);
                store_cell(tape->F[2], x, y, 2, 3, none);
            }
            if (row) {
                store_cell(tape->B1, x, y, 2, 3, v);
                store_cell(tape->F[3], x, y, 2, 3, none);
            }
        }
    }

    // branch A's result at tile cell (r, c)
    auto branch_a = [&](int r, int c) {
        const Real *const ra = sU + r * RS + c;
        const Cell<Real> A = {ra[0], ra[NC], ra[2 * NC], ra[3 * NC]};
        if constexpr (kResidual)
            return join_cell(A, lo_parts(lU[r * T::kLo + c], false));
        else
            return A;
    };
    // the step's result there: branch A averaged with branch B in primitive
    // variables (src/basicFuns.cuh:264-274); residual builds: averaged already
    auto finish = [&](int r, int c, auto b) {
        const int x = x0 - 2 + c, y = y0 - 2 + r;
        Cell<Real> o;
        if constexpr (kResidual) {
            o = store_split(a.dst, x, y, 2, 3, b);
        } else {
            const Cell<Real> A = branch_a(r, c);
            o.rho = (A.rho + b.rho) * Real(0.5);
            o.p = (A.p + b.p) * Real(0.5);
            o.un = (A.un + b.un) * Real(0.5);
            o.ut = (A.ut + b.ut) * Real(0.5);
            store_cell(a.dst, x, y, 2, 3, o);
        }
        vmax = fmax(vmax, wave_speed(o.rho, o.p, o.un, o.ut, a.gamma));
        bad |= !(o.rho > Real(0) && o.p > Real(0));  // NaN fails both tests
    };

    // tasks along x and along y of the two sweeps of each branch
    const int nx0 = (nrow + T::RX - 1) / T::RX, ny0 = (ncol + T::CY - 1) / T::CY;
    const int ny1 = (ncol - 4 + T::CY - 1) / T::CY, nx1 = (nrow - 4 + T::RX - 1) / T::RX;
    for (int phase = 0; phase < (MERGE ? 2 : 3); ++phase) {
        const int ntask = phase == 0 ? nx0 + ny0 : MERGE ? ny1 + nx1 : phase == 1 ? ny1 : nx1;
        for (int t = warp; t < ntask; t += T::NW) {
            const bool xdir = phase == 0 ? t < nx0 : MERGE ? t >= ny1 : phase == 2;
            // this lane's cell: row r, column c of the loaded tile; k its place on the line
            int k, r, c, s;
            bool mine;
            if (xdir) {
                k = lane & (T::SX - 1);
                const int line = (MERGE && phase ? t - ny1 : t) * T::RX + lane / T::SX;
                const int n = phase == 0 ? nrow : nrow - 4;
                mine = line < n;
                r = min(line, n - 1) + (phase == 0 ? 0 : 2);
                c = k + 1;
                s = 1;
            } else {
                k = lane & (T::SY - 1);
                const int line = (phase == 0 ? t - nx0 : t) * T::CY + lane / T::SY, n = phase == 0 ? ncol : ncol - 4;
                mine = line < n;
                c = min(line, n - 1) + (phase == 0 ? 0 : 2);
                r = T::TY + 2 - k;  // lines along y start at the bottom (u_n = v)
                s = -RS;
            }
            const Real *const from = phase == 0 ? sU : xdir ? sB : sA;
            const Real *const q = from + r * RS + c;
            const int on = xdir ? 2 * NC : 3 * NC, ot = 5 * NC - on;
            auto get = [&](const Real *p) { return Cell<Real>{p[0], p[NC], p[on], p[ot]}; };
            const Consts &K = KK[xdir ? 0 : 1];
            Cell<Real> s0, F;
            {
                const Cell<Real> cm1 = get(q - s), c0 = get(q);
                s0 = Phys::slope(cm1, c0, get(q + s), K);
                F = sweep_flux<Phys>(!xdir, phase == 2, cm1, c0, shfl_up(s0), s0, K);
            }
            // (a residual build's update takes them in FP64: widened once, four
            // conversions a task less than after the shuffle)
            using Flux = std::conditional_t<kResidual, double, Real>;
            const Cell<Flux> FR = {Flux(F.rho), Flux(F.p), Flux(F.un), Flux(F.ut)}, FL = shfl_up(FR);
            // the updated cell: one back along the line
            const int ru = xdir ? r : r + 1, cu = xdir ? c - 1 : c;
            if constexpr (TAPE) {
                // the interface before this lane's cell, kept at the cell:
                // cells 2 .. n-2 along x, rows n-3 .. 1 along y
                const int x = x0 - 2 + c, y = y0 - 2 + r;
                const bool in = xdir ? x <= a.nx - 2 && (x < x0 + T::TX || x == a.nx - 2) && (phase || owns_y(y))
                                     : y <= a.ny - 3 && (y >= y0 || by == 0) && (phase || owns_x(x));
                if (mine && k >= 1 && in) store_cell(tape->F[phase == 0 ? (xdir ? 0 : 1) : xdir ? 3 : 2], x, y, 2, 3, F);
            }
            if (!mine || k < 2) continue;
            auto old = [&] {
                if constexpr (kResidual)
                    return join_cell(get(q - s), lo_parts((phase == 0 ? lU : xdir ? lB : lA)[ru * T::kLo + cu], !xdir));
                else
                    return get(q - s);
            };
            auto updated = [&] {
                if constexpr (kResidual)
                    return Phys::update_split(old(), FL, FR, K);
                else
                    return Phys::update(old(), FL, FR, K);
            };
            if (!MERGE && phase == 2) {
                if (x0 - 2 + cu > a.nx - 3) continue;
                if constexpr (kResidual)
                    finish(ru, cu, Phys::template update_split<true>(old(), FL, FR, K, branch_a(ru, cu)));
                else
                    finish(ru, cu, updated());
                continue;
            }
            Real *const d = (phase == 0 ? (xdir ? sA : sB) : xdir ? sR : sU) + ru * RS + cu;
            const auto v = updated();
            if constexpr (kResidual) {
                const Cell<Real> h =
                    split_cell<Real>(v, !xdir, (phase == 0 ? (xdir ? lA : lB) : lU)[ru * T::kLo + cu]);
                d[0] = h.rho;
                d[NC] = h.p;
                d[on] = h.un;
                d[ot] = h.ut;
            } else {
                d[0] = v.rho;
                d[NC] = v.p;
                d[on] = v.un;
                d[ot] = v.ut;
                if constexpr (TAPE) {
                    const int x = x0 - 2 + cu, y = y0 - 2 + ru;
                    if (phase == 0 && xdir && x <= a.nx - 3 && owns_y(y)) store_cell(tape->A1, x, y, 2, 3, v);
                    if (phase == 0 && !xdir && y <= a.ny - 3 && owns_x(x)) store_cell(tape->B1, x, y, 3, 2, v);
                }
            }
        }
        __syncthreads();
    }
    if constexpr (MERGE) {
        for (int i = tid; i < T::TX * T::TY; i += T::NT) {
            const int r = 2 + i / T::TX, c = 2 + i % T::TX;
            if (c >= ncol - 2 || r >= nrow - 2) continue;
            const Real *const rb = sR + r * RS + c;
            finish(r, c, Cell<Real>{rb[0], rb[NC], rb[2 * NC], rb[3 * NC]});
        }
    }
    return true;
}

// Largest value of a warp's lanes, all non-negative (NaN loses): as unsigned
// integers, high words first.
__device__ __forceinline__ double warp_max(double v)
{
#if defined(__CUDA_ARCH__)
    const unsigned long long b = v > 0.0 ? (unsigned long long)__double_as_longlong(v) : 0ull;
    const unsigned hi = unsigned(b >> 32), top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = __reduce_max_sync(0xffffffffu, hi == top ? unsigned(b) : 0u);
    return __longlong_as_double((long long)((unsigned long long)top << 32 | lo));
#else
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
#endif
}

// The record of the step in place `slot` (0, 1) of a group, with the step
// before it committed and the next one planned as finish_step does.  Every
// block of a step makes it for itself, the whole warp alike.  (Of smax a
// value being gathered or cleared is read as well, and not used.)
__device__ __forceinline__ TileRecord fold_record(const StepControl *ctl, int slot, const PlanParams &plan)
{
    TileRecord r = ctl->rec[slot];
    unsigned long long m[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) m[k] = ctl->smax[k];
    const int limit = ctl->step_limit;
    if (r.pending) {
        const int k = (r.steps + 1) & 3;
        r.smax_last = __longlong_as_double((long long)(k < 2 ? (k ? m[1] : m[0]) : (k == 2 ? m[2] : m[3])));
        r.t = r.t + r.dt;
        r.steps += 1;
        r.pending = 0;
        r.parity ^= 1;
        r.ring_due = 1;
        plan_step(&r, limit, plan);
    }
    return r;
}

// The step of a group in place `slot`, for tile_step; in the first block of
// its problem the record is also handed on.
__device__ __forceinline__ TileStep begin_tile(StepControl *ctl, int slot, const PlanParams &plan, bool first)
{
    TileRecord r = fold_record(ctl, slot, plan);
    const TileStep now = {r.t, r.dt, r.active, r.steps};
    if (first && (threadIdx.x & 31) == 0) {
        r.pending = r.active;
        ctl->rec[slot ^ 1] = r;
        ctl->smax[(r.steps + 2) & 3] = 0ull;
    }
    return now;
}

// Folds the block's wave-speed maximum and health into the record of the step
// that follows `steps` committed ones.  Nothing waits for them: the next
// kernel starts when this one has ended.
template <int NT>
__device__ __forceinline__ void end_tile(double vmax, int bad, StepControl *ctl, int steps)
{
    __shared__ double red[NT / 32];
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicCAS(&ctl->first_bad, 0, steps + 1);
    vmax = warp_max(vmax);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x / 32] = vmax;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    vmax = warp_max(threadIdx.x < NT / 32 ? red[threadIdx.x] : 0.0);
    if (threadIdx.x == 0 && vmax > 0.0)
        atomicMax(&ctl->smax[(steps + 1) & 3], (unsigned long long)__double_as_longlong(vmax));
}

// Ends a group of steps: commits record `r`, folded from the group's last
// step, and opens the next group.  One thread, after every block's fold.
__device__ __forceinline__ void commit_record(StepControl *ctl, const TileRecord &r)
{
    ctl->t = r.t;
    ctl->dt = r.dt;
    ctl->smax_last = r.smax_last;
    ctl->steps = r.steps;
    ctl->active = r.active;
    ctl->done = r.done;
    ctl->parity = r.parity;
    ctl->smax_bits = 0ull;
    ctl->ticket = 0u;
    open_record(ctl);
}

#ifdef __CUDACC__  // (host builds of this file call tile_step)
// A block per tile.  A grid's second dimension ends at 65535; the tile rows of
// an array of more (30 cells each: 1,966,054 rows) go on in the third, whose
// last layer has blocks past the end.  (One dimension and a division per block
// measured 0.3% slower at 4096^2.)
constexpr int kTileRowsPerLayer = 65535;
template <class T>
dim3 tile_grid(int nx, int ny)
{
    const int rows = (ny - 4 + T::TY - 1) / T::TY, layers = (rows + kTileRowsPerLayer - 1) / kTileRowsPerLayer;
    return dim3((nx - 4 + T::TX - 1) / T::TX, rows < kTileRowsPerLayer ? rows : kTileRowsPerLayer, layers);
}
__device__ __forceinline__ int tile_row() { return int(blockIdx.y) + kTileRowsPerLayer * int(blockIdx.z); }

// Step `place` of its group.
template <typename Real, class Phys, class T, int MINB>
__global__ void __launch_bounds__(T::NT, MINB) step_tile_kernel(TileArgs<Real> a, int place)
{
    extern __shared__ __align__(16) unsigned char tile_smem[];
    pdl_launch();
    pdl_wait();
    const int by = tile_row();
    if (by >= (a.ny - 4 + T::TY - 1) / T::TY) return;
    const bool first = blockIdx.x == 0 && by == 0;
    double vmax = first && threadIdx.x == 0 ? ring_speed<Real>(a.strategy, a.gamma) : 0.0;
    int bad = 0;
    if (tile_step<Real, Phys, T>(a, blockIdx.x, by, tile_smem,
                                 [&] { return begin_tile(a.ctl, place & 1, a.plan, first); }, place > 0, vmax, bad))
        end_tile<T::NT>(vmax, bad, a.ctl, reinterpret_cast<TileHead<Real, Phys> *>(tile_smem)->step.steps);
}

// A taped step.
template <typename Real, class Phys, class T, int MINB>
__global__ void __launch_bounds__(T::NT, MINB) step_tape_kernel(TileArgs<Real> a, TapeArgs<Real> tape, int place)
{
    extern __shared__ __align__(16) unsigned char tile_smem[];
    pdl_launch();
    pdl_wait();
    const int by = tile_row();
    if (by >= (a.ny - 4 + T::TY - 1) / T::TY) return;
    const bool first = blockIdx.x == 0 && by == 0;
    double vmax = first && threadIdx.x == 0 ? ring_speed<Real>(a.strategy, a.gamma) : 0.0;
    int bad = 0;
    if (tile_step<Real, Phys, T, true>(a, blockIdx.x, by, tile_smem,
                                       [&] { return begin_tile(a.ctl, place & 1, a.plan, first); }, place > 0, vmax, bad,
                                       &tape))
        end_tile<T::NT>(vmax, bad, a.ctl, reinterpret_cast<TileHead<Real, Phys> *>(tile_smem)->step.steps);
}

// Ends a group of `steps` steps in tiles (src, dst: the state if the parity
// is even, odd): stores the ghost ring, one thread per ring cell, and, in the
// last block, commits the record.
template <typename Real, int NT>
__global__ void __launch_bounds__(NT) end_steps_kernel(TileArgs<Real> a, int steps, int residual)
{
    pdl_launch();
    pdl_wait();
    const TileRecord r = fold_record(a.ctl, steps & 1, a.plan);
    if (r.ring_due) {
        if (r.parity) a.src = a.dst;
        GhostArgs<Real> g = ring_args(a);
        g.residual = residual;
        const int k = blockIdx.x * NT + threadIdx.x;
        if (k < 4 * a.nx + 4 * (a.ny - 4)) ghost_cell(g, k, r.t);
    }
    if (last_block_done(&a.ctl->ticket)) commit_record(a.ctl, r);
}
#endif

} // namespace FVM2D_VARIANT
} // namespace fvm2d
