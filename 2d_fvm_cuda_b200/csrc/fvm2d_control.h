// fvm2d_control.h -- records shared by every build of the kernels and the host runtime.
#pragma once

#include <cuda_runtime.h>

namespace fvm2d {

// What a step in tiles hands the next one: the loop as that step began and,
// while `pending`, its own commit (t + dt, steps + 1, its wave-speed maximum)
// and the next plan, which the next kernel makes for itself (fold_record).
struct TileRecord {
    double t, dt, smax_last;
    int steps, active, done;
    int pending;   // 1: the step of size dt has run and is not committed here
    int parity;    // which of the two state buffers holds the state
    int ring_due;  // 1: that state's ghost ring in memory is not filled (steps in
                   // tiles compute the ring cells they load; the end of a group stores them)
};

// Device-resident loop state, one per solver handle.  The kernels of a step
// read the step size from it and the step's last kernel advances it, so the
// time loop of src/wrappers.cuh:196-284 runs without a host round trip.
struct StepControl {
    double t;                      // committed simulation time
    double dt;                     // step size of the step in flight
    double smax_last;              // max wave speed of the committed state
    unsigned long long smax_bits;  // running max (bit pattern of a non-negative double)
    int steps;                     // committed steps
    int step_limit;                // no step starts once `steps` reaches this
    int active;                    // 1 while a step is in flight
    int done;                      // 1 once the loop of wrappers.cuh:196 has ended
    unsigned int ticket;           // last-block detection in grid reductions
    int first_bad;                 // 1-based step that first left an interior cell with NaN or
                                   // non-positive density or pressure; 0: none
    int parity;                    // steps in tiles: which of the two state buffers holds the state
    // Steps in tiles, between the record as planned (open_record) and the end
    // of their group (end_steps): step k of a group reads rec[k % 2] and writes
    // rec[(k + 1) % 2]; a step from n committed steps gathers its wave-speed
    // maximum in smax[(n + 1) % 4] and clears smax[(n + 2) % 4].
    TileRecord rec[2];
    unsigned long long smax[4];
};

// Begins a group of steps in tiles at the record as it stands.
__host__ __device__ inline void open_record(StepControl *c)
{
    TileRecord r;
    r.t = c->t;
    r.dt = c->dt;
    r.smax_last = c->smax_last;
    r.steps = c->steps;
    r.active = c->active;
    r.done = c->done;
    r.pending = 0;
    r.parity = c->parity;
    r.ring_due = 0;
    c->rec[0] = c->rec[1] = r;
    for (int k = 0; k < 4; ++k) c->smax[k] = 0ull;
}

struct PlanParams {
    double t_end;     // end time
    double cfl;       // CFL number
    double hmin;      // min(width/nx, height/ny), wrappers.cuh:202
    double fixed_dt;  // > 0: every step uses this dt (no CFL rule), for differentiation
};

// Everything one build of the kernels needs to enqueue a step.
struct LaunchConfig {
    int nx, ny, pitch;
    long long plane;       // elements between field planes
    void *U, *A, *B;       // state buffers: U holds the state, A and B are sweep scratch
    // steps in tiles: the two state buffers a step goes from one to the other
    // of, the one (0, 1) that holds the state as the group of steps begins,
    // and the step's place in its group (for end_steps: the group's steps)
    void *pair[2] = {nullptr, nullptr};
    int parity = 0, step = 0;
    StepControl *ctl;
    double hx, hy;         // width/nx, height/ny
    double rhx, rhy;       // 1.0/hx, 1.0/hy
    double alpha, gamma;
    int strategy;
    PlanParams plan;
    // Row frame when the array is one row slab of a larger one (a problem
    // split across processes): the global row of local row 0, the global row
    // count (0: ny), and whether the preset fills the top ghost rows (0, 1)
    // and the bottom ones.  Ring rows it does not fill are halo rows, left out
    // of the wave-speed max.
    int row0 = 0, ny_global = 0, fill_top = 1, fill_bottom = 1;
};

// Kernels per step: sweep X, sweep Y, sweep Y, sweep X + average, ghost ring.
// A step in tiles is one kernel, and one more commits a group of them and
// stores the ghost ring.
constexpr int kStepKernels = 5;

// Steps enqueued before the first look at a run's record, of a run that may
// end at any of them.  A step past the end still loads its tiles: 185 us of
// 4096^2 cells, 11 of 1003^2, 2.6 of 100^2, where a look costs about 15.  (One
// step to the end, 4096^2: 4.7 ms with 16 of them, 1.9 so.)
inline long long first_group(long long cells)
{
    const long long n = (1ll << 23) / cells;
    return n < 1 ? 1 : n > 16 ? 16 : n;
}

// x-sweep work items: a warp walks `chunks` chunks of 32 cells of one row and
// updates 32 chunks - 2 cells (the first chunk's first two lanes only feed
// their neighbours).  Item seg of a row updates cells 2 + cells seg ..
// 1 + cells (seg + 1).  Long items waste less; an array must still give
// every resident warp a couple of items, so the chunk count is the largest
// of 8, 4, 2, 1 that does (x_chunks_for).
__host__ __device__ constexpr int x_item_cells(int chunks) { return 32 * chunks - 2; }
__host__ __device__ constexpr int x_items_per_row(int nx, int chunks)
{
    return (nx - 4 + x_item_cells(chunks) - 1) / x_item_cells(chunks);
}
inline int x_chunks_for(long long rows, int nx, long long resident_warps)
{
    int c = 8;
    while (c > 1 && rows * x_items_per_row(nx, c) < 2 * resident_warps) c /= 2;
    return c;
}

// The entry points each build of the kernels provides (namespaces fp64,
// fp64_strict, fp64_reforder, fp32, and jvp: FP64 values with tangents).
#define FVM2D_DECLARE_VARIANT(ns)                                              \
    namespace ns {                                                             \
    cudaError_t prepare();                                                     \
    cudaError_t enqueue_init(const LaunchConfig &c, cudaStream_t s);           \
    cudaError_t enqueue_plan(const LaunchConfig &c, cudaStream_t s);           \
    cudaError_t enqueue_plan_from(const LaunchConfig &c, cudaStream_t s, const double *smax); \
    cudaError_t enqueue_step(const LaunchConfig &c, cudaStream_t s, cudaEvent_t *ev); \
    cudaError_t enqueue_tile_step(const LaunchConfig &c, cudaStream_t s);      \
    cudaError_t enqueue_end_steps(const LaunchConfig &c, cudaStream_t s);      \
    }

FVM2D_DECLARE_VARIANT(fp64)
FVM2D_DECLARE_VARIANT(fp64_strict)
FVM2D_DECLARE_VARIANT(fp64_reforder)
FVM2D_DECLARE_VARIANT(fp32)
FVM2D_DECLARE_VARIANT(fp32r)
FVM2D_DECLARE_VARIANT(jvp)

// The FP64 and FP32 steps keeping what their adjoint needs: X(U) in c.A, Y(U)
// in c.B and the interface fluxes of the four sweeps (X of U, Y of U, Y of A,
// X of B), each stored at the interface's right cell in planes mass, normal
// momentum, energy, tangential momentum.  The step reads c.U and writes its
// result to `out`.  In tiles (whole problems) the result's ghost ring is left
// to the next taped step of its group, which fills it as it loads it, or to
// enqueue_end_steps; the step sweep by sweep is for row slabs.
#define FVM2D_DECLARE_TAPED(ns)                                                                             \
    namespace ns {                                                                                          \
    cudaError_t enqueue_step_taped(const LaunchConfig &c, cudaStream_t s, void *const flux[4], void *out);  \
    cudaError_t enqueue_tile_step_taped(const LaunchConfig &c, cudaStream_t s, void *const flux[4], void *out); \
    }

FVM2D_DECLARE_TAPED(fp64)
FVM2D_DECLARE_TAPED(fp32)

// Records `msg` as the calling thread's fvm2d_last_error() text; returns code.
int report_error(int code, const char *msg);

} // namespace fvm2d
