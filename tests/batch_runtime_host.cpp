// batch_runtime_host.cpp -- the batch's host runtime (fvm2d_batch_host.cu) over
// a stand-in for the CUDA runtime and for the builds' kernels, so that its
// decisions can be tested without a GPU (tests/test_batch_runtime_host.py).
// Build k's tile of shape s is (k + 1) x (s + 1) tiles a problem; a step takes
// step_ms[1] in tiles and step_ms[0] sweep by sweep, and the first of the
// process first_ms more.  Problem p ends after ends + stagger p steps.
#include "fake_cudart.h"

#include "../2d_fvm_cuda_b200/csrc/fvm2d_batch_control.h"

using fvm2d::BatchLaunch;
using fvm2d::StepControl;

namespace {
const BatchLaunch *last = nullptr;
double step_ms[2] = {2.0, 1.0}, first_ms = 0.0;
int ends = 20, stagger = 0;
long fail_at = -1;            // this sweep by sweep group fails
long groups = 0, bad = 0;     // groups of sweeps; steps whose tile plan was not their build's
long tile_steps = 0, sweep_steps = 0, mixed = 0;

void run_steps(long n, int tiles)
{
    fake::clock_ms += n * step_ms[tiles] + first_ms;
    first_ms = 0.0;
    (tiles ? tile_steps : sweep_steps) += n;
    for (int p = 0; p < last->np; ++p) {
        StepControl &c = last->ctl[p];
        if (!c.active) continue;
        c.steps += int(n);
        c.t += n * c.dt;
        c.parity ^= tiles ? int(n & 1) : 0;
        const int end = c.step_limit < ends + stagger * p ? c.step_limit : ends + stagger * p;
        if (c.steps >= end) c.steps = end, c.active = 0;
    }
}
cudaError_t graph(long n)
{
    if (groups++ == fail_at) return cudaErrorUnknown;
    if (last->t0) ++mixed;
    run_steps(n, 0);
    return cudaSuccess;
}
cudaError_t init(const BatchLaunch &L)
{
    last = &L;
    fake::graph_launch = graph;
    for (int p = 0; p < L.np; ++p) L.ctl[p].active = 1, L.ctl[p].dt = L.prob[p].plan.t_end / (ends + stagger * p);
    return cudaSuccess;
}
long long tiles_of(int build, int shape) { return (build + 1) * (shape + 1); }
cudaError_t step(const BatchLaunch &L, int build)
{
    if (fake::captured >= 0) return ++fake::captured, cudaSuccess;
    if (!L.t0) return ++mixed, cudaSuccess;  // a step in tiles without its plan
    const long long want = tiles_of(build, L.tile_shape);
    for (int p = 0; p < L.np; ++p) {
        const long long n = L.t0[p + 1] - L.t0[p];
        if (n != want && (n || L.ctl[p].active)) ++bad;
    }
    if (L.t0[L.np] != L.tile_total || L.tile_shape != build) ++bad;
    return cudaSuccess;
}
} // namespace

#define BUILD(ns, k)                                                                            \
    namespace fvm2d {                                                                           \
    namespace ns {                                                                              \
    cudaError_t batch_prepare(int *x, int *y) { return *x = *y = 296, cudaSuccess; }            \
    cudaError_t batch_enqueue_init(const BatchLaunch &L, cudaStream_t) { return init(L); }      \
    cudaError_t batch_enqueue_plan(const BatchLaunch &, cudaStream_t) { return cudaSuccess; }   \
    cudaError_t batch_enqueue_step(const BatchLaunch &L, cudaStream_t) { return step(L, k); }   \
    cudaError_t batch_enqueue_end_steps(const BatchLaunch &L, cudaStream_t)                     \
    {                                                                                           \
        if (!L.t0) ++mixed;                                                                     \
        run_steps(L.step, 1);                                                                   \
        return cudaSuccess;                                                                     \
    }                                                                                           \
    int batch_tile_shape(int, const int *, const int *) { return k; }                           \
    long long batch_tiles(int shape, int, int) { return tiles_of(k, shape); }                   \
    }                                                                                           \
    }
BUILD(fp64, 0)
BUILD(fp64_strict, 1)
BUILD(fp64_reforder, 2)
BUILD(fp32, 3)

namespace fvm2d {
int report_error(int code, const char *) { return code; }
} // namespace fvm2d

extern "C" {
void br_set(double sweep, double tile, double first, long fail, int apart)
{
    stagger = apart;
    step_ms[0] = sweep, step_ms[1] = tile, first_ms = first, fail_at = fail;
    groups = bad = tile_steps = sweep_steps = mixed = 0;
}
void br_ends(int n) { ends = n; }
// steps in tiles, steps sweep by sweep, steps whose plan was another build's,
// calls that mixed the two ways
void br_seen(long *out) { out[0] = tile_steps, out[1] = sweep_steps, out[2] = bad, out[3] = mixed; }
}
