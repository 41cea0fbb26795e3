// solver_runtime_host.cpp -- the solver's host runtime (fvm2d_capi.cu) over a
// stand-in for the CUDA runtime and for the builds' kernels, so that its
// decisions can be tested without a GPU (tests/test_solver_runtime_host.py).
// A run's steps are of size step_dt, the last one shorter.
#include "fake_cudart.h"

#include "../2d_fvm_cuda_b200/csrc/fvm2d_adjoint.h"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_control.h"

using fvm2d::LaunchConfig;
using fvm2d::StepControl;

namespace {
double step_dt = 1.0;
long enqueued = 0, ran = 0, groups = 0;

void plan(StepControl *c, const LaunchConfig &l)
{
    c->active = 0;
    if (c->done || c->steps >= c->step_limit) return;
    if (!(c->t < l.plan.t_end)) {
        c->done = 1;
        return;
    }
    c->dt = step_dt < l.plan.t_end - c->t ? step_dt : l.plan.t_end - c->t;
    c->active = 1;
}
void kernel(const std::string &name, void **args)
{
    if (name.find("show_record") != std::string::npos)
        **static_cast<StepControl **>(args[1]) = **static_cast<const StepControl **>(args[0]);
}
cudaError_t init(const LaunchConfig &l)
{
    fake::on_kernel = kernel;
    plan(l.ctl, l);
    return cudaSuccess;
}
cudaError_t end_steps(const LaunchConfig &l)
{
    ++groups;
    enqueued += l.step;
    StepControl *c = l.ctl;
    for (int k = 0; k < l.step && c->active; ++k) {
        c->t = c->t + c->dt;
        c->steps += 1;
        c->parity ^= 1;
        ++ran;
        plan(c, l);
    }
    return cudaSuccess;
}
} // namespace

#define BUILD(ns)                                                                                        \
    namespace fvm2d {                                                                                    \
    namespace ns {                                                                                       \
    cudaError_t prepare() { return cudaSuccess; }                                                        \
    cudaError_t enqueue_init(const LaunchConfig &c, cudaStream_t) { return init(c); }                    \
    cudaError_t enqueue_plan(const LaunchConfig &c, cudaStream_t) { return init(c); }                    \
    cudaError_t enqueue_plan_from(const LaunchConfig &, cudaStream_t, const double *) { return cudaSuccess; } \
    cudaError_t enqueue_step(const LaunchConfig &, cudaStream_t, cudaEvent_t *) { return cudaSuccess; }  \
    cudaError_t enqueue_tile_step(const LaunchConfig &, cudaStream_t) { return cudaSuccess; }            \
    cudaError_t enqueue_end_steps(const LaunchConfig &c, cudaStream_t) { return end_steps(c); }          \
    }                                                                                                    \
    }
#define TAPED(ns)                                                                                        \
    namespace fvm2d {                                                                                    \
    namespace ns {                                                                                       \
    cudaError_t enqueue_step_taped(const LaunchConfig &, cudaStream_t, void *const *, void *) { return cudaSuccess; } \
    cudaError_t enqueue_tile_step_taped(const LaunchConfig &, cudaStream_t, void *const *, void *) { return cudaSuccess; } \
    }                                                                                                    \
    }
#define ADJOINT(ns)                                                                                      \
    namespace fvm2d {                                                                                    \
    namespace ns {                                                                                       \
    cudaError_t adjoint_step(const AdjointLaunch &, cudaStream_t) { return cudaSuccess; }                \
    cudaError_t adjoint_sum(const AdjointLaunch &, cudaStream_t) { return cudaSuccess; }                 \
    }                                                                                                    \
    }
BUILD(fp64)
BUILD(fp64_strict)
BUILD(fp64_reforder)
BUILD(fp32)
BUILD(fp32r)
BUILD(jvp)
TAPED(fp64)
TAPED(fp32)
ADJOINT(adj)
ADJOINT(adj32)

extern "C" {
// Buffers that count as the caller's device memory from now on (n = 0: none).
void sr_device(void *p, size_t n)
{
    fake::device.clear();
    fake::device_copies = 0;
    if (n) fake::device.push_back({static_cast<char *>(p), n});
}
long sr_device_copies() { return fake::device_copies; }
void sr_run(double dt) { step_dt = dt, enqueued = ran = groups = 0; }
// steps enqueued, steps that ran, groups of steps
void sr_seen(long *out) { out[0] = enqueued, out[1] = ran, out[2] = groups; }
}
