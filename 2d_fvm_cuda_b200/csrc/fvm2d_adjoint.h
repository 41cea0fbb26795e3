// fvm2d_adjoint.h -- entry points of the adjoint step (fvm2d_adjoint.inc,
// built as fvm2d_adjoint.cu in FP64 and fvm2d_adjoint32.cu in FP32).
#pragma once

#include <cuda_runtime.h>

namespace fvm2d {

// One reverse step of a build with shared reciprocals at fixed dt, from the
// tape of its forward step (enqueue_step_taped of fp64 or fp32).  All buffers
// are state-sized, 4 planes of pitch x ny values of the build's type.
struct AdjointLaunch {
    int nx, ny, pitch, strategy;
    long long plane;
    double hx, hy, rhx, rhy, alpha, gamma, dt;
    const void *U;         // input state of the step
    const void *A1, *B1;   // X(U) and Y(U)
    const void *flux[4];   // interface fluxes of the sweeps X(U), Y(U), Y(A1), X(B1)
    void *lb[2];           // in: the adjoint of the step's output state, the sum of the two;
                           // out: the adjoint of its input state, likewise (branch A's and branch B's)
    void *work[3];         // work states
};

#define FVM2D_DECLARE_ADJOINT(ns)                                                 \
    namespace ns {                                                                \
    cudaError_t adjoint_step(const AdjointLaunch &L, cudaStream_t s);            \
    /* lb[0] += lb[1]: the adjoint as one state, after the last step */          \
    cudaError_t adjoint_sum(const AdjointLaunch &L, cudaStream_t s);             \
    }

FVM2D_DECLARE_ADJOINT(adj)    // FP64
FVM2D_DECLARE_ADJOINT(adj32)  // FP32

} // namespace fvm2d
