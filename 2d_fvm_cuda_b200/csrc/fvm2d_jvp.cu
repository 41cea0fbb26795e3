// fvm2d_jvp.cu -- tangent-linear build: the FP64 kernels with shared
// reciprocals (Hoisted) instantiated on dual numbers, so every state value
// carries a tangent through the same arithmetic (forward-mode
// differentiation of the step, almost everywhere).
#include "fvm2d_dual.cuh"
#define FVM2D_VARIANT jvp
#define FVM2D_REAL fvm2d::ad::Dual
#define FVM2D_PHYS Hoisted
#define FVM2D_X_MINB 2
#define FVM2D_Y_MINB 2
// tiles of a step (fvm2d_tile.cuh): warps per block and resident blocks per SM
#define FVM2D_TILE0_WARPS 8
#define FVM2D_TILE0_MINB 1
#define FVM2D_TILE1_WARPS 8
#define FVM2D_TILE1_MINB 1
#define FVM2D_TILE2_WARPS 8
#define FVM2D_TILE2_MINB 1
#define FVM2D_TILE3_WARPS 5
#define FVM2D_TILE3_MINB 1
#include "fvm2d_variant.inc"
