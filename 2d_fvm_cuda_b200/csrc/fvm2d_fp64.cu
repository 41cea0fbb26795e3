// fvm2d_fp64.cu -- FP64 kernels with hoisted reciprocals and every FMA written
// out (compiled without contraction): the product default (FVM2D_FP64).
// Checked against the reference within a relative L1 tolerance.
#define FVM2D_VARIANT fp64
#define FVM2D_REAL double
#define FVM2D_PHYS Hoisted
#define FVM2D_TAPED_STEP  // also the taped step of the differentiation form
// reciprocals and reciprocal square roots from the hardware seeds and one
// third-order refinement (rrcp/rrsqrt in fvm2d_math.cuh)
#define FVM2D_FAST_RCP
// resident sweep blocks per SM (128 threads each) that the register
// budget is fitted to; measured best for this build at 4096^2
#ifdef FVM2D_TUNE_X
#define FVM2D_X_MINB FVM2D_TUNE_X
#define FVM2D_Y_MINB FVM2D_TUNE_Y
#else
#define FVM2D_X_MINB 5
#define FVM2D_Y_MINB 5
#endif
// tiles of a step (fvm2d_tile.cuh): warps per block and resident blocks per SM,
// and the rule on sizes (best_tile_shape); measured best of several for this build
#define FVM2D_TILE0_WARPS 10
#define FVM2D_TILE0_MINB 2
#define FVM2D_TILE1_WARPS 5
#define FVM2D_TILE1_MINB 4
#define FVM2D_TILE2_WARPS 7
#define FVM2D_TILE2_MINB 3
#define FVM2D_TILE3_WARPS 10
#define FVM2D_TILE3_MINB 2
#define FVM2D_TILE1_TX 14
// (30 x 30 against 14 x 14 around 1.3 x 296 tiles: 520^2, 324 tiles, 43.9 / 39.5
// us per step; 610^2, 441, 47.8 / 50.9)
#define FVM2D_TILE0_NEED 1.3
#include "fvm2d_variant.inc"
