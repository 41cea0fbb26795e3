// fvm2d_fp64_reforder.cu -- FP64 kernels in the reference's operation order
// with nvcc's default FMA contraction (FVM2D_FP64_REFORDER): the arithmetic
// the reference's own build performs, up to the compiler's contraction
// choices.
#define FVM2D_VARIANT fp64_reforder
#define FVM2D_REAL double
#define FVM2D_PHYS RefOrder
// resident sweep blocks per SM (128 threads each) that the register
// budget is fitted to; measured best for this build at 4096^2
#define FVM2D_X_MINB 4
#define FVM2D_Y_MINB 4
// tiles of a step (fvm2d_tile.cuh): warps per block and resident blocks per SM,
// and the rule on sizes (best_tile_shape); measured best of several for this build
#define FVM2D_TILE0_WARPS 10
#define FVM2D_TILE0_MINB 2
#define FVM2D_TILE1_WARPS 10
#define FVM2D_TILE1_MINB 2
#define FVM2D_TILE2_WARPS 14
#define FVM2D_TILE2_MINB 2
#define FVM2D_TILE3_WARPS 10
#define FVM2D_TILE3_MINB 2
// (30 x 30, 30 x 14 and 14 x 14, us per step: 400^2 151 / 137 / 118, 700^2, 576
// tiles of 30 x 30 on 296 resident blocks, 284 / 306 / 283, 1003^2, 1156, 505 /
// 521 / 521: 30 x 14 is never best by more than 1%)
#define FVM2D_TILE0_NEED 3
#define FVM2D_TILE1_NEED 1e9
#include "fvm2d_variant.inc"
