// fvm2d_fp64_strict.cu -- FP64 kernels in the reference's operation order,
// compiled with -fmad=false (FVM2D_FP64_STRICT): every operation rounds on its
// own, in the reference's order, so results agree bit for bit with the
// reference built with -fmad=false and with the CPU oracle.
#define FVM2D_VARIANT fp64_strict
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
#define FVM2D_TILE0_NEED 3
#define FVM2D_TILE1_NEED 1e9
#include "fvm2d_variant.inc"
