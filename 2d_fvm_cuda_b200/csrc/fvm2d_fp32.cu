// fvm2d_fp32.cu -- FP32 storage and arithmetic (FVM2D_FP32): the hoisted
// physics in single precision with the compensated conservative update, the
// update and face states in packed FP32x2 instructions; the
// wave-speed reduction, dt and time stay in FP64.  Reports its error against
// the FP64 path rather than matching the reference bit for bit.  Built with
// -prec-div=false -prec-sqrt=false (FP32 division and square root within
// 2 ulp).
#define FVM2D_VARIANT fp32
#define FVM2D_REAL float
#define FVM2D_PHYS PackedCompensated
#define FVM2D_BATCH_PHYS PackedBatch
#define FVM2D_TAPED_STEP  // also the taped step of FP32 differentiation runs
// the FP64 wave speed from reciprocal square roots (fvm2d_math.cuh)
#define FVM2D_FAST_RCP
// resident sweep blocks per SM (128 threads each) that the register
// budget is fitted to
#ifdef FVM2D_TUNE_X
#define FVM2D_X_MINB FVM2D_TUNE_X
#define FVM2D_Y_MINB FVM2D_TUNE_Y
#else
#define FVM2D_X_MINB 6
#define FVM2D_Y_MINB 6
#endif
// tiles of a step (fvm2d_tile.cuh): warps per block and resident blocks per SM,
// and the rule on sizes (best_tile_shape); measured best of several for this build
#define FVM2D_TILE0_WARPS 8
#define FVM2D_TILE0_MINB 4
#define FVM2D_TILE1_WARPS 10
#define FVM2D_TILE1_MINB 3
#define FVM2D_TILE2_WARPS 9
#define FVM2D_TILE2_MINB 3
#define FVM2D_TILE3_WARPS 10
#define FVM2D_TILE3_MINB 2
// (us per step around 0.9 x the resident blocks, the NEEDs of fvm2d_variant.inc:
// 30 x 30 against 30 x 14, 592 blocks: 610^2, 441 tiles, 43.9 / 40.3; 700^2, 576,
// 43.8 / 50.6.  30 x 14 against 14 x 14, 444: 330^2, 264, 20.2 / 17.7; 400^2, 406,
// 20.3 / 21.6)
#include "fvm2d_packed.cuh"
#include "fvm2d_variant.inc"
