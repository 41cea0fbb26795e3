// fvm2d_fp64_strict.cu -- FP64 kernels in the reference's operation order,
// compiled with -fmad=false (FVM2D_FP64_STRICT): every operation rounds on its
// own, in the reference's order, so results agree bit for bit with the
// reference built with -fmad=false and with the CPU oracle.  Most of its
// quotients come from shared reciprocals, correctly rounded (fvm2d_quotient.cuh).
#define FVM2D_VARIANT fp64_strict
#define FVM2D_REAL double
#define FVM2D_PHYS RefOrderShared
// resident sweep blocks per SM (128 threads each) that the register
// budget is fitted to; measured best for this build (1003^2: 383 us per step,
// 393 with 3, 437 with 2, 687 with divisions)
#define FVM2D_X_MINB 4
#define FVM2D_Y_MINB 4
// tiles of a step (fvm2d_tile.cuh): warps per block and resident blocks per SM,
// and the rule on sizes (best_tile_shape).  Quotients from shared reciprocals
// keep many values at hand: one block per SM with 113-204 registers a thread
// beat two with 72-96 and their spills (us per step, best shape at each size,
// divisions in two blocks / quotients in two / quotients in one: 100^2
// 27 / 26 / 11, 280^2 79 / 58 / 41, 400^2 119 / 91 / 72, 1003^2 524 / 389 / 324,
// 2048^2 1760 / 1375 / 1290)
#define FVM2D_TILE0_WARPS 16
#define FVM2D_TILE0_MINB 1
#define FVM2D_TILE1_WARPS 16
#define FVM2D_TILE1_MINB 1
#define FVM2D_TILE2_WARPS 18
#define FVM2D_TILE2_MINB 1
#define FVM2D_TILE3_WARPS 10
#define FVM2D_TILE3_MINB 1
// 30 x 30 against 30 x 14 around 2 x 148 tiles: 400^2, 196 tiles, 87 / 73; 520^2,
// 324, 119 / 118; 610^2, 441, 128 / 155.  30 x 14 against 14 x 14 around 2 x 148:
// 280^2, 200, 50 / 41; 330^2, 264, 50 / 54; 400^2, 406, 73 / 78.
#define FVM2D_TILE0_NEED 2
#define FVM2D_TILE1_NEED 2
#include "fvm2d_quotient.cuh"
#include "fvm2d_variant.inc"
