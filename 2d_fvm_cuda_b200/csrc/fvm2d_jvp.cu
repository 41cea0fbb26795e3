// fvm2d_jvp.cu -- tangent-linear build: the FP64 kernels with shared
// reciprocals (Hoisted) instantiated on dual numbers, so every state value
// carries a tangent through the same arithmetic (forward-mode
// differentiation of the step, almost everywhere).
//
// Values take the FP64 product build's reciprocals (the hardware seeds with
// one third-order step) and its fma calls, and with them its bits; a
// reciprocal's tangent comes from the reciprocal itself.  Dividing duals
// instead (two IEEE divisions each) took 1.6 times the step.
#define FVM2D_DUAL_RECIPROCALS
#include "fvm2d_dual.cuh"
#define FVM2D_VARIANT jvp
#define FVM2D_FAST_RCP
#include "fvm2d_math.cuh"

namespace fvm2d {
namespace ad {
__device__ __forceinline__ Dual rrcp(Dual a)
{
    const double r = jvp::rrcp(a.v);
    return Dual(r, -(r * r) * a.d);
}
__device__ __forceinline__ Dual rrsqrt(Dual a)
{
    const double r = jvp::rrsqrt(a.v);
    return Dual(r, (-0.5 * r * a.d) * (r * r));
}
} // namespace ad
} // namespace fvm2d

#define FVM2D_REAL fvm2d::ad::Dual
#define FVM2D_PHYS Hoisted
#define FVM2D_X_MINB 2
#define FVM2D_Y_MINB 2
// tiles of a step (fvm2d_tile.cuh): warps per block and resident blocks per SM,
// and the rule on sizes (best_tile_shape); measured best of several: 256 x 300
// 47 -> 40 us per step, 100^2 13.9 -> 10.3
#define FVM2D_TILE0_WARPS 10
#define FVM2D_TILE0_MINB 1
#define FVM2D_TILE1_WARPS 10
#define FVM2D_TILE1_MINB 1
#define FVM2D_TILE2_WARPS 5
#define FVM2D_TILE2_MINB 2
#define FVM2D_TILE3_WARPS 10
#define FVM2D_TILE3_MINB 1
// (30 x 30, 30 x 14 and 14 x 14, us per step: 330^2 45 / 46 / 44, 400^2, 196 tiles
// of 30 x 30 on 148 resident blocks, 81 / 69 / 65, 520^2, 324, 110 / 112 / 103,
// 700^2, 576, 154 / 191 / 175: 30 x 14 is never best)
#define FVM2D_TILE0_NEED 2
#define FVM2D_TILE1_NEED 1e9
#include "fvm2d_variant.inc"
