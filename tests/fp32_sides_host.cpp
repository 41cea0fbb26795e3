// fp32_sides_host.cpp -- which side of the contact the single-precision flux
// and its adjoint take, compiled for the host (tests/test_fp32_sides_host.py).
#include "cuda_host_emu.h"

#define FVM2D_VARIANT host32
#define FVM2D_REAL float
#include "../2d_fvm_cuda_b200/csrc/fvm2d_kernels.cuh"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_adjoint.inc"
#include "../2d_fvm_cuda_b200/csrc/fvm2d_packed.cuh"

using namespace fvm2d::host32;

extern "C" {

// v: n interfaces, each UL, UR, sL, sR as (rho, p, un, ut).  The side whose
// tangential velocity the flux carries, found by changing the right one's:
// taken[0] interfaces of the left, taken[1] of the right, and in *wrong those
// whose adjoint reaches the other side's.
void fs_sides(const float *v, long n, double h, double dt, double alpha, double gamma, long *taken, long *wrong)
{
    SweepConsts<float> K;
    K.h = float(h);
    K.rh = float(1.0 / h);
    K.alpha = float(alpha);
    set_gamma_consts(K, gamma);
    K.k = float(dt);
    K.lambda = float(dt / h);
    K.lambda_lo = 0.f;
    taken[0] = taken[1] = *wrong = 0;
    for (long i = 0; i < n; ++i) {
        Cell<float> c[4];
        for (int q = 0; q < 4; ++q) c[q] = {v[16 * i + 4 * q], v[16 * i + 4 * q + 1], v[16 * i + 4 * q + 2], v[16 * i + 4 * q + 3]};
        const Cell<float> F = PackedCompensated::interface_flux(c[0], c[1], c[2], c[3], K);
        Cell<float> other = c[1];
        other.ut += 1.f;
        const bool right = PackedCompensated::interface_flux(c[0], other, c[2], c[3], K).ut != F.ut;
        Cell<float> a = {0, 0, 0, 0}, b = a, sa = a, sb = a;
        interface_flux_adjoint(c[0], c[1], c[2], c[3], K, Cell<float>{0, 0, 0, 1}, a, b, sa, sb);
        ++taken[right];
        *wrong += right ? a.ut != 0.f || b.ut == 0.f : a.ut == 0.f || b.ut != 0.f;
    }
}

} // extern "C"
