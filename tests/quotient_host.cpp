// quotient_host.cpp -- correctly rounded quotients from shared reciprocals
// (2d_fvm_cuda_b200/csrc/fvm2d_quotient.cuh) compiled for the host with g++,
// against division and against the reference-order arithmetic they stand in
// for, for tests/test_quotient_host.py.
#include "cuda_host_emu.h"

#define FVM2D_VARIANT host
#define FVM2D_REAL double
#include "../2d_fvm_cuda_b200/csrc/fvm2d_quotient.cuh"

using namespace fvm2d::host;

namespace {

bool same(double x, double y) { return std::isnan(x) ? std::isnan(y) : std::memcmp(&x, &y, 8) == 0; }
bool same(const Cell<double> &x, const Cell<double> &y)
{
    return same(x.rho, y.rho) && same(x.p, y.p) && same(x.un, y.un) && same(x.ut, y.ut);
}

} // namespace

// Of n quotients a[k] / b[k]: how many were taken (in range), and how many of
// those differ from division.
extern "C" void qh_quotients(const double *a, const double *b, long n, long *taken, long *wrong)
{
    *taken = *wrong = 0;
    for (long k = 0; k < n; ++k) {
        bool ok = true;
        const double q = quotient(a[k], Divisor(b[k], ok), ok);
        *taken += ok;
        *wrong += ok && !same(q, a[k] / b[k]);
    }
}

// n interfaces and updates from rows of 16 values (two cells, two slopes; of
// the update: cell, two fluxes): how many differ from RefOrder's, and how many
// interfaces took no division path.
extern "C" void qh_physics(const double *v, long n, double gamma, double h, double dt, long *wrong, long *shared)
{
    SweepConsts<double> K;
    K.h = h;
    K.rh = 1.0 / h;
    K.alpha = 1.9;
    set_gamma_consts(K, gamma);
    K.k = dt;
    K.lambda = dt / h;
    K.lambda_lo = 0.0;
    *wrong = *shared = 0;
    for (long k = 0; k < n; ++k) {
        const double *r = v + 16 * k;
        const Cell<double> c[4] = {{r[0], r[1], r[2], r[3]}, {r[4], r[5], r[6], r[7]}, {r[8], r[9], r[10], r[11]},
                                   {r[12], r[13], r[14], r[15]}};
        *wrong += !same(RefOrderShared::interface_flux(c[0], c[1], c[2], c[3], K),
                        RefOrder::interface_flux(c[0], c[1], c[2], c[3], K));
        *wrong += !same(RefOrderShared::update(c[0], c[2], c[3], K), RefOrder::update(c[0], c[2], c[3], K));
        bool ok = true;
        Cell<double> L, R;
        face_states(c[0], c[1], c[2], c[3], K.h, L, R);
        relaxation_grp_shared(L, R, c[2], c[3], K.g, K.gm1, K.igm1, ok);
        *shared += ok;
    }
}
