// flux_guard_host.cpp -- TEST INFRASTRUCTURE.  The exact HLLD flux's common
// path (hlld_flux_sel) and the reference's arithmetic in full
// (hlld_flux_ieee), as host functions.
#include "physics.cuh"

using namespace rmhd2d;

// n interfaces: states of 8 doubles (rho, u, v, w, bX, bY, bZ, p) on each
// side, fluxes of 8 out.  taken[k]: hlld_flux_sel formed interface k.
extern "C" void host_fluxes(int n, const double *L, const double *R, double gm, double eps, double *sel, double *full,
                            int *taken)
{
    MdDiv g1;
    const double ygm1 = g1.recip(gm - 1.0);
    for (int k = 0; k < n; ++k) {
        const double *a = L + 8 * k, *b = R + 8 * k;
        const Prim p{a[0], a[1], a[2], a[3], a[4], a[5], a[6], a[7]}, q{b[0], b[1], b[2], b[3], b[4], b[5], b[6], b[7]};
        hlld_flux_ieee(p, q, gm, eps, full + 8 * k);
        taken[k] = hlld_flux_sel(p, q, gm, eps, ygm1, g1.ok, sel + 8 * k);
    }
}
