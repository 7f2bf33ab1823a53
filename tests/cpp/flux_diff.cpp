// hllc_flux_diff_side, the HLLC face difference of the resident barotropic form, compiled for the host:
// the flux difference of n pairs of states, each across side s[i], into d.
#include <math.h>

#include "drifter_b200.h"
#include "flux.cuh"

extern "C" void hllc_diff_batch(int n, const double *UL, const double *UR, const int *s, double g, double *d) {
    for (int i = 0; i < n; ++i)
        drf::hllc_flux_diff_side(UL + 3 * i, 1.0 / UL[3 * i], UR + 3 * i, s[i], g, d + 3 * i);
}
