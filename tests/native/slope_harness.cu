// Host harness of the limited slopes: half_slope (the limiter a compile-time
// choice, the signs applied once) next to half of slope_interior, the
// reference's expression, for the CPU test of their bits.
#include "../../piernik_b200/csrc/pk_device.cuh"

using namespace pk;

extern "C" void half_slopes(int lim, const double* dl, const double* dr, long long n, double* got, double* want)
{
    for (long long i = 0; i < n; ++i) {
        want[i] = 0.5 * slope_interior(lim, dl[i], dr[i]);
        got[i] = lim == L_MINMOD   ? half_slope<L_MINMOD>(dl[i], dr[i])
                 : lim == L_MONCEN ? half_slope<L_MONCEN>(dl[i], dr[i])
                                   : half_slope<L_SUPERBEE>(dl[i], dr[i]);
    }
}
