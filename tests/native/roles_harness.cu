// Host harness of the fused sweep's tile roles (fused_end, fused_roles): for the
// CPU test that no role depends on a cell that the tile does not hold.
#include "../../piernik_b200/csrc/pk_kernels.cuh"

using namespace pk;

// out[stage][t]: bits 0-3 q, slope, flux, upd of position t of the tile whose
// first owned cell is c0, of a pencil of n cells; returns the tile's end
extern "C" int fused_tile_roles(int T, int wrap, int circ, int c0, int n, unsigned char* out)
{
    const int end = fused_end(T, wrap, c0, n);
    for (int stage = 0; stage < 2; ++stage)
        for (int t = 0; t < T; ++t) {
            const unsigned r = t < end ? fused_roles(circ, t, end) : 0u;
            out[stage * T + t] = (unsigned char)((r >> (4 * stage)) & 15u);
        }
    return end;
}
