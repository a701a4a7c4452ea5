// CheckReconstruction on bit planes (bits_close_level) on the CPU, one warp, for test_mask_closure.py.
#include "host_warp.hpp"

#include "awcm2d_bits.cuh"

// plane: ny + 6 rows of nwx words.  The levels of spacing 2^t0 .. 2^(maxl-1), fine to coarse.
extern "C" int close_plane(int nx, int ny, int maxl, int nwx, int t0, uint32_t* plane)
{
    using namespace awcm;
    Grid2 g{};
    g.nx = nx, g.ny = ny, g.maxl = maxl, g.pitch = 32 * nwx, g.rows = ny + 2 * kGhost;
    Bits2 B{};
    B.nwx = nwx;
    B.rpw = close_rows_per_warp(nwx);
    B.chunks = (nwx + kCloseKeep - 1) / kCloseKeep;
    for (int t = t0; t < maxl; ++t)
        if (!host_warp::run([&](unsigned lane) {
                bits_close_level(g, B, plane + (size_t)kGhost * nwx, t, Span{lane, host_warp::kLanes}, 0);
            }))
            return 1;
    return 0;
}
