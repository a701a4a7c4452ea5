// The storage layout of a 1D instance on the CPU, for test_layout_1d.py.
#include "host_warp.hpp"

#include "awcm1d_layout.cuh"

// out: tier, list entries per region, bytes.
extern "C" void layout(int nx, int maxl, long avail, int scalar, long* out)
{
    const awcm::Layout1 l = awcm::pick_layout(nx, maxl, (size_t)avail, scalar != 0);
    out[0] = l.tier;
    out[1] = (long)l.cap;
    out[2] = (long)l.bytes;
}
